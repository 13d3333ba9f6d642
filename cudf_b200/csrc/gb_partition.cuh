// gb_partition.cuh -- hash-partitioned aggregation for high group counts.
//
// When the groups do not fit one CTA's shared memory, per-row global atomics
// into an L2/HBM table are bound by the L2 atomic rate (~0.15-0.19 G/s per
// SM-free table op on B200), far below HBM bandwidth.  This path trades one
// extra write+read of the rows for atomics that stay in shared memory:
//
//   k_rec_scatter     pass 1 (gb_record.cuh): pack each row's key, take its
//                     hash bucket as partition, and store the row as one record
//                     in that partition's region.
//   k_rec_aggregate   pass 2 (gb_record.cuh): one CTA at a time owns a work item
//                     -- a partition, or a record range of a heavy partition --
//                     and aggregates it in a shared-memory table; its groups then
//                     leave as result rows (or are merged into a global spill
//                     table: split partitions, partitions that did not fit, and
//                     VARIANCE/STD, whose second pass looks every group up there).
//   k_rec_spill       applies the records that did not fit their partition's
//                     table to the global spill table.
//
// This file holds what they share with the shared-stage mode (gb_stage.cuh).
#pragma once
#include <cub/block/block_scan.cuh>

#include "gb_kernels.cuh"

namespace gb {

// One unit of pass-2 work: rows [begin, end) of partition `part`'s region.
// `merge` = 1 when the partition is split over several items, whose tables
// then all go to the global table.
struct PartItem {
  int32_t part;
  int32_t merge;
  int64_t begin, end;
};

// Where a partition's groups leave as result rows.
struct EmitRef {
  int64_t limit;                 // rows the columns hold
  unsigned long long* count;     // groups written this way
};

// ---- explicit shared-memory operations (32-bit shared-window addresses) ----
__device__ __forceinline__ void sred_add_u32(uint32_t a, uint32_t v) { asm volatile("red.shared.add.u32 [%0], %1;" ::"r"(a), "r"(v)); }
__device__ __forceinline__ void sred_add_u64(uint32_t a, uint64_t v) { asm volatile("red.shared.add.u64 [%0], %1;" ::"r"(a), "l"(v)); }
__device__ __forceinline__ void sred_add_f64(uint32_t a, double v) { asm volatile("red.shared.add.f64 [%0], %1;" ::"r"(a), "d"(v)); }
__device__ __forceinline__ void sred_min_u32(uint32_t a, uint32_t v) { asm volatile("red.shared.min.u32 [%0], %1;" ::"r"(a), "r"(v)); }
__device__ __forceinline__ void sred_max_u32(uint32_t a, uint32_t v) { asm volatile("red.shared.max.u32 [%0], %1;" ::"r"(a), "r"(v)); }
__device__ __forceinline__ void sred_min_u64(uint32_t a, uint64_t v) { asm volatile("red.shared.min.u64 [%0], %1;" ::"r"(a), "l"(v)); }
__device__ __forceinline__ void sred_max_u64(uint32_t a, uint64_t v) { asm volatile("red.shared.max.u64 [%0], %1;" ::"r"(a), "l"(v)); }
__device__ __forceinline__ uint32_t sld_u32(uint32_t a)
{
  uint32_t v;
  asm volatile("ld.volatile.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ uint64_t sld_u64(uint32_t a)
{
  uint64_t v;
  asm volatile("ld.volatile.shared.u64 %0, [%1];" : "=l"(v) : "r"(a));
  return v;
}

// ---- pass 2 ----
// Per-item prologue: claim a work item, reset the shared table (`scap`
// slots plus, for one-word keys, the slot of the all-ones key).  Returns the
// item index (>= nitems: no work left).
template <int NT>
__device__ __forceinline__ int p2_claim(unsigned int* work, uint8_t* smem, int scap, int nw,
                                        const SlotTemplate& tmpl, int* s_part, unsigned int* s_used,
                                        unsigned int* s_spill)
{
  if (threadIdx.x == 0) {
    *s_part = (int)atomicAdd(work, 1u);
    *s_used = 0;
    *s_spill = 0;
  }
  // word by word: every thread reads the same template word (no divergent
  // parameter loads, no division by the slot width)
  for (int w = 0; w < nw; ++w) {
    const unsigned long long t = tmpl.w[w];
    for (int s = threadIdx.x; s < scap; s += NT) *(unsigned long long*)(smem + ((size_t)s * nw + w) * 8) = t;
  }
  __syncthreads();
  return *s_part;
}

// Per-partition epilogue: the partition's groups leave as result rows, or are
// merged into the global spill table when some of its rows went there.  The
// all-ones key's slot (one-word keys; it cannot be told from an empty slot)
// is always merged into the global table's dedicated slot.
// The rows are written column by column with consecutive lanes on consecutive
// rows.  Against copying the slots out and compacting them afterwards: pass 2
// 2.09 -> 2.23 ms at 1M groups (the compaction took 0.09), 3.52 -> 3.58 at 7.8M
// (0.28), 1.98 -> 1.92 at 25M (0.53).  Out of line it was slower still (2.32 at
// 1M): the plan's fields are then read through generic addresses.
template <int NT, typename ScanT>
__device__ __forceinline__ void p2_flush(const Plan& P2, const TableRef& G, const EmitRef& D, const OutPtrs& O,
                                         const uint8_t* smem, int scap, bool spilled,
                                         typename ScanT::TempStorage& scan_tmp, unsigned int* s_cnt,
                                         unsigned int* s_base, unsigned int* s_new)
{
  const int stride = G.stride;
  if (P2.key_words == 1 && threadIdx.x == 0) {
    const uint8_t* sp = smem + (size_t)scap * stride;
    if (*(const uint32_t*)(sp + P2.rows_off) > 0) merge_slot(P2, G, sp, s_new);
  }
  if (spilled) {
    for (int i = threadIdx.x; i < scap; i += NT) {
      const uint8_t* s = smem + i * stride;
      if (slot_occupied(P2, s, false)) merge_slot(P2, G, s, s_new);
    }
    return;
  }
  // groups per (round of NT slots, warp), then their places
  const int rounds = (scap + NT - 1) / NT;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int k = 0; k < rounds; ++k) {
    const int i = k * NT + threadIdx.x;
    const unsigned m = __ballot_sync(0xFFFFFFFFu, i < scap && slot_occupied(P2, smem + (size_t)i * stride, false));
    if (lane == 0) s_cnt[k * (NT / 32) + warp] = __popc(m);
  }
  __syncthreads();
  const int n = rounds * (NT / 32);  // <= NT
  unsigned off, total;
  ScanT(scan_tmp).ExclusiveSum(threadIdx.x < n ? s_cnt[threadIdx.x] : 0u, off, total);
  if (threadIdx.x < n) s_cnt[threadIdx.x] = off;
  if (threadIdx.x == 0) {
    *s_base = total ? atomicAdd(O.counters + 2, total) : 0u;
    atomicAdd(D.count, (unsigned long long)total);
  }
  __syncthreads();
#pragma unroll 1
  for (int k = 0; k < rounds; ++k) {
    const int i = k * NT + threadIdx.x;
    const uint8_t* s = smem + (size_t)i * stride;
    bool occ = i < scap && slot_occupied(P2, s, false);
    const unsigned m = __ballot_sync(0xFFFFFFFFu, occ);
    if (!m) continue;
    const int64_t pos = (int64_t)*s_base + s_cnt[k * (NT / 32) + warp] + __popc(m & ((1u << lane) - 1));
    if (occ && pos >= D.limit) {
      atomicOr(O.counters + 1, 1u);  // more groups than the columns hold
      occ = false;
    }
    emit_slot(P2, s, occ, pos, O);
  }
}

}  // namespace gb
