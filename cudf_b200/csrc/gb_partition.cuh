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
//                     and aggregates it in a shared-memory table; its groups are
//                     then copied out as dense slots (or merged into a global
//                     spill table for split partitions and partitions that did
//                     not fit).
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

struct DenseRef {
  uint8_t* T;                    // dense slots
  int64_t cap;
  unsigned long long* count;     // slots written
  unsigned int* overflow;
};

// ---- explicit shared-memory operations (32-bit shared-window addresses) ----
__device__ __forceinline__ void sred_add_u32(uint32_t a, uint32_t v) { asm volatile("red.shared.add.u32 [%0], %1;" ::"r"(a), "r"(v)); }
__device__ __forceinline__ void sred_add_u64(uint32_t a, uint64_t v) { asm volatile("red.shared.add.u64 [%0], %1;" ::"r"(a), "l"(v)); }
__device__ __forceinline__ void sred_add_f32(uint32_t a, float v) { asm volatile("red.shared.add.f32 [%0], %1;" ::"r"(a), "f"(v)); }
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

// Per-partition epilogue: the partition's groups leave as dense slots, or are
// merged into the global spill table when some of its rows went there.  The
// all-ones key's slot (one-word keys; it cannot be told from an empty slot)
// is always merged into the global table's dedicated slot.
template <int NT, typename ScanT>
__device__ __forceinline__ void p2_flush(const Plan& P2, const TableRef& G, const DenseRef& D,
                                         const uint8_t* smem, int scap, bool spilled,
                                         typename ScanT::TempStorage& scan_tmp,
                                         unsigned long long* s_base, unsigned int* s_new)
{
  const int stride = G.stride;
  const int nw = stride / 8;
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
  const int per = (scap + NT - 1) / NT;
  int first = threadIdx.x * per;
  unsigned mine = 0;
  for (int i = first; i < min(first + per, scap); ++i) mine += slot_occupied(P2, smem + i * stride, false);
  unsigned off, total;
  ScanT(scan_tmp).ExclusiveSum(mine, off, total);
  if (threadIdx.x == 0) *s_base = total ? atomicAdd(D.count, (unsigned long long)total) : 0ull;
  __syncthreads();
  unsigned long long o = *s_base + off;
  for (int i = first; i < min(first + per, scap); ++i) {
    const uint8_t* s = smem + i * stride;
    if (!slot_occupied(P2, s, false)) continue;
    if ((int64_t)o >= D.cap) {
      atomicOr(D.overflow, 1u);
      break;
    }
    unsigned long long* dst = (unsigned long long*)(D.T + o * stride);
    for (int w = 0; w < nw; ++w) dst[w] = ((const unsigned long long*)s)[w];
    ++o;
  }
}

}  // namespace gb
