// gb_stage.cuh -- the shared-stage mode: groups that fit one CTA's shared
// memory.
//
//   k_stage_aggregate  each CTA aggregates a contiguous row range of the
//                      caller's own columns in shared memory and merges its
//                      table into the global one
//   k_stage_spill      rows whose key fitted no shared table
#pragma once
#include "gb_record.cuh"
#include "gb_stage.h"

namespace gb {

// One CTA, one contiguous row range.  The CTA keeps `replicas` copies of its
// table and thread t works on copy t mod replicas: with few groups the lanes of
// a warp would otherwise queue on the same few slots, whose 64-bit and floating
// reductions are compare-and-swap loops.  The copies are folded into the first
// one at the end, and that one is merged into the global table.  The lanes of a
// warp then meet the same slot of neighbouring copies, so the copies lie an odd
// number of 8-byte units apart (16 for two-word keys): without that pad 60M rows
// of six groups kept the shared-memory pipe 90% busy on bank conflicts.
// Shared memory: per copy tags u32[slots], then per copy slots and pad, then
// the all-ones key's slot.
template <int KW, int MAXV, bool FOLD>
__global__ void __launch_bounds__(1024, 1) k_stage_aggregate(const __grid_constant__ Plan P,
                                                             const __grid_constant__ StageArgs A,
                                                             const __grid_constant__ RecSpec S, TableRef G,
                                                             const __grid_constant__ SlotTemplate tmpl)
{
  constexpr int NT = 1024;
  constexpr int R = MAXV <= 4 ? 2 : 1;
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ unsigned int s_used[kMaxReplicas];
  __shared__ unsigned int s_new;
  const int stride = G.stride;
  const int nw = stride / 8;
  const int total = A.replicas * A.slots;
  uint8_t* const slots = smem + (size_t)total * 4;
  // slot i over all copies; slot `total` is the all-ones key's
  auto slot_at = [&](int i) {
    const int copy = i / A.slots;
    return slots + (size_t)copy * A.pitch + (size_t)(i - copy * A.slots) * stride;
  };
  const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(smem);
  auto table_of = [&](int copy) {
    return RecTable{sbase + 4u * (uint32_t)(copy * A.slots), sbase + 4u * (uint32_t)total + (uint32_t)(copy * A.pitch),
                    (uint32_t)A.slots / 4, stride, A.sfill, (uint32_t)__cvta_generic_to_shared(s_used + copy)};
  };
  for (int i = threadIdx.x; i < total / 4; i += NT) ((uint4*)smem)[i] = make_uint4(0, 0, 0, 0);
  for (int i = threadIdx.x; i < total + (KW == 1); i += NT) {
    uint8_t* const s = slot_at(i);
    for (int w = 0; w < nw; ++w) *(unsigned long long*)(s + w * 8) = tmpl.w[w];
  }
  for (int i = threadIdx.x; i < A.replicas; i += NT) s_used[i] = 0;
  if (threadIdx.x == 0) s_new = 0;
  __syncthreads();
  const RecTable table = table_of(threadIdx.x % A.replicas);
  const uint32_t ones = sbase + 4u * (uint32_t)total + (uint32_t)(A.replicas * A.pitch);
  const int nc = S.ncols;
  const int lane = threadIdx.x & 31;
  const int64_t b = (int64_t)blockIdx.x * A.rows_per_cta;
  const int64_t e = min(P.num_rows, b + A.rows_per_cta);
  // a lane's line of the warp's step (32 R rows of one column) to fetch ahead into L2
  const uint8_t* line = nullptr;
  int line_w = 0;
  {
    int left = lane;
    auto take = [&](const void* data, int64_t offset, int width) {
      const int lines = (32 * R * width + 127) / 128;
      if (left >= 0 && left < lines) {
        line = (const uint8_t*)data + offset * width + left * 128;
        line_w = width;
      }
      left -= lines;
    };
    for (int k = 0; k < P.num_keys; ++k) take(P.keys[k].data, P.keys[k].offset, P.keys[k].width);
    for (int v = 0; v < nc; ++v) take(P.vals[v].data, P.vals[v].offset, P.vals[v].width);
  }
  for (int64_t w0 = b + (threadIdx.x >> 5) * (32 * R); w0 < e; w0 += R * NT) {
    const int64_t row = w0 + lane;
    if (line && w0 + 2 * R * NT + 32 * R <= e)
      asm volatile("prefetch.global.L2 [%0];" ::"l"(line + (w0 + 2 * R * NT) * line_w));
    uint64_t k0[R], k1[R], x[R][MAXV];
    bool live[R];
    unsigned vb[R];
#pragma unroll
    for (int r = 0; r < R; ++r) live[r] = row + 32 * r < e;
    pack_rows<KW, R>(P, row, k0, k1, live);
#pragma unroll
    for (int r = 0; r < R; ++r) vb[r] = 0xFFu;
#pragma unroll
    for (int v = 0; v < MAXV; ++v) {
      if (v >= nc) break;
      const ValCol& c = P.vals[v];
      const int64_t at = row + c.offset;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        x[r][v] = live[r] ? load_bits(c.data, at + 32 * r, c.width) : 0;
        if (c.mask && live[r] && !((__ldg(c.mask + ((at + 32 * r) >> 5)) >> (at & 31)) & 1u)) vb[r] &= ~(1u << v);
      }
    }
    uint32_t sa[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      sa[r] = 0;
      if (live[r]) {
        sa[r] = (KW == 1 && k0[r] == kEmpty) ? ones : rec_slot<KW>(table, k0[r], k1[r], hash_key(k0[r], k1[r], KW));
        if (sa[r] == 0) {
          // listed for the global table; one list reservation per group of lanes
          const unsigned mates = __activemask();
          const int leader = __ffs(mates) - 1;
          unsigned at = 0;
          if (lane == leader) at = atomicAdd(A.counters + 12, (unsigned)__popc(mates));
          at = __shfl_sync(mates, at, leader) + __popc(mates & ((1u << lane) - 1));
          if (at < A.spill_cap) A.spill_rows[at] = row + 32 * r;
          else atomicOr(A.counters + 13, 1u);
        }
      }
    }
    __syncwarp();
    apply_columns<R, MAXV, FOLD>(S, nc, P.rows_off, sa, vb, x);
  }
  // the list overflowed: the call is redone, and its merges would search a full
  // table for each group
  if (__syncthreads_or(threadIdx.x == 0 && *(volatile unsigned int*)(A.counters + 13))) return;
  // the other copies into the first
  const RecTable first = table_of(0);
  for (int i = A.slots + threadIdx.x; i < total; i += NT) {
    const uint8_t* s = slot_at(i);
    if (!slot_occupied(P, s, false)) continue;
    const uint64_t w0 = ((const uint64_t*)s)[0], w1 = KW == 2 ? ((const uint64_t*)s)[1] : 0;
    const uint32_t d = rec_slot<KW>(first, w0, w1, hash_key(w0, w1, KW));
    if (d) merge_fields(P, (uint8_t*)__cvta_shared_to_generic(d), s);
    else merge_slot(P, G, s, &s_new);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < A.slots; i += NT) {
    const uint8_t* s = slots + (size_t)i * stride;
    if (slot_occupied(P, s, false)) {
      if (*(volatile unsigned int*)(G.counters + 1)) break;  // the global table is full: as above
      merge_slot(P, G, s, &s_new);
    }
  }
  if (KW == 1 && threadIdx.x == 0) {
    const uint8_t* s = slot_at(total);
    if (*(const uint32_t*)(s + P.rows_off) > 0) merge_slot(P, G, s, &s_new);
  }
  __syncthreads();
  if (threadIdx.x == 0 && s_new) atomicAdd(G.counters, s_new);
}

static __global__ void __launch_bounds__(256) k_stage_spill(const __grid_constant__ Plan P, TableRef G,
                                                            const __grid_constant__ StageArgs A)
{
  __shared__ unsigned int s_new;
  if (threadIdx.x == 0) s_new = 0;
  __syncthreads();
  unsigned cnt = min(*(volatile unsigned int*)(A.counters + 12), A.spill_cap);
  if (*(volatile unsigned int*)(A.counters + 13) || *(volatile unsigned int*)(G.counters + 1)) cnt = 0;  // redone anyway
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < cnt; i += gridDim.x * blockDim.x) {
    const int64_t r = A.spill_rows[i];
    uint64_t w0, w1;
    if (!pack_key(P, r, w0, w1)) continue;  // not listed: null keys are skipped first
    const int64_t gi = global_slot(P, G, w0, w1, hash_key(w0, w1, P.key_words), &s_new);
    if (gi < 0) {
      atomicOr(G.counters + 1, 1u);
      continue;
    }
    update_slot(P, G.T + gi * (int64_t)G.stride, r);
  }
  __syncthreads();
  if (threadIdx.x == 0 && s_new) atomicAdd(G.counters, s_new);
}

}  // namespace gb
