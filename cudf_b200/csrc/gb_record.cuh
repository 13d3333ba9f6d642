// gb_record.cuh -- the partitioned path's kernels over row records.
//
//   k_rec_scatter    pass 1: every row leaves as one record (key word(s), value
//                    bits, validity byte; see RecSpec) stored at its place in
//                    its hash partition's region
//   k_rec_aggregate  pass 2: one CTA at a time owns a work item (a partition or
//                    a range of a heavy one) and aggregates it in a shared table
//   k_rec_spill      records that did not fit their partition's table
#pragma once
#include <type_traits>

#include "gb_record.h"

namespace gb {

template <int V>
using IntC = std::integral_constant<int, V>;

// Partition of a hash: its bucket (top kBucketBits bits, the sketch's exact
// row counts) scaled to the partition count.
__device__ __forceinline__ unsigned part_of(uint64_t h, int nparts)
{
  return ((unsigned)(h >> (64 - kBucketBits)) * (unsigned)nparts) >> kBucketBits;
}

__device__ __forceinline__ void bulk_prefetch_l2(const void* p, unsigned bytes)
{
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

// ---- record loads ------------------------------------------------
// The record array starts on a multiple of 32 bytes, so a record starts on a
// multiple of 16, and where its size is a multiple of 32 on one of 32: it moves
// as 16- or 32-byte vectors.
template <int RW>
__device__ __forceinline__ void rec_load(const uint64_t* p, uint64_t (&w)[RW])
{
  if constexpr (RW % 4 == 0) {
#pragma unroll
    for (int j = 0; j < RW; j += 4)
      asm volatile("ld.global.nc.v4.b64 {%0, %1, %2, %3}, [%4];"
                   : "=l"(w[j]), "=l"(w[j + 1]), "=l"(w[j + 2]), "=l"(w[j + 3])
                   : "l"(p + j));
  } else {
#pragma unroll
    for (int j = 0; j < RW; j += 2) {
      const ulonglong2 v = __ldg((const ulonglong2*)(p + j));
      w[j] = v.x;
      w[j + 1] = v.y;
    }
  }
}

// ---- pass 1 -----------------------------------------------------------------
// Elements first + k*NT + tid of a column into x (rows with pr = 0xFFFFFFFF are
// skipped), all loads in flight together.
template <typename W, int NT, int RPT>
__device__ __forceinline__ void load_rows(const void* data, int64_t first, const uint32_t (&pr)[RPT], uint64_t (&x)[RPT])
{
  const W* p = (const W*)data + first + threadIdx.x;
#pragma unroll
  for (int k = 0; k < RPT; ++k) x[k] = pr[k] != 0xFFFFFFFFu ? (uint64_t)__ldg(p + k * NT) : 0;
}
__device__ __forceinline__ void sst_u64(uint32_t a, uint64_t v) { asm volatile("st.shared.u64 [%0], %1;" ::"r"(a), "l"(v) : "memory"); }
__device__ __forceinline__ void sst_u32(uint32_t a, uint32_t v) { asm volatile("st.shared.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory"); }
__device__ __forceinline__ void sst_u16(uint32_t a, uint32_t v) { asm volatile("st.shared.u16 [%0], %1;" ::"r"(a), "h"((uint16_t)v) : "memory"); }
__device__ __forceinline__ void sst_u8(uint32_t a, uint32_t v) { asm volatile("st.shared.u8 [%0], %1;" ::"r"(a), "r"(v) : "memory"); }
// Shared -> global bulk copy (multiples of 16 bytes, both ends aligned).
__device__ __forceinline__ void bulk_s2g(void* dst, uint32_t src, unsigned bytes)
{
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(src), "r"(bytes) : "memory");
}
// Global -> shared copy of 4 or 8 bytes without a register in between.
__device__ __forceinline__ void async_copy4(uint32_t dst, const void* src)
{
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void async_copy8(uint32_t dst, const void* src)
{
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}

// Pass 1.  Each CTA walks tiles of T = RPT * NT rows:
//   A  hash the rows' packed keys; partition = hash bucket scaled to the
//      partition count, rank within the (tile, partition) run from a shared
//      histogram;
//   B  one reservation per partition present on its region cursor, issued
//      here and read after C, and the runs' places in the sorted tile
//      (exclusive scan of the histogram);
//   C  the records are put together at their rows' sorted positions in shared
//      memory: 4- and 8-byte columns by asynchronous copies straight from the
//      columns, all of a tile's in flight together, the narrower columns, the
//      keys and the validity bytes through registers;
//   D  every run leaves by one bulk copy; the copies drain while the next tile
//      goes through A and B.  The next tile's keys are loaded before C waits.
// What bounds it is the number of stores that reach L2, not their bytes: this
// GPU takes about 40 G stores a second to different lines, and 32-byte rows go
// out at 40 / 117 / 155 / 174 G rows/s in runs of 1 / 3 / 4 / 5.  So a row is
// one record instead of one element in each of several arrays, and a tile is
// sorted to make runs.
// Shared memory: stage u64[T * words] | hist u32[2][nparts] | validity words u32[nmask][T / 32 + 1]
template <int KW, int NT, int RPT, int MINB, int EARLY>
__global__ void __launch_bounds__(NT, MINB) k_rec_scatter(const __grid_constant__ Plan P,
                                                          const __grid_constant__ RecArgs A,
                                                          const __grid_constant__ RecSpec S)
{
  constexpr int T = NT * RPT;
  static_assert(T < 65536 && NT % 32 == 0, "a run's place and length are 16-bit; a thread's rows share their mask bit");
  using Scan = cub::BlockScan<unsigned, NT, cub::BLOCK_SCAN_WARP_SCANS>;
  __shared__ typename Scan::TempStorage scan_tmp;
  extern __shared__ __align__(16) uint8_t sm[];
  unsigned int* hist = (unsigned int*)(sm + (size_t)T * S.words * 8);  // this tile's; the next tile's is zeroed in B
  unsigned int* next_hist = hist + A.nparts;
  uint32_t* mwords = next_hist + A.nparts;
  const uint32_t sstage = (uint32_t)__cvta_generic_to_shared(sm);
  const int64_t n = P.num_rows;
  const int64_t ntiles = (n + T - 1) / T;
  uint64_t kw0[RPT], kw1[KW == 2 ? RPT : 1];
  uint32_t pr[RPT];  // partition << 16 | rank, then the sorted position; 0xFFFFFFFF: no row
  // the keys of a tile, packed column by column with the loads of all rows in
  // flight together (as pack_key, per row)
  auto load_keys = [&](int64_t tile, uint32_t (&live)[RPT]) {
    const int64_t t0 = tile * T;
#pragma unroll
    for (int k = 0; k < RPT; ++k) {
      kw0[k] = 0;
      if (KW == 2) kw1[k] = 0;
      live[k] = t0 + k * NT + threadIdx.x < n ? 0u : 0xFFFFFFFFu;
    }
    if (KW == 1 && S.key8) {
      load_rows<unsigned long long, NT, RPT>(P.keys[0].data, t0 + P.keys[0].offset, live, kw0);
      return;
    }
#pragma unroll 1
    for (int kc = 0; kc < P.num_keys; ++kc) {
      const KeyCol& c = P.keys[kc];
      const int64_t first = t0 + c.offset;
      uint64_t x[RPT];
      uint32_t valid[RPT];
      switch (c.width) {
        case 1: load_rows<uint8_t, NT, RPT>(c.data, first, live, x); break;
        case 2: load_rows<uint16_t, NT, RPT>(c.data, first, live, x); break;
        case 4: load_rows<uint32_t, NT, RPT>(c.data, first, live, x); break;
        default: load_rows<unsigned long long, NT, RPT>(c.data, first, live, x); break;
      }
#pragma unroll
      for (int k = 0; k < RPT; ++k) valid[k] = 1u;
      if (c.mask) {
        const int64_t r = first + threadIdx.x;
        const uint32_t* m = c.mask + (r >> 5);  // rows NT apart: NT / 32 words apart, one bit position
#pragma unroll
        for (int k = 0; k < RPT; ++k) valid[k] = live[k] != 0xFFFFFFFFu ? __ldg(m + k * (NT / 32)) >> (r & 31) : 0u;
      }
      bool in[RPT];
#pragma unroll
      for (int k = 0; k < RPT; ++k) in[k] = live[k] != 0xFFFFFFFFu;
      if constexpr (KW == 2) fold_key_column<2, RPT>(P, c, x, valid, kw0, kw1, in);
      else fold_key_column<1, RPT>(P, c, x, valid, kw0, kw0, in);
#pragma unroll
      for (int k = 0; k < RPT; ++k)
        if (!in[k]) live[k] = 0xFFFFFFFFu;
    }
  };
  for (int q = threadIdx.x; q < A.nparts; q += NT) hist[q] = 0;
  if (blockIdx.x < ntiles) load_keys(blockIdx.x, pr);
  __syncthreads();
  for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int64_t t0 = tile * T;
    // this tile's validity words on their way into shared memory
    for (int i = threadIdx.x; i < S.nmask * (T / 32 + 1); i += NT) {
      const int m = i / (T / 32 + 1), w = i - m * (T / 32 + 1);
      const ValCol& v = P.vals[S.mask_col[m]];
      const int64_t at = ((t0 + v.offset) >> 5) + w;
      if (at <= (n - 1 + v.offset) >> 5) async_copy4((uint32_t)__cvta_generic_to_shared(mwords + i), v.mask + at);
    }
    // A
#pragma unroll
    for (int k = 0; k < RPT; ++k) {
      if (pr[k] == 0xFFFFFFFFu) continue;
      const unsigned p = part_of(hash_key(kw0[k], KW == 2 ? kw1[k] : 0, KW), A.nparts);
      pr[k] = (p << 16) | atomicAdd(&hist[p], 1u);
    }
    __syncthreads();
    // B
    for (int q = threadIdx.x; q < A.nparts; q += NT) next_hist[q] = 0;  // the last tile's: its D is over
    // thread t holds partitions t, t + NT, ...: neighbouring threads reserve on
    // neighbouring cursors, and the tile is sorted in that order
    auto reserve = [&](int q, unsigned h) -> long long {
      return h ? (long long)atomicAdd(&A.cursor[q], (unsigned long long)h) : 0;
    };
    long long g[EARLY];
    unsigned mine = 0;
    if (EARLY > 1) {
#pragma unroll
      for (int j = 0; j < EARLY; ++j) {
        const int q = threadIdx.x + j * NT;
        const unsigned h = q < A.nparts ? hist[q] : 0u;
        g[j] = reserve(q, h);
        mine += h;
      }
    } else {
      for (int q = threadIdx.x; q < A.nparts; q += NT) mine += hist[q];
    }
    unsigned pre;
    Scan(scan_tmp).ExclusiveSum(mine, pre);
    for (int q = threadIdx.x; q < A.nparts; q += NT) {  // row count << 16 | place in the sorted tile
      const unsigned h = hist[q];
      hist[q] = h << 16 | pre;
      pre += h;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");                // the validity words are here
    asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // the last tile's runs have left the stage
    __syncthreads();
    // C; pr becomes the address of the row's record in the stage
#pragma unroll
    for (int k = 0; k < RPT; ++k) {
      if (pr[k] == 0xFFFFFFFFu) continue;
      const unsigned p = pr[k] >> 16;
      pr[k] = sstage + ((hist[p] & 0xFFFFu) + (pr[k] & 0xFFFFu)) * (8u * S.words);
    }
#pragma unroll 1
    for (int c = 0; c < S.ncols; ++c) {
      const ValCol& v = P.vals[S.src_col[c]];
      if (v.width < 4) continue;
      const uint32_t j = (uint32_t)S.off[c];
      const uint8_t* p = (const uint8_t*)v.data + (t0 + v.offset + threadIdx.x) * v.width;
      if (v.width == 8) {
#pragma unroll
        for (int k = 0; k < RPT; ++k)
          if (pr[k] != 0xFFFFFFFFu) async_copy8(pr[k] + j, p + (size_t)k * NT * 8);
      } else {
#pragma unroll
        for (int k = 0; k < RPT; ++k)
          if (pr[k] != 0xFFFFFFFFu) async_copy4(pr[k] + j, p + (size_t)k * NT * 4);
      }
    }
    // keys: a four-byte key leaves the other half of its word to the columns
#pragma unroll
    for (int k = 0; k < RPT; ++k) {
      if (pr[k] == 0xFFFFFFFFu) continue;
      if (KW == 1 && S.keymask != ~0ull) sst_u32(pr[k], (uint32_t)kw0[k]);
      else sst_u64(pr[k], kw0[k]);
      if (KW == 2) sst_u64(pr[k] + 8u, kw1[k]);
    }
#pragma unroll 1
    for (int c = 0; c < S.ncols; ++c) {
      const ValCol& v = P.vals[S.src_col[c]];
      if (v.width >= 4) continue;
      uint64_t x[RPT];
      if (v.width == 2) load_rows<uint16_t, NT, RPT>(v.data, t0 + v.offset, pr, x);
      else load_rows<uint8_t, NT, RPT>(v.data, t0 + v.offset, pr, x);
      const uint32_t j = (uint32_t)S.off[c];
#pragma unroll
      for (int k = 0; k < RPT; ++k) {
        if (pr[k] == 0xFFFFFFFFu) continue;
        if (v.width == 2) sst_u16(pr[k] + j, (uint32_t)x[k]);
        else sst_u8(pr[k] + j, (uint32_t)x[k]);
      }
    }
    if (S.has_bits) {
      uint32_t vb[RPT];
#pragma unroll
      for (int k = 0; k < RPT; ++k) vb[k] = S.vb_const;
#pragma unroll 1
      for (int m = 0; m < S.nmask; ++m) {
        const uint32_t r = (uint32_t)(P.vals[S.mask_col[m]].offset & 31) + threadIdx.x;  // tiles start on a word
        const uint32_t* w = mwords + m * (T / 32 + 1) + (r >> 5);
        const int bit = S.mask_bit[m];
#pragma unroll
        for (int k = 0; k < RPT; ++k) vb[k] |= ((w[k * (NT / 32)] >> (r & 31)) & 1u) << bit;
      }
      const uint32_t j = 8u * S.words - 1u;
#pragma unroll
      for (int k = 0; k < RPT; ++k)
        if (pr[k] != 0xFFFFFFFFu) sst_u8(pr[k] + j, vb[k]);
    }
    if (tile + gridDim.x < ntiles) load_keys(tile + gridDim.x, pr);
    asm volatile("cp.async.wait_all;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    // D
    auto leave = [&](int q, unsigned run, long long g) {
      const unsigned from = run & 0xFFFFu, h = run >> 16;
      if (!h) return;
      if (g + (long long)h > __ldg(A.end + q)) {  // region sized too small: reported, the run is dropped
        atomicOr(A.counters + 5, 1u);
        return;
      }
      bulk_s2g(A.recs + g * S.words, sstage + from * (8u * S.words), h * (8u * S.words));
    };
    if (EARLY > 1) {
#pragma unroll
      for (int j = 0; j < EARLY; ++j) {
        const int q = threadIdx.x + j * NT;
        if (q < A.nparts) leave(q, hist[q], g[j]);
      }
    } else {
      for (int qa = threadIdx.x; qa < A.nparts; qa += 8 * NT) {
        long long g8[8];
        unsigned run[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          run[j] = qa + j * NT < A.nparts ? hist[qa + j * NT] : 0u;
          g8[j] = reserve(qa + j * NT, run[j] >> 16);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) leave(qa + j * NT, run[j], g8[j]);
      }
    }
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    unsigned int* const used = hist;
    hist = next_hist;
    next_hist = used;
  }
  asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

// ---- pass 2 -----------------------------------------------------------------
// Lanes of a warp that share a slot, chained from each lane to the next higher
// one of its group: five steps of pointer doubling fold any mix of groups at
// once, and the lowest lane of each group ends with the group's result.
struct LaneChain {
  unsigned next;   // 5 bits per step: source lane
  unsigned has;    // 1 bit per step: a source exists
  int steps;       // warp-uniform: steps that cover the largest group
};
__device__ __forceinline__ LaneChain lane_chain(unsigned peers, int largest)
{
  LaneChain L;
  const int lane = threadIdx.x & 31;
  const unsigned above = peers & (0xFFFFFFFEu << lane);
  unsigned has = above != 0;
  unsigned nx = has ? (unsigned)(__ffs(above) - 1) : (unsigned)lane;
  L.next = nx;
  L.has = has;
  L.steps = 32 - __clz(largest - 1);
#pragma unroll
  for (int s = 1; s < 5; ++s) {
    if (s >= L.steps) break;
    const unsigned n2 = __shfl_sync(0xFFFFFFFFu, nx, nx);
    const unsigned h2 = __shfl_sync(0xFFFFFFFFu, has, nx);
    has = has & h2;
    nx = has ? n2 : (unsigned)lane;
    L.next |= nx << (5 * s);
    L.has |= has << s;
  }
  return L;
}
template <typename T, typename F>
__device__ __forceinline__ T chain_fold(const LaneChain& L, T v, F op)
{
#pragma unroll 1
  for (int s = 0; s < L.steps; ++s) {
    const T o = __shfl_sync(0xFFFFFFFFu, v, (L.next >> (5 * s)) & 31u);
    if ((L.has >> s) & 1u) v = op(v, o);
  }
  return v;
}

// One column's elements `x` (right-aligned bits) of R rows into their slots
// `sa`.  Rows with up[r] = false update nothing.  With FOLD (R = 1) the
// element of every lane of a group is folded first, up[0] marks the groups'
// lowest lanes, and a lane without a valid element (ok = false) brings the
// identity.  64-bit and floating shared reductions are compare-and-swap loops
// on this architecture; MIN/MAX read the field first and skip the reduction
// when the value cannot improve it.
template <bool FOLD, int R>
__device__ __forceinline__ void rec_update(const RecCol& c, const uint32_t (&sa)[R], const uint64_t (&x)[R],
                                           const bool (&ok)[R], const bool (&up)[R], const LaneChain& L)
{
  const int so = c.sum(), mo = c.min(), xo = c.max(), qo = c.sq();
  auto add = [](auto a, auto b) { return a + b; };
  auto lower = [](auto a, auto b) { return a < b ? a : b; };
  auto higher = [](auto a, auto b) { return a > b ? a : b; };
  // MIN and MAX of one type: the fields of all rows read before the reductions
  auto min_max = [&](auto (&lo)[R], auto (&hi)[R], auto read, auto red_min, auto red_max) {
    using T = std::remove_reference_t<decltype(lo[0])>;
    T cur[R];
    if (mo >= 0) {
      if (FOLD) lo[0] = chain_fold(L, ok[0] ? lo[0] : (T)~(T)0, lower);
#pragma unroll
      for (int r = 0; r < R; ++r) cur[r] = up[r] ? read(sa[r] + mo) : (T)0;
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (lo[r] < cur[r]) red_min(sa[r] + mo, lo[r]);
    }
    if (xo >= 0) {
      if (FOLD) hi[0] = chain_fold(L, ok[0] ? hi[0] : (T)0, higher);
#pragma unroll
      for (int r = 0; r < R; ++r) cur[r] = up[r] ? read(sa[r] + xo) : (T)~(T)0;
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (hi[r] > cur[r]) red_max(sa[r] + xo, hi[r]);
    }
  };
  auto min_max64 = [&](uint64_t (&lo)[R], uint64_t (&hi)[R]) {
    min_max(lo, hi, [](uint32_t a) { return sld_u64(a); }, [](uint32_t a, uint64_t v) { sred_min_u64(a, v); },
            [](uint32_t a, uint64_t v) { sred_max_u64(a, v); });
  };
  auto min_max32 = [&](uint32_t (&lo)[R], uint32_t (&hi)[R]) {
    min_max(lo, hi, [](uint32_t a) { return sld_u32(a); }, [](uint32_t a, uint32_t v) { sred_min_u32(a, v); },
            [](uint32_t a, uint32_t v) { sred_max_u32(a, v); });
  };
  // a sum of one type
  auto sum = [&](int off, auto value, auto red) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      auto t = value(r);
      if (FOLD) t = chain_fold(L, ok[r] ? t : (decltype(t))0, add);
      if (up[r]) red(sa[r] + off, t);
    }
  };
  switch (c.kind()) {
    case RK_F64: {
      auto d = [&](int r) { return __longlong_as_double((long long)x[r]); };
      if (so >= 0) sum(so, d, [](uint32_t a, double v) { sred_add_f64(a, v); });
      if (mo >= 0 || xo >= 0) {
        uint64_t lo[R], hi[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
          // as ord64_f: NaN just above +inf for MIN, just below -inf for MAX
          const bool nan = (x[r] << 1) > 0xFFE0000000000000ull;
          const uint64_t o = (int64_t)x[r] < 0 ? ~x[r] : (x[r] | 0x8000000000000000ull);
          lo[r] = nan ? 0xFFF8000000000000ull : o;
          hi[r] = nan ? 0x0007FFFFFFFFFFFFull : o;
        }
        min_max64(lo, hi);
      }
      if (qo >= 0) sum(qo, [&](int r) { return d(r) * d(r); }, [](uint32_t a, double v) { sred_add_f64(a, v); });
      break;
    }
    case RK_F32: {
      auto f = [&](int r) { return __uint_as_float((uint32_t)x[r]); };
      auto d = [&](int r) { return (double)f(r); };
      if (so >= 0) sum(so, d, [](uint32_t a, double v) { sred_add_f64(a, v); });
      if (mo >= 0 || xo >= 0) {
        uint32_t lo[R], hi[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
          lo[r] = ord32_f(f(r), true);
          hi[r] = ord32_f(f(r), false);
        }
        min_max32(lo, hi);
      }
      if (qo >= 0) sum(qo, [&](int r) { return d(r) * d(r); }, [](uint32_t a, double v) { sred_add_f64(a, v); });
      break;
    }
    case RK_W64: {
      if (so >= 0) sum(so, [&](int r) { return x[r]; }, [](uint32_t a, uint64_t v) { sred_add_u64(a, v); });
      if (mo >= 0 || xo >= 0) {
        const uint64_t flip = (c.flags() & RF_SIGNED) ? 0x8000000000000000ull : 0ull;
        uint64_t lo[R], hi[R];
#pragma unroll
        for (int r = 0; r < R; ++r) lo[r] = hi[r] = x[r] ^ flip;
        min_max64(lo, hi);
      }
      if (qo >= 0) sum(qo, [&](int r) { return x[r] * x[r]; }, [](uint32_t a, uint64_t v) { sred_add_u64(a, v); });
      break;
    }
    case RK_NONE: break;
    default: {
      // integers of at most 32 bits, extended to 64; MIN/MAX in the
      // order-preserving unsigned encoding of 32 bits
      uint64_t iv[R];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const uint32_t raw = (uint32_t)x[r] << c.ext();
        iv[r] = c.kind() == RK_S32 ? (uint64_t)(int64_t)((int32_t)raw >> c.ext()) : (uint64_t)(raw >> c.ext());
        if (c.flags() & RF_BOOL) iv[r] = iv[r] != 0;
      }
      if (so >= 0) {
        auto v = [&](int r) { return iv[r]; };
        if (c.flags() & RF_SUM32) sum(so, v, [](uint32_t a, uint64_t t) { sred_add_u32(a, (uint32_t)t); });
        else sum(so, v, [](uint32_t a, uint64_t t) { sred_add_u64(a, t); });
      }
      if (mo >= 0 || xo >= 0) {
        const uint32_t flip = c.kind() == RK_S32 ? 0x80000000u : 0u;
        uint32_t lo[R], hi[R];
#pragma unroll
        for (int r = 0; r < R; ++r) lo[r] = hi[r] = (uint32_t)iv[r] ^ flip;
        min_max32(lo, hi);
      }
      if (qo >= 0) sum(qo, [&](int r) { return iv[r] * iv[r]; }, [](uint32_t a, uint64_t v) { sred_add_u64(a, v); });
      break;
    }
  }
}

// ---- the shared table of pass 2 ---------------------------------------------
// `scap` slots (a multiple of four) in buckets of four, with one 32-bit tag
// per slot: a lookup reads a bucket's four tags in one 16-byte load and then
// only the key of the slot whose tag matches.  A bucket that is full sends the
// search to the next one.  Tags only point the way: a slot is claimed by
// compare-and-swap on its key, its tag is written afterwards, and a lookup that
// sees an unset tag walks the keys themselves.  Against probing the keys two at
// a time this keeps its speed at 70% fill, which is what allows fewer, fuller
// partitions and so longer runs in pass 1.
struct RecTable {
  uint32_t tags, slots;  // shared-window addresses
  uint32_t nb;           // buckets
  int stride, sfill;
  uint32_t used;         // shared-window address of the claimed-slot count
};
__device__ __forceinline__ uint32_t rec_tag(uint64_t h) { return (uint32_t)(h >> 18) | 1u; }
__device__ __forceinline__ ulonglong2 sld_u64x2(uint32_t a)
{
  ulonglong2 v;
  asm volatile("ld.volatile.shared.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "r"(a) : "memory");
  return v;
}

// Claims the empty slot i (address s) for a key: 1 it holds the key now, 0
// another key took it, -1 the table is at its fill limit.
template <int KW>
__device__ __forceinline__ int rec_claim(const RecTable& t, uint32_t i, uint32_t s, uint32_t tag, uint64_t w0, uint64_t w1)
{
  if (sld_u32(t.used) >= (unsigned)t.sfill) return -1;
  bool claimed, mine;
  if constexpr (KW == 1) {
    uint64_t old;
    asm volatile("atom.shared.cas.b64 %0, [%1], %2, %3;" : "=l"(old) : "r"(s), "l"(kEmpty), "l"(w0) : "memory");
    claimed = old == kEmpty;
    mine = old == w0;
  } else {
    unsigned __int128* kp = (unsigned __int128*)__cvta_shared_to_generic(s);
    const unsigned __int128 want = ((unsigned __int128)w1 << 64) | w0;
    const unsigned __int128 old = atomicCAS(kp, ~(unsigned __int128)0, want);
    claimed = old == ~(unsigned __int128)0;
    mine = old == want;
  }
  if (claimed) {
    sred_add_u32(t.used, 1u);
    asm volatile("st.volatile.shared.u32 [%0], %1;" ::"r"(t.tags + 4 * i), "r"(tag) : "memory");
  }
  return claimed || mine;
}

// The authoritative walk over the keys from the home bucket on; 0 when the
// table is at its fill limit.
template <int KW>
__device__ __forceinline__ uint32_t rec_slot_walk(const RecTable& t, uint32_t bucket, uint32_t tag, uint64_t w0,
                                                  uint64_t w1)
{
  uint32_t i = 4 * bucket;
  const uint32_t scap = 4 * t.nb;
#pragma unroll 1
  for (uint32_t p = 0; p < scap; ++p) {
    const uint32_t s = t.slots + i * t.stride;
    bool mine, empty;
    // two-word keys: an empty slot has the top bit of its second word set
    // (never set in a packed key); a first word of all ones is a valid key and
    // is matched through the compare-and-swap
    if constexpr (KW == 1) {
      const uint64_t c = sld_u64(s);
      mine = c == w0;
      empty = c == kEmpty;
    } else {
      const ulonglong2 c = sld_u64x2(s);
      mine = c.x == w0 && c.y == w1 && w0 != kEmpty;
      empty = (c.y >> 63) || c.x == kEmpty;
    }
    if (mine) return s;
    if (empty) {
      const int r = rec_claim<KW>(t, i, s, tag, w0, w1);
      if (r > 0) return s;
      if (r < 0) return 0;
    }
    i = i + 1 == scap ? 0 : i + 1;
  }
  return 0;
}

template <int KW>
__device__ __forceinline__ uint32_t rec_slot(const RecTable& t, uint64_t w0, uint64_t w1, uint64_t h)
{
  const uint32_t home = (uint32_t)(((uint64_t)(uint32_t)h * t.nb) >> 32);
  const uint32_t tag = rec_tag(h);
  uint32_t b = home;
#pragma unroll 1
  for (uint32_t p = 0; p < t.nb; ++p) {
    uint4 g;
    asm volatile("ld.volatile.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(g.x), "=r"(g.y), "=r"(g.z), "=r"(g.w)
                 : "r"(t.tags + 16 * b));
    const int m = g.x == tag ? 0 : g.y == tag ? 1 : g.z == tag ? 2 : g.w == tag ? 3 : -1;
    const int z = g.x == 0 ? 0 : g.y == 0 ? 1 : g.z == 0 ? 2 : g.w == 0 ? 3 : -1;
    const uint32_t i = 4 * b + (m >= 0 ? m : z);
    const uint32_t s = t.slots + i * t.stride;
    if (m >= 0) {
      if constexpr (KW == 1) {
        if (sld_u64(s) == w0) return s;
      } else {
        const ulonglong2 c = sld_u64x2(s);
        if (c.x == w0 && c.y == w1) return s;
      }
      break;  // another key with this tag: settle it by the keys
    }
    if (z >= 0) {
      // every slot of the sequence before this one holds another key, so the
      // key is here, is claimed here, or (the slot taken meanwhile) is settled
      // by the keys
      const int r = rec_claim<KW>(t, i, s, tag, w0, w1);
      if (r > 0) return s;
      if (r < 0) return 0;
      break;
    }
    b = b + 1 == t.nb ? 0 : b + 1;
  }
  return rec_slot_walk<KW>(t, home, tag, w0, w1);
}

// Rows of one slot inside a warp from which folding them first is cheaper than
// letting their updates queue on the slot.
constexpr int kFoldFrom = 4;

// The columns of R rows per thread into their slots sa (0: no row).  Column j's
// bits come out of the front word of `rec`, which moves up by the words its
// descriptor names; validity bits in vb.  One copy of the per-kind update code
// is looped over the columns (an unrolled copy per column does not fit the
// instruction cache), so its dispatch is paid once per R rows.  With FOLD, a
// warp in which a slot occurs kFoldFrom times or more folds the rows of one
// slot before their updates.  Every lane of a warp calls it.
//
// With MORE, `rec` holds a record's first RW words only: after `left` words have
// gone by the next RW are loaded from `more` (rows with sa = 0 load nothing).
template <int R, int RW, bool FOLD, bool MORE = false>
__device__ __forceinline__ void apply_columns(const RecSpec& S, int nc, int rows_off, const uint32_t (&sa)[R],
                                              const unsigned (&vb)[R], uint64_t (&rec)[R][RW],
                                              const uint64_t* more = nullptr, int left = 0)
{
  static_assert(!MORE || R == 1, "wide records go one row at a time");
  const int lane = threadIdx.x & 31;
  // the front word goes by
  auto next_word = [&](uint64_t (&w)[RW], uint32_t slot) {
    if (MORE && --left == 0) {
      left = RW;
      if (slot) rec_load<RW>(more, w);
      more += RW;
      return;
    }
#pragma unroll
    for (int q = 0; q + 1 < RW; ++q) w[q] = w[q + 1];
  };
  LaneChain L{0, 0, 0};
  if constexpr (FOLD) {
    bool fold = false;  // a slot occurs often enough in the warp to fold its rows first
    int most[R];
    unsigned peers[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      peers[r] = __match_any_sync(0xFFFFFFFFu, sa[r] ? sa[r] : (0x80000000u | (unsigned)lane));
      most[r] = (int)__reduce_max_sync(0xFFFFFFFFu, (unsigned)__popc(peers[r]));
      fold = fold || most[r] >= kFoldFrom;
    }
    if (fold) {
      // one row of the thread at a time
#pragma unroll
      for (int r = 0; r < R; ++r) {
        L = lane_chain(peers[r], most[r]);
        const bool lead[1] = {sa[r] != 0 && lane == __ffs(peers[r]) - 1};
        const uint32_t at[1] = {sa[r]};
        if (lead[0]) sred_add_u32(sa[r] + rows_off, __popc(peers[r]));
#pragma unroll 1
        for (int j = 0; j < nc; ++j) {
          const RecCol c = S.col[j];
          for (int a = 0; a < c.adv(); ++a) next_word(rec[r], sa[r]);
          const bool valid = (vb[r] >> c.bit()) & 1;
          if (c.nulls() >= 0) {
            const unsigned ng = peers[r] & __ballot_sync(0xFFFFFFFFu, sa[r] != 0 && !valid);
            if (lead[0] && ng) sred_add_u32(sa[r] + c.nulls(), __popc(ng));
          }
          const uint64_t x[1] = {rec[r][0] >> c.shift()};
          const bool ok[1] = {sa[r] != 0 && valid};
          rec_update<true, 1>(c, at, x, ok, lead, L);
        }
      }
      return;
    }
  }
#pragma unroll
  for (int r = 0; r < R; ++r)
    if (sa[r]) sred_add_u32(sa[r] + rows_off, 1u);
#pragma unroll 1
  for (int j = 0; j < nc; ++j) {
    const RecCol c = S.col[j];
    for (int a = 0; a < c.adv(); ++a) {
#pragma unroll
      for (int r = 0; r < R; ++r) next_word(rec[r], sa[r]);
    }
    uint64_t x[R];
    bool ok[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const bool valid = (vb[r] >> c.bit()) & 1;
      ok[r] = sa[r] != 0 && valid;
      x[r] = rec[r][0] >> c.shift();
      if (c.nulls() >= 0 && sa[r] != 0 && !valid) sred_add_u32(sa[r] + c.nulls(), 1u);
    }
    rec_update<false, R>(c, sa, x, ok, ok, L);
  }
}

// Pass 2.  One CTA owns a work item at a time and aggregates its records in a
// shared table of `scap` slots (plus the all-ones key's).  Every thread takes
// R records per step (a warp 32 R consecutive ones), the records two steps
// ahead being on their way into L2.
template <int KW, int RW, bool WAGG>
__global__ void __launch_bounds__(1024, 1) k_rec_aggregate(const __grid_constant__ Plan P,
                                                           const __grid_constant__ RecArgs A,
                                                           const __grid_constant__ RecSpec S, TableRef G, EmitRef D,
                                                           const __grid_constant__ OutPtrs O, int scap, int sfill,
                                                           const __grid_constant__ SlotTemplate tmpl)
{
  constexpr int NT = 1024;
  constexpr int R = RW <= 4 && !WAGG ? 2 : 1;
  // words of a record held at a time.  A whole 96-byte record in registers, moved
  // up a word per column, spilled 248 bytes a thread and cost 2.30 ms for 20M
  // rows of eight sums in 4M groups; by fours it takes 1.40 (by sixes 1.53).
  constexpr int HW = RW > 8 ? 4 : RW;
  constexpr int64_t STEP = R * NT;
  extern __shared__ __align__(16) uint8_t smem[];
  using ScanT = cub::BlockScan<unsigned, NT>;
  __shared__ typename ScanT::TempStorage scan_tmp;
  __shared__ int s_part;
  __shared__ unsigned int s_used, s_spill, s_new, s_base;
  __shared__ unsigned int s_cnt[NT / 2];  // (16 rounds of NT slots, each at least 24 bytes, fill shared memory) x 32 warps
  if (threadIdx.x == 0) s_new = 0;
  const int stride = G.stride;
  const int nw = stride / 8;
  uint8_t* slots = smem + (size_t)scap * 4;
  const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(smem);
  const RecTable table{sbase, sbase + 4 * (uint32_t)scap, (uint32_t)scap / 4, stride, sfill,
                       (uint32_t)__cvta_generic_to_shared(&s_used)};
  const int nc = S.ncols;
  const int rows_off = P.rows_off;
  const int lane = threadIdx.x & 31;
  for (;;) {
    for (int i = threadIdx.x; i < scap / 4; i += NT) ((uint4*)smem)[i] = make_uint4(0, 0, 0, 0);
    const int it = p2_claim<NT>(A.work, slots, scap + (KW == 1), nw, tmpl, &s_part, &s_used, &s_spill);
    if (it >= A.nitems) break;
    const PartItem item = A.items[it];
    const int64_t e = min(item.end, min((int64_t)A.cursor[item.part], A.end[item.part]));
    // a warp's rows are consecutive: warps without rows left leave together
    for (int64_t w0 = item.begin + (threadIdx.x >> 5) * (32 * R); w0 < e; w0 += STEP) {
      const int64_t row = w0 + lane;
      if (lane == 0 && w0 + 2 * STEP + 32 * R <= e)
        bulk_prefetch_l2(A.recs + (w0 + 2 * STEP) * RW, 32 * R * RW * 8);
      uint64_t rec[R][HW];
      uint32_t sa[R];
      unsigned vb[R];
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (row + 32 * r < e) rec_load<HW>(A.recs + (row + 32 * r) * RW, rec[r]);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        sa[r] = 0;
        vb[r] = 0xFFu;
        if (HW == RW && S.has_bits) vb[r] = (unsigned)(rec[r][HW - 1] >> 56);
        if (row + 32 * r < e) {
          if (HW < RW && S.has_bits) vb[r] = __ldg((const uint8_t*)(A.recs + (row + 32 * r + 1) * RW) - 1);
          const uint64_t k0 = KW == 1 ? rec[r][0] & S.keymask : rec[r][0];
          const uint64_t k1 = KW == 2 ? rec[r][1] : 0;
          sa[r] = (KW == 1 && k0 == kEmpty) ? table.slots + scap * stride
                                            : rec_slot<KW>(table, k0, k1, hash_key(k0, k1, KW));
          if (sa[r] == 0) {
            // listed for the global table; one list reservation per group of lanes
            s_spill = 1;
            const unsigned mates = __activemask();
            const int leader = __ffs(mates) - 1;
            unsigned at = 0;
            if (lane == leader) at = atomicAdd(A.counters + 12, (unsigned)__popc(mates));
            at = __shfl_sync(mates, at, leader) + __popc(mates & ((1u << lane) - 1));
            if (at < A.spill_cap) A.spill_rows[at] = row + 32 * r;
            else atomicOr(A.counters + 13, 1u);
          }
        }
        // a two-word key's second word is the front word of the first column
        if constexpr (KW == 2) {
#pragma unroll
          for (int j = 0; j + 1 < HW; ++j) rec[r][j] = rec[r][j + 1];
        }
      }
      __syncwarp();
      apply_columns<R, HW, WAGG, (HW < RW)>(S, nc, rows_off, sa, vb, rec, A.recs + row * RW + HW, HW - (KW - 1));
    }
    __syncthreads();
    p2_flush<NT, ScanT>(P, G, D, O, slots, scap, s_spill != 0 || item.merge, scan_tmp, s_cnt, &s_base, &s_new);
    __syncthreads();
  }
  if (threadIdx.x == 0 && s_new) atomicAdd(G.counters, s_new);
}

// Records whose key did not fit their partition's shared table (a partition
// with more groups than expected) are listed by pass 2 and applied to the
// global spill table here, so the hot loop carries no call into the generic
// update code.
static __global__ void __launch_bounds__(256) k_rec_spill(const __grid_constant__ Plan P, TableRef G,
                                                          const __grid_constant__ RecArgs A,
                                                          const __grid_constant__ RecSpec S)
{
  __shared__ unsigned int s_new;
  if (threadIdx.x == 0) s_new = 0;
  __syncthreads();
  const unsigned cnt = min(*(volatile unsigned int*)(A.counters + 12), A.spill_cap);
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < cnt; i += gridDim.x * blockDim.x) {
    const uint64_t* rec = A.recs + A.spill_rows[i] * (int64_t)S.words;
    const uint64_t w0 = P.key_words == 1 ? rec[0] & S.keymask : rec[0];
    const uint64_t w1 = P.key_words == 2 ? rec[1] : 0;
    const unsigned vb = S.has_bits ? (unsigned)(rec[S.words - 1] >> 56) : 0xFFu;
    const uint64_t h = hash_key(w0, w1, P.key_words);
    const int64_t gi = global_slot(P, G, w0, w1, h, &s_new);
    if (gi < 0) {
      atomicOr(G.counters + 1, 1u);
      continue;
    }
    uint8_t* slot = G.T + gi * (int64_t)G.stride;
    atomicAdd((unsigned int*)(slot + P.rows_off), 1u);
#pragma unroll 1
    for (int j = 0; j < S.ncols; ++j) {
      ValCol c = P.vals[S.src_col[j]];
      if (!((vb >> S.col[j].bit()) & 1)) {
        if (c.nulls_off >= 0) atomicAdd((unsigned int*)(slot + c.nulls_off), 1u);
        continue;
      }
      if (c.acc_begin == c.acc_end) continue;
      c.data = (const uint8_t*)rec + S.off[j];
      const Elem el = load_elem(c, 0);
      apply_elem(P, c, c.acc_begin, c.acc_end, slot, el, 0);
    }
  }
  __syncthreads();
  if (threadIdx.x == 0 && s_new) atomicAdd(G.counters, s_new);
}

}  // namespace gb
