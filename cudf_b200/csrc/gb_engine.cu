// gb_engine.cu -- host orchestration of the hash groupby: planning, table
// sizing from a key sample, launches, overflow retry and compaction.
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <set>
#include <string>
#include <tuple>
#include <vector>

#include "gb_engine.h"
#include "gb_kernels.cuh"
#include "gb_partition.cuh"
#include "gb_record.h"
#include "gb_stage.h"

namespace gb {

// ---------------------------------------------------------------------------
// type system (cpp/include/cudf/detail/aggregation/aggregation.hpp:1168-1290)
int type_width(int t)
{
  switch (t) {
    case T_INT8: case T_UINT8: case T_BOOL8: return 1;
    case T_INT16: case T_UINT16: return 2;
    case T_INT32: case T_UINT32: case T_FLOAT32: case T_TS_D: case T_DUR_D: return 4;
    case T_INT64: case T_UINT64: case T_FLOAT64: case T_TS_S: case T_TS_MS: case T_TS_US:
    case T_TS_NS: case T_DUR_S: case T_DUR_MS: case T_DUR_US: case T_DUR_NS: return 8;
    default: return 0;
  }
}
static bool is_ts(int t) { return t >= T_TS_D && t <= T_TS_NS; }
static bool is_dur(int t) { return t >= T_DUR_D && t <= T_DUR_NS; }
static uint8_t type_cat(int t)
{
  if (t == T_FLOAT32) return CAT_F32;
  if (t == T_FLOAT64) return CAT_F64;
  if (t == T_BOOL8) return CAT_BOOL;
  if (t >= T_UINT8 && t <= T_UINT64) return CAT_UNSIGNED;
  return CAT_SIGNED;
}

bool valid_agg(int t, int k)
{
  if (type_width(t) == 0) return false;
  bool numeric = !is_ts(t) && !is_dur(t);
  switch (k) {
    case K_MIN: case K_MAX: case K_COUNT_VALID: case K_COUNT_ALL: case K_ARGMIN: case K_ARGMAX: return true;
    case K_SUM: case K_MEAN: return numeric || is_dur(t);
    case K_PRODUCT: case K_SUM_OF_SQUARES: case K_VARIANCE: case K_STD: return numeric;
    default: return false;
  }
}

int target_type(int t, int k)
{
  switch (k) {
    case K_COUNT_VALID: case K_COUNT_ALL: case K_ARGMIN: case K_ARGMAX: return T_INT32;
    case K_MIN: case K_MAX: return t;
    case K_VARIANCE: case K_STD: return T_FLOAT64;
    case K_MEAN: return is_dur(t) ? t : T_FLOAT64;
    case K_SUM: case K_PRODUCT: case K_SUM_OF_SQUARES:
      return (t == T_FLOAT32 || t == T_FLOAT64 || is_dur(t)) ? t : T_INT64;
    default: return T_EMPTY;
  }
}

// ---------------------------------------------------------------------------
static void ck(cudaError_t e, const char* what)
{
  if (e == cudaSuccess) return;
  cudaGetLastError();
  throw Error(e == cudaErrorMemoryAllocation ? ERR_ALLOC : ERR_CUDA,
              std::string(what) + ": " + cudaGetErrorString(e));
}

// Blocks below this come from a pool of their own.
constexpr size_t kSmallBlock = size_t(1) << 20;

// The device's pool for small blocks (its default pool is the other one),
// made on first use.  Both keep freed blocks, so that repeated calls allocate
// in O(1); the small one at most 64 MB across a synchronisation.
static cudaMemPool_t small_pool()
{
  static std::mutex mu;
  static std::map<int, cudaMemPool_t> pools;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return nullptr;
  std::lock_guard<std::mutex> g(mu);
  auto it = pools.find(dev);
  if (it != pools.end()) return it->second;
  cudaMemPool_t pool;
  uint64_t keep = UINT64_MAX;
  if (cudaDeviceGetDefaultMemPool(&pool, dev) == cudaSuccess)
    cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
  cudaMemPoolProps props;
  std::memset(&props, 0, sizeof(props));
  props.allocType = cudaMemAllocationTypePinned;
  props.location.type = cudaMemLocationTypeDevice;
  props.location.id = dev;
  keep = 64 << 20;
  if (cudaMemPoolCreate(&pool, &props) == cudaSuccess) {
    cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
  } else {
    cudaGetLastError();
    pool = nullptr;  // then the default pool serves every size
  }
  return pools[dev] = pool;
}

// The pool places a block in the smallest free range that holds it.  With one
// pool for all sizes a call's first 168 KB of counters took the front of the
// result block that the caller had just freed; the next result block, of the
// same size, then fitted no range, and the pool remapped freed pages under new
// addresses for it on every call: 0.8 ms for the 188 MB of 1M groups with 15
// aggregations, 3.9 ms for 728 MB, in some calls 20 to 50 ms on a shared host.
// Apart, equal calls find the ranges they left.
static void* default_alloc(void*, size_t bytes, void* stream)
{
  void* p = nullptr;
  if (bytes == 0) bytes = 16;
  cudaMemPool_t small = small_pool();
  cudaError_t e = small && bytes < kSmallBlock ? cudaMallocFromPoolAsync(&p, bytes, small, (cudaStream_t)stream)
                                               : cudaMallocAsync(&p, bytes, (cudaStream_t)stream);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  return p;
}
static void default_free(void*, void* p, size_t, void* stream)
{
  if (p) cudaFreeAsync(p, (cudaStream_t)stream);
}
Allocator default_allocator() { return Allocator{default_alloc, default_free, nullptr}; }

// Scratch buffers of one call, returned to the allocator on scope exit.
struct Scratch {
  Allocator A;
  cudaStream_t s;
  struct Buf { void* p; size_t n; };
  std::vector<Buf> bufs;
  Scratch(const Allocator& a, cudaStream_t st) : A(a), s(st) {}
  void* get(size_t n)
  {
    void* p = A.allocate(A.ctx, n, (void*)s);
    if (!p) throw Error(ERR_ALLOC, "device allocation of " + std::to_string(n) + " bytes failed");
    bufs.push_back({p, n});
    // kernels read scratch arrays with 16-byte vector loads and bulk copies
    if ((uintptr_t)p & 15) throw Error(ERR_LOGIC, "the allocator returned a block that is not 16-byte aligned");
    return p;
  }
  void put(void* p)
  {
    for (size_t i = 0; i < bufs.size(); ++i)
      if (bufs[i].p == p) {
        A.deallocate(A.ctx, p, bufs[i].n, (void*)s);
        bufs.erase(bufs.begin() + i);
        return;
      }
  }
  void clear()
  {
    for (auto& b : bufs) A.deallocate(A.ctx, b.p, b.n, (void*)s);
    bufs.clear();
  }
  ~Scratch() { clear(); }
};

void Result::release()
{
  auto fr = [&](void* p, size_t n) {
    if (p && alloc.deallocate) alloc.deallocate(alloc.ctx, p, n, (void*)stream);
  };
  if (block) {
    fr(block, block_bytes);
    block = nullptr;
  } else {
    for (auto& c : keys) { fr(c.data, c.data_bytes); fr(c.mask, c.mask_bytes); }
    for (auto& r : results)
      for (auto& c : r) { fr(c.data, c.data_bytes); fr(c.mask, c.mask_bytes); }
  }
  keys.clear();
  results.clear();
}

struct DevInfo {
  int sms = 148;
  int smem_optin = 227 * 1024;
};
static DevInfo dev_info()
{
  static std::mutex mu;
  static DevInfo cache[64];
  static bool have[64] = {};
  int dev = 0;
  ck(cudaGetDevice(&dev), "cudaGetDevice");
  std::lock_guard<std::mutex> g(mu);
  if (dev < 64 && !have[dev]) {
    cudaDeviceGetAttribute(&cache[dev].sms, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&cache[dev].smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    have[dev] = true;
  }
  return cache[dev < 64 ? dev : 0];
}

static uint64_t next_pow2(uint64_t x)
{
  uint64_t p = 1;
  while (p < x) p <<= 1;
  return p;
}

// ---------------------------------------------------------------------------
// planning
void build_plan(const std::vector<Column>& keys, int null_policy, const std::vector<Request>& reqs,
                Plan& P, std::vector<int>& out_types, bool wide_f32)
{
  std::memset(&P, 0, sizeof(P));
  if (keys.empty()) throw Error(ERR_LOGIC, "groupby needs at least one key column");
  if (keys.size() > (size_t)kMaxKeyCols) throw Error(ERR_UNSUPPORTED, "too many key columns");
  int64_t n = keys[0].size;
  for (auto& k : keys) {
    if (k.size != n) throw Error(ERR_LOGIC, "Size mismatch between key columns.");
    if (type_width(k.type_id) == 0) throw Error(ERR_UNSUPPORTED, "unsupported key column type");
  }
  // cpp/src/groupby/groupby.cu:208-212
  for (auto& r : reqs)
    if (r.values.size != n) throw Error(ERR_LOGIC, "Size mismatch between request values and groupby keys.");
  // cpp/src/groupby/groupby.cu:174-190
  for (auto& r : reqs)
    for (auto& a : r.aggs)
      if (!valid_agg(r.values.type_id, a.kind)) throw Error(ERR_LOGIC, "Invalid type/aggregation combination.");
  if (n >= (int64_t)0xFFFFFFF0ll) throw Error(ERR_UNSUPPORTED, "more than 2^32-16 rows in one groupby");

  P.num_rows = n;
  P.include_nulls = null_policy == 1;
  P.num_keys = (int)keys.size();
  // key packing, first-fit decreasing: value bits never straddle a word, null
  // flags (INCLUDE only) are single bits; word 0 holds 64 bits, word 1 at most
  // 63 so that its top bit stays clear (the empty-slot marker of 2-word keys)
  struct Item { int bits, key; bool null_flag; };
  std::vector<Item> items;
  for (int k = 0; k < P.num_keys; ++k) {
    KeyCol& c = P.keys[k];
    c.data = keys[k].data;
    c.mask = keys[k].mask;
    c.offset = keys[k].offset;
    c.type_id = keys[k].type_id;
    c.width = (uint8_t)type_width(c.type_id);
    c.cat = type_cat(c.type_id);
    if (c.mask) P.any_key_nullable = 1;
    items.push_back({8 * c.width, k, false});
    if (c.mask && P.include_nulls) {
      items.push_back({1, k, true});
      c.has_null_bit = 1;
    }
  }
  std::stable_sort(items.begin(), items.end(), [](const Item& a, const Item& b) { return a.bits > b.bits; });
  int used[2] = {0, 0};
  const int room[2] = {64, 63};
  int words = 1;
  for (auto& it : items) {
    int w = 0;
    while (w < 2 && used[w] + it.bits > room[w]) ++w;
    if (w == 2) throw Error(ERR_UNSUPPORTED, "key rows wider than 127 packed bits are not supported");
    KeyCol& c = P.keys[it.key];
    if (it.null_flag) { c.null_word = (uint8_t)w; c.null_shift = (uint8_t)used[w]; }
    else { c.word = (uint8_t)w; c.shift = (uint8_t)used[w]; }
    used[w] += it.bits;
    words = std::max(words, w + 1);
  }
  P.key_words = words;

  // value columns: one entry per distinct (column view, ddof of VAR/STD)
  struct VKey { Column c; int ddof; };
  std::vector<VKey> vk;
  std::vector<std::vector<int>> need(0);
  auto find_col = [&](const Column& c, int ddof) {
    for (size_t i = 0; i < vk.size(); ++i)
      if (vk[i].c.data == c.data && vk[i].c.mask == c.mask && vk[i].c.offset == c.offset &&
          vk[i].c.type_id == c.type_id && vk[i].ddof == ddof)
        return (int)i;
    vk.push_back({c, ddof});
    return (int)vk.size() - 1;
  };
  // per request/agg: column index
  std::vector<std::vector<int>> colof(reqs.size());
  for (size_t r = 0; r < reqs.size(); ++r)
    for (auto& a : reqs[r].aggs) {
      bool var = a.kind == K_VARIANCE || a.kind == K_STD;
      colof[r].push_back(find_col(reqs[r].values, var ? a.ddof : -1));
    }
  if (vk.size() > (size_t)kMaxValCols) throw Error(ERR_UNSUPPORTED, "too many distinct value columns");
  P.num_vals = (int)vk.size();

  // which accumulator ops each column needs
  const uint8_t sq_f32 = wide_f32 ? OP_SQ_F64 : OP_SQ_F32;
  std::vector<std::vector<uint8_t>> ops(vk.size());
  std::vector<bool> need_nulls(vk.size(), false), need_m2(vk.size(), false);
  auto add = [&](int v, uint8_t op) {
    if (std::find(ops[v].begin(), ops[v].end(), op) == ops[v].end()) ops[v].push_back(op);
  };
  for (size_t r = 0; r < reqs.size(); ++r)
    for (size_t j = 0; j < reqs[r].aggs.size(); ++j) {
      int v = colof[r][j];
      const Column& c = vk[v].c;
      int t = c.type_id, w = type_width(t);
      uint8_t cat = type_cat(t);
      bool fl = cat == CAT_F32 || cat == CAT_F64;
      int k = reqs[r].aggs[j].kind;
      if (c.mask && k != K_COUNT_ALL) need_nulls[v] = true;
      auto sum_op = [&]() -> uint8_t {
        if (cat == CAT_F32) return wide_f32 ? OP_SUM_F64 : OP_SUM_F32;
        if (cat == CAT_F64) return OP_SUM_F64;
        if (is_dur(t) && w == 4) return OP_SUM_I32;
        return OP_SUM_I64;
      };
      switch (k) {
        case K_SUM: case K_MEAN: add(v, sum_op()); break;
        case K_VARIANCE: case K_STD: add(v, sum_op()); need_m2[v] = true; break;
        case K_MIN: add(v, w == 8 ? OP_MIN_U64 : OP_MIN_U32); break;
        case K_MAX: add(v, w == 8 ? OP_MAX_U64 : OP_MAX_U32); break;
        case K_SUM_OF_SQUARES: add(v, cat == CAT_F32 ? sq_f32 : cat == CAT_F64 ? OP_SQ_F64 : OP_SQ_I64); break;
        case K_PRODUCT: add(v, cat == CAT_F32 ? OP_PROD_F32 : cat == CAT_F64 ? OP_PROD_F64 : OP_PROD_I64); break;
        case K_ARGMIN: add(v, w == 8 ? OP_ARGMIN_R64 : OP_ARGMIN_P32); P.has_arg = 1; break;
        case K_ARGMAX: add(v, w == 8 ? OP_ARGMAX_R64 : OP_ARGMAX_P32); P.has_arg = 1; break;
        default: break;
      }
      (void)fl;
    }

  // slot layout: key words | rows u32 | null counters u32 | 4-byte accs | 8-byte accs
  auto op_size = [](uint8_t op) {
    switch (op) {
      case OP_SUM_I32: case OP_SUM_F32: case OP_MIN_U32: case OP_MAX_U32: case OP_SQ_F32:
      case OP_PROD_F32: return 4;
      default: return 8;
    }
  };
  int off = 8 * P.key_words;
  P.rows_off = off;
  off += 4;
  for (size_t v = 0; v < vk.size(); ++v) {
    ValCol& c = P.vals[v];
    c.data = vk[v].c.data;
    c.mask = vk[v].c.mask;
    c.offset = vk[v].c.offset;
    c.type_id = vk[v].c.type_id;
    c.width = (uint8_t)type_width(c.type_id);
    c.cat = type_cat(c.type_id);
    c.ddof = vk[v].ddof < 0 ? 1 : vk[v].ddof;
    c.nulls_off = -1;
    c.sum_off = -1;
    c.m2_off = -1;
    c.wide = wide_f32 && c.cat == CAT_F32;
    if (need_nulls[v]) { c.nulls_off = (int16_t)off; off += 4; }
  }
  // accumulators grouped per column, 4-byte ones first within the slot
  std::vector<std::pair<int, int>> acc_off;  // (col, op) -> offset resolved below
  int na = 0;
  for (int pass = 0; pass < 2; ++pass) {
    if (pass == 1) off = (off + 7) & ~7;
    for (size_t v = 0; v < vk.size(); ++v)
      for (uint8_t op : ops[v]) {
        if ((op_size(op) == 4) != (pass == 0)) continue;
        if (na >= kMaxAccs) throw Error(ERR_UNSUPPORTED, "too many aggregations in one call");
        P.accs[na].op = op;
        P.accs[na].col = (uint8_t)v;
        P.accs[na].off = (uint16_t)off;
        off += op_size(op);
        ++na;
      }
  }
  for (size_t v = 0; v < vk.size(); ++v)
    if (need_m2[v]) {
      P.vals[v].m2_off = (int16_t)off;
      off += 8;
      P.need_second_pass = 1;
    }
  P.num_accs = na;
  // stride: an odd multiple of 8 bytes (16 for two-word keys, whose 128-bit
  // CAS needs 16-byte alignment) so that one field of 32 different slots
  // falls into many shared-memory banks
  {
    int unit = P.key_words == 2 ? 16 : 8;
    int q = (off + unit - 1) / unit;
    if ((q & 1) == 0) ++q;
    P.slot_bytes = q * unit;
  }
  if (P.slot_bytes > kMaxSlotBytes) throw Error(ERR_UNSUPPORTED, "too many aggregations in one call");
  // reorder accs by column so each column owns a contiguous range
  std::stable_sort(P.accs, P.accs + na, [](const Acc& a, const Acc& b) { return a.col < b.col; });
  for (size_t v = 0; v < vk.size(); ++v) {
    ValCol& c = P.vals[v];
    c.acc_begin = c.acc_end = 0;
    c.min_off = c.max_off = c.sq_off = -1;
    c.sum_op = 0;
    c.basic = 1;
    bool first = true;
    for (int a = 0; a < na; ++a)
      if (P.accs[a].col == v) {
        if (first) { c.acc_begin = (int16_t)a; first = false; }
        c.acc_end = (int16_t)(a + 1);
        uint8_t op = P.accs[a].op;
        int16_t o = (int16_t)P.accs[a].off;
        if (op == OP_SUM_I64 || op == OP_SUM_I32 || op == OP_SUM_F32 || op == OP_SUM_F64) { c.sum_off = o; c.sum_op = op; }
        else if (op == OP_MIN_U32 || op == OP_MIN_U64) c.min_off = o;
        else if (op == OP_MAX_U32 || op == OP_MAX_U64) c.max_off = o;
        else if (op == OP_SQ_I64 || op == OP_SQ_F32 || op == OP_SQ_F64) c.sq_off = o;
        else c.basic = 0;
      }
  }
  auto acc_for = [&](int v, uint8_t op) -> int16_t {
    for (int a = 0; a < na; ++a)
      if (P.accs[a].col == v && P.accs[a].op == op) return (int16_t)P.accs[a].off;
    return -1;
  };

  // outputs in request order
  out_types.clear();
  int no = 0;
  for (size_t r = 0; r < reqs.size(); ++r)
    for (size_t j = 0; j < reqs[r].aggs.size(); ++j) {
      if (no >= kMaxOutputs) throw Error(ERR_UNSUPPORTED, "too many aggregations in one call");
      int v = colof[r][j];
      const ValCol& c = P.vals[v];
      OutSpec& o = P.outs[no++];
      o.kind = reqs[r].aggs[j].kind;
      o.col = v;
      o.out_type = target_type(c.type_id, o.kind);
      o.out_width = (uint8_t)type_width(o.out_type);
      o.ddof = reqs[r].aggs[j].ddof;
      bool has_nulls = c.mask != nullptr;
      int w = c.width;
      switch (o.kind) {
        case K_COUNT_VALID: case K_COUNT_ALL: o.nullable = 0; o.acc_off = -1; break;
        case K_SUM: case K_MEAN: o.nullable = has_nulls; o.acc_off = c.sum_off; break;
        case K_VARIANCE: case K_STD: o.nullable = 1; o.acc_off = c.m2_off; break;
        case K_MIN: o.nullable = has_nulls; o.acc_off = acc_for(v, w == 8 ? OP_MIN_U64 : OP_MIN_U32); break;
        case K_MAX: o.nullable = has_nulls; o.acc_off = acc_for(v, w == 8 ? OP_MAX_U64 : OP_MAX_U32); break;
        case K_SUM_OF_SQUARES: o.nullable = has_nulls;
          o.acc_off = acc_for(v, c.cat == CAT_F32 ? sq_f32 : c.cat == CAT_F64 ? OP_SQ_F64 : OP_SQ_I64); break;
        case K_PRODUCT: o.nullable = has_nulls;
          o.acc_off = acc_for(v, c.cat == CAT_F32 ? OP_PROD_F32 : c.cat == CAT_F64 ? OP_PROD_F64 : OP_PROD_I64); break;
        case K_ARGMIN: o.nullable = has_nulls; o.acc_off = acc_for(v, w == 8 ? OP_ARGMIN_R64 : OP_ARGMIN_P32); break;
        case K_ARGMAX: o.nullable = has_nulls; o.acc_off = acc_for(v, w == 8 ? OP_ARGMAX_R64 : OP_ARGMAX_P32); break;
        default: break;
      }
      out_types.push_back(o.out_type);
    }
  P.num_outs = no;
}

static void build_template(const Plan& P, SlotTemplate& t)
{
  std::memset(&t, 0, sizeof(t));
  uint8_t* b = (uint8_t*)&t.w[0];
  std::memset(b, 0xFF, 8 * P.key_words);
  for (int a = 0; a < P.num_accs; ++a) {
    uint8_t* p = b + P.accs[a].off;
    switch (P.accs[a].op) {
      case OP_MIN_U32: std::memset(p, 0xFF, 4); break;
      case OP_MIN_U64: case OP_ARGMIN_P32: case OP_ARGMIN_R64: case OP_ARGMAX_R64: std::memset(p, 0xFF, 8); break;
      case OP_PROD_I64: { int64_t one = 1; std::memcpy(p, &one, 8); break; }
      case OP_PROD_F32: { float one = 1.0f; std::memcpy(p, &one, 4); break; }
      case OP_PROD_F64: { double one = 1.0; std::memcpy(p, &one, 8); break; }
      default: break;
    }
  }
}

void allow_max_smem(const void* kernel)
{
  static std::mutex mu;
  static std::set<std::pair<int, const void*>> done;
  int dev = 0;
  ck(cudaGetDevice(&dev), "cudaGetDevice");
  std::lock_guard<std::mutex> lk(mu);
  if (done.count({dev, kernel})) return;
  int optin = 0;
  ck(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev), "smem attr");
  cudaFuncAttributes fa;
  ck(cudaFuncGetAttributes(&fa, kernel), "func attr");
  ck(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - (int)fa.sharedSizeBytes),
     "smem attr");
  done.insert({dev, kernel});
}

// ---------------------------------------------------------------------------
namespace {
thread_local uint32_t* t_pinned = nullptr;
thread_local cudaEvent_t t_ev[6] = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};
cudaEvent_t* events()
{
  if (!t_ev[0])
    for (auto& e : t_ev) ck(cudaEventCreate(&e), "cudaEventCreate");
  return t_ev;
}
// Per-thread pinned host words: [0, 1024) counters read back by the host,
// [1024, 1040) the sample flag, then 2^kHllBits + 2^kBucketBits words of the key
// sketch.
constexpr size_t kPinnedWords = 1024 + 16 + (size_t(1) << kHllBits) + (size_t(1) << kBucketBits);
uint32_t* pinned()
{
  if (!t_pinned) ck(cudaMallocHost((void**)&t_pinned, kPinnedWords * 4), "cudaMallocHost");
  return t_pinned;
}
// Pinned staging of the partitioned path's region table (starts, ends,
// cursors: 3 x 8 bytes for up to kMaxParts partitions), per host thread.  A call
// finishes with a stream synchronisation, so the copy out of it is done before
// the thread's next call writes it again.
thread_local int64_t* t_regions = nullptr;
constexpr size_t kRegionWords = 3 * kMaxParts;
int64_t* pinned_regions()
{
  if (!t_regions) ck(cudaMallocHost((void**)&t_regions, kRegionWords * 8), "cudaMallocHost");
  return t_regions;
}

// HyperLogLog cardinality from 2^kHllBits registers (Flajolet et al. 2007):
// E = alpha_m m^2 / sum 2^-M[j], with linear counting m ln(m/V) while E is
// below 2.5 m and V registers are still zero.  64-bit hashes need no
// large-range correction.
double hll_estimate(const uint32_t* regs, int count)
{
  const double m = (double)count;
  int ranks[64] = {};
  for (int i = 0; i < count; ++i) ++ranks[regs[i] & 63u];
  const int zeros = ranks[0];
  double z = 0;
  for (int r = 63; r >= 0; --r) z += ranks[r] * std::ldexp(1.0, -r);
  const double alpha = 0.7213 / (1.0 + 1.079 / m);
  double e = alpha * m * m / z;
  if (e <= 2.5 * m && zeros > 0) e = m * std::log(m / zeros);
  return e;
}


OutColumn make_out(const Allocator& A, cudaStream_t s, int type_id, int64_t rows, bool nullable)
{
  OutColumn c;
  c.type_id = type_id;
  c.size = rows;
  c.data_bytes = (size_t)std::max<int64_t>(rows, 1) * type_width(type_id);
  c.data = A.allocate(A.ctx, c.data_bytes, (void*)s);
  if (!c.data) throw Error(ERR_ALLOC, "device allocation of an output column failed");
  if (nullable) {
    c.mask_bytes = (size_t)((std::max<int64_t>(rows, 1) + 511) / 512) * 64;
    c.mask = (uint32_t*)A.allocate(A.ctx, c.mask_bytes, (void*)s);
    if (!c.mask) throw Error(ERR_ALLOC, "device allocation of an output mask failed");
    ck(cudaMemsetAsync(c.mask, 0, c.mask_bytes, s), "memset mask");
  }
  return c;
}
}  // namespace

int grid_for(const void* kernel, int block, size_t smem, int bps_cap)
{
  DevInfo d = dev_info();
  // the occupancy of a (kernel, block, shared memory) launch does not change
  // once allow_max_smem has raised the kernel's limit: ask the runtime once
  // per device and launch shape
  static std::mutex mu;
  static std::map<std::tuple<int, const void*, int, size_t>, int> memo;
  int dev = 0;
  ck(cudaGetDevice(&dev), "cudaGetDevice");
  const auto key = std::make_tuple(dev, kernel, block, smem);
  int bps = 0;
  {
    std::lock_guard<std::mutex> lk(mu);
    auto it = memo.find(key);
    if (it != memo.end()) bps = it->second;
  }
  if (bps == 0) {
    ck(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, kernel, block, smem), "occupancy");
    if (bps < 1) bps = 1;
    std::lock_guard<std::mutex> lk(mu);
    memo[key] = bps;
  }
  if (bps < 1) bps = 1;
  if (bps_cap > 0) bps = std::min(bps, bps_cap);
  return d.sms * bps;
}

namespace {
std::mutex g_rules_mu;
std::vector<TuningRule> g_rules;
}  // namespace

void set_tuning_rules(const std::vector<TuningRule>& rules)
{
  std::lock_guard<std::mutex> lk(g_rules_mu);
  g_rules = rules;
}

int apply_tuning_rules(Options& o, int64_t rows, int64_t groups, int key_words, uint32_t* applied)
{
  std::lock_guard<std::mutex> lk(g_rules_mu);
  if (applied) *applied = 0;
  for (size_t i = 0; i < g_rules.size(); ++i) {
    const TuningRule& r = g_rules[i];
    if (rows > r.max_rows || groups > r.max_groups || (r.key_words && r.key_words != key_words)) continue;
    const uint32_t m = r.mask & ~o.set_mask;
    if (applied) *applied = m;
    if (m & OPT_BLOCK) o.block = r.opt.block;
    if (m & OPT_BPS) o.blocks_per_sm = r.opt.blocks_per_sm;
    if (m & OPT_SMEM) o.smem_bytes = r.opt.smem_bytes;
    if (m & OPT_FILL) o.smem_fill = r.opt.smem_fill;
    if (m & OPT_SMEM_MAX) o.smem_max_groups = r.opt.smem_max_groups;
    if (m & OPT_LOAD) o.load_factor = r.opt.load_factor;
    if (m & OPT_MODE) o.force_mode = r.opt.force_mode;
    if (m & OPT_PART_FILL) o.part_fill = r.opt.part_fill;
    if (m & OPT_WAGG) o.wagg_pct = r.opt.wagg_pct;
    return (int)i;
  }
  return -1;
}

namespace {
// What a call that throws leaves behind.
struct CallState {
  bool staged = false;       // copies out of the thread's pinned staging were queued
  bool partitioned = false;  // the partitioned path was entered
};

Result aggregate_call(const std::vector<Column>& keys, int null_policy, const std::vector<Request>& reqs,
                      cudaStream_t stream, const Allocator& alloc, const Options& opt_in, Stats* stats, CallState& state)
{
  Options opt = opt_in;  // tuning rules may adjust it once the group estimate is known
  Plan P;
  std::vector<int> out_types;
  build_plan(keys, null_policy, reqs, P, out_types, true);
  Stats st;
  Result R;
  R.alloc = alloc;
  R.stream = stream;
  const int64_t n = P.num_rows;
  static const bool trace = std::getenv("GB_TRACE") != nullptr;
  auto t0 = std::chrono::steady_clock::now();
  auto mark = [&](const char* what) {
    if (!trace) return;
    auto t = std::chrono::steady_clock::now();
    std::fprintf(stderr, "[gb] %-28s %9.3f ms\n", what, std::chrono::duration<double, std::milli>(t - t0).count());
  };

  // cpp/src/groupby/groupby.cu:216 -- empty input gives empty outputs
  if (n == 0) {
    for (auto& k : keys) R.keys.push_back(make_out(alloc, stream, k.type_id, 0, k.mask != nullptr));
    int j = 0;
    for (auto& r : reqs) {
      std::vector<OutColumn> cols;
      for (size_t a = 0; a < r.aggs.size(); ++a, ++j)
        cols.push_back(make_out(alloc, stream, out_types[j], 0, P.outs[j].nullable));
      R.results.push_back(cols);
    }
    if (stats) *stats = st;
    return R;
  }

  constexpr int kNumBuckets = 1 << kBucketBits;
  Scratch S(alloc, stream);
  mark("begin");
  const bool sketch = opt.groups_hint < 0 && n > 65536;
  // From 8M rows on a sample of 512Ki rows is looked at first: with few groups
  // it is the sketch (60M rows of six groups: 0.31 ms for all of them), else it
  // costs about 16 us ahead of the pass over all rows (0.1 to 0.6 ms).
  constexpr int64_t kSampleFrom = 8 << 20, kSampleChunks = 4096;
  const bool sample = sketch && !opt.full_sketch && n >= kSampleFrom;
  const size_t sketch_bytes = (sketch ? sketch_smem() : 0) * (sample ? 2 : 1) + (sketch ? 64 : 0);
  unsigned int* counters = (unsigned int*)S.get(4096 + sketch_bytes);
  ck(cudaMemsetAsync(counters, 0, 4096 + sketch_bytes, stream), "memset counters");
  mark("counters");
  uint32_t* host = pinned();
  DevInfo dev = dev_info();
  SlotTemplate tmpl;
  build_template(P, tmpl);

  // ---- group-count estimate from a key sample ----
  int64_t est;
  const uint32_t* buckets = nullptr;  // rows per hash bucket, in this thread's pinned memory
  std::vector<uint32_t> flat;         // stand-in without a sketch
  bool exact_buckets = false;  // buckets hold exact row counts (full-pass sketch)
  int64_t nsamp = 0;
  int filled = 0;  // buckets with rows
  bool sampled = false;  // the sketch is a sample's
  bool clustered = false;  // a quarter of the rows or more have the key of the row before them
  bool hot = false;        // a bucket holds a sixteenth of the rows
  if (opt.groups_hint >= 0) {
    est = std::max<int64_t>(1, opt.groups_hint);
  } else if (!sketch) {
    est = n;
  } else {
    // full pass over the keys: exact rows per hash bucket (partition region
    // sizes) and a HyperLogLog estimate of the number of distinct keys
    // [0] flag, [2..3] the sample's runs, [4..5] all rows'; then registers and buckets, then the sample's
    unsigned int* few = counters + 1024;
    unsigned int* hll = few + 16;
    unsigned int* bk = hll + (1 << kHllBits);
    {
      const size_t sm = sketch_smem();
      allow_max_smem((const void*)k_sketch);
      // at least 16Ki rows per CTA: each CTA clears and merges 80 KB of
      // shared counters, which dominates on small inputs
      const int full = grid_for((const void*)k_sketch, 512, sm, 0);
      int grid = (int)std::min<int64_t>(full, (n + 16383) / 16384);
      if (sample) {
        unsigned int* shll = bk + kNumBuckets;
        k_sketch<<<std::min(full, 128), 512, sm, stream>>>(P, shll, shll + (1 << kHllBits), kSampleChunks, nullptr, few + 2);
        k_sketch_few<<<1, 1024, 0, stream>>>(shll, hll, few);
        st.kernels += 2;
      }
      k_sketch<<<grid, 512, sm, stream>>>(P, hll, bk, 0, sample ? few : nullptr, few + 4);
    }
    st.kernels += 1;
    ck(cudaGetLastError(), "sketch launch");
    mark("sketch launched");
    uint32_t* hs = host + 1024 + 16;  // registers then buckets, adjacent on the device too
    ck(cudaMemcpyAsync(hs - 16, few, 64 + sketch_smem(), cudaMemcpyDeviceToHost, stream), "sketch d2h");
    ck(cudaStreamSynchronize(stream), "sketch sync");
    buckets = hs + (size_t(1) << kHllBits);
    sampled = sample && hs[-16] != 0;
    exact_buckets = !sampled;
    const uint32_t* runs = hs - 16 + (sampled ? 2 : 4);
    clustered = runs[0] && 4 * (uint64_t)runs[1] >= runs[0];
    int64_t valid_rows = 0;
    uint32_t top = 0;
    for (int b = 0; b < kNumBuckets; ++b) {
      valid_rows += buckets[b];
      filled += buckets[b] > 0;
      top = std::max(top, buckets[b]);
    }
    hot = (int64_t)top * 16 > valid_rows;
    est = (int64_t)std::llround(hll_estimate(hs, 1 << kHllBits));
    est = std::min<int64_t>(std::max<int64_t>(est, valid_rows > 0 ? 1 : 0), valid_rows);
    est = std::max<int64_t>(est, 1);
    nsamp = valid_rows;
  }
  st.est_groups = est;
  uint32_t rule_fields = 0;
  st.rule = apply_tuning_rules(opt, n, est, P.key_words, &rule_fields);
  mark("estimate");

  // ---- mode ----
  auto smem_cap_for = [&](int budget) {
    int sb = std::min(budget, dev.smem_optin - 4096);
    int c = 0;
    if (sb > 0 && P.slot_bytes <= sb) {
      c = 1;
      while ((int64_t)c * 2 * P.slot_bytes <= sb) c *= 2;
    }
    return c;
  };
  int scap = smem_cap_for(opt.smem_bytes);
  int sfill = std::max(1, (int)(scap * opt.smem_fill));
  // groups that outgrow the configured shared-stage table but fit a larger
  // one (up to ~200 KB at fill 0.7) get the larger one, unless the caller
  // sized the table
  if (!(opt.set_mask & (OPT_SMEM | OPT_FILL))) {
    const int big = smem_cap_for(200 * 1024);
    if (est > sfill && est <= (int64_t)(0.7 * big)) {
      scap = big;
      sfill = std::max(1, (int)(0.7 * big));
    }
  }
  // partitioned pass 2 and the shared stage of its plans (closed-form updates):
  // as many slots as fit ~220 KB (any count, tags beside them), one more for the
  // all-ones key
  const int table_bytes = std::min(220 * 1024, dev.smem_optin - 8192);
  const int scap_rec = std::max(0, table_bytes / (P.slot_bytes + 4) - 1) & ~3;  // with tags
  const int scap2 = std::max(0, table_bytes / P.slot_bytes - 1);
  RecSpec rec;
  bool part_ok = !P.has_arg && P.num_vals <= 8 && scap2 >= 256;
  for (int v = 0; v < P.num_vals; ++v) part_ok = part_ok && P.vals[v].basic;
  for (int a = 0; a < P.num_accs; ++a) {
    uint8_t op = P.accs[a].op;
    if (op >= OP_PROD_I64 && op <= OP_PROD_F64) part_ok = false;
  }
  // From 1M rows on the shared stage takes groups up to the fill that the whole
  // of shared memory stands, where they would otherwise go through partitions or
  // the global table (FLOAT32 sums in 64 bits widen the slots, and would be the
  // first to leave it).  Shared stage / else in ms: six FLOAT32 sums, 1800 groups
  // 1.1M rows 0.21 / 0.54, 2M 0.25 / 0.38, 20M 1.00 / 1.24; two, 4000 groups
  // (78% fill) 2M 0.21 / 0.34, 20M 0.57 / 0.75.  VARIANCE/STD, 3300 groups (64%)
  // 2M 0.23 / 0.24, 20M 0.92 / 0.96, 4000 1.06 / 0.96.  Generic updates (ARGMAX),
  // 2100 groups (52%) 2M 0.23 / 0.24, 20M 1.24 / 1.44; 2500 1.31 / 1.24.
  // With a hot key or in sorted order from 64Ki rows on: those queue on the
  // global table's slots (880K rows, 1700 groups, 70% of them one's: 2.7 ms).
  const bool own_table = !(opt.set_mask & (OPT_SMEM | OPT_FILL));
  const int stage_max = (int)(part_ok ? (P.need_second_pass ? 0.7 : 0.85) * scap_rec : 0.55 * scap2);
  if (own_table && (n >= (1 << 20) || hot || clustered) && est > sfill && est <= stage_max) {
    scap = scap2;
    sfill = std::max(1, stage_max);
  }
  int64_t smem_max = opt.smem_max_groups >= 0 ? opt.smem_max_groups : (int64_t)sfill;
  // partitions: enough for the wanted table fill.  Up to 2048 they are a
  // multiple of the SM count, so that pass 2 ends in whole waves and a tile's
  // runs are no shorter than the tables need; a partition then holds 8 or more
  // of the 2^14 hash buckets, give or take one.  Above that a power of two,
  // whose partitions hold equally many buckets, at most kMaxParts (the scatter
  // keeps 8 B per partition in shared memory, so kAllParts for some of the
  // widest records); beyond 80% of that capacity the shared tables would spill
  // and the global table is faster.  (100M rows, two FLOAT32 sums, 33M groups:
  // 6.2 ms, global table 16.7, 36M over 8192 partitions 8.8; 30M groups of six
  // 8-byte accumulators: 9.5 and 35.)
  int nparts = 0, max_parts = 0;
  const bool may_part = part_ok && opt.partition && (opt.force_mode == 2 || (opt.force_mode < 0 && n >= (1 << 20))) &&
                        record_layout(P, rec);
  if (may_part) {
    max_parts = rec_shape(P.key_words, rec.words, kMaxParts, rec.nmask, dev.smem_optin).threads ? kMaxParts : kAllParts;
    const int64_t sms = dev.sms;
    const int64_t want = std::max<int64_t>(2, (int64_t)std::ceil((double)est / (scap_rec * opt.part_fill)));
    const int64_t tight = (int64_t)std::ceil((double)est / (scap_rec * std::max(opt.part_fill, 0.78)));
    // A partition per 32Ki rows, up to four per SM, keeps partitions whole (a
    // split one's tables all merge into the global table), as long as each
    // still has 128 groups: with fewer, the rows of a warp queue on few slots
    // (20M rows, 400 groups over 148 partitions 2.35 ms, over 2 split ones 0.68).
    const int64_t spread = std::min<int64_t>(4, (n + 32768 * sms - 1) / (32768 * sms)) * sms;
    const int64_t whole = (std::max(want, std::min(spread, est / 128 / sms * sms)) + sms - 1) / sms * sms;
    if (want < sms && est < 128 * sms) nparts = (int)std::max(want, est / 128);
    else if (whole <= 2048) nparts = (int)whole;
    else nparts = (int)std::min<uint64_t>(max_parts, next_pow2((uint64_t)tight));
  }
  const bool part_fits = (double)est <= 0.8 * (double)max_parts * scap_rec;
  // VARIANCE/STD look every group up in the global table in their second pass,
  // so partitions only save updates: worth a copy of the rows from a few million
  // of them on, sooner with several accumulators a row than with one or two, and
  // not where groups have only a few rows.  Global table / partitioned in ms,
  // one accumulator: 1.1M rows, 50K groups 0.19 / 0.24; 4M, 200K 0.35 / 0.36;
  // 8M, 500K 0.67 / 0.58; 8M, 4M 1.31 / 1.49; 40M, 20M 9.1 / 10.0.  Four: 1.1M,
  // 50K 0.27 / 0.28; 2M, 5K 0.31 / 0.42; 2M, 200K 0.36 / 0.35; 2M, 1M 0.61 / 0.69;
  // 4M, 5K 0.47 / 0.43; 4M, 200K 0.54 / 0.46; 8M, 4M 2.96 / 2.51.
  const bool few = est < 128 * (int64_t)dev.sms;  // no partition per SM
  bool part_pays = true;
  if (P.need_second_pass)
    part_pays = P.num_accs > 2 ? n >= 3500000 || (n >= 2000000 && !few && n >= 4 * est)
                               : n >= 6000000 && n >= 5 * est;
  int mode;
  if (opt.force_mode >= 0) mode = opt.force_mode;
  else if (scap >= 64 && est <= smem_max) mode = 1;
  else if (may_part && part_fits && part_pays && est > smem_max) mode = 2;
  else mode = 0;
  if (mode == 1 && scap < 16) mode = 0;
  if (mode == 2 && !may_part) mode = 0;
  if (mode == 2 && !rec_shape(P.key_words, rec.words, nparts, rec.nmask, dev.smem_optin).threads) mode = 0;

  if (sampled && mode != 1) {  // only the shared stage does without every row's count
    Options o2 = opt_in;
    o2.full_sketch = 1;
    S.clear();
    return aggregate_call(keys, null_policy, reqs, stream, alloc, o2, stats, state);
  }

  // region sizes of the partitioned path: exact rows per partition from the
  // full-pass sketch (else the sample's share with slack)
  std::vector<int64_t> pbase, pend, prows;
  std::vector<uint8_t> phot;  // partitions that hold a hot key
  bool long_tail = false;
  if (mode == 2) {
    if (!buckets) {  // no sketch (hint given or small input): uniform regions
      flat.assign(kNumBuckets, 1);
      buckets = flat.data();
      nsamp = kNumBuckets;
    }
    auto first_bucket = [&](int64_t p) { return (p * kNumBuckets + nparts - 1) / nparts; };  // see part_of
    phot.resize(nparts);
    const double mean = (double)nsamp / std::max(1, filled);
    for (int b = 0, over = 0; exact_buckets && b < kNumBuckets; ++b)
      if ((double)buckets[b] > 4 * mean && ++over == 32) long_tail = true;
    pbase.resize(nparts);
    pend.resize(nparts);
    prows.resize(nparts);
    int64_t total = 0, maxload = 0;
    const double samp = (double)nsamp;
    for (int p = 0; p < nparts; ++p) {
      double c = 0;
      uint32_t top = 0;
      for (int64_t b = first_bucket(p); b < first_bucket(p + 1); ++b) {
        c += buckets[b];
        top = std::max(top, buckets[b]);
      }
      // a key with an eighth of the partition's rows (four lanes of a warp)
      // shows as a bucket that far above the usual one
      phot[p] = exact_buckets && (((double)top - mean) * 8 > c || est < 16 * (int64_t)nparts);
      int64_t capp;
      if (exact_buckets) {
        capp = (int64_t)c;
        prows[p] = capp;
      } else {
        int64_t expect = (int64_t)std::ceil((double)n * c / std::max(1.0, samp));
        capp = std::max<int64_t>((int64_t)(1.3 * expect), (int64_t)(1.15 * n / nparts)) + 2048;
        capp = std::min<int64_t>(capp, n);
        prows[p] = expect;
        maxload = std::max<int64_t>(maxload, expect);
      }
      pbase[p] = total;
      total += (capp + 31) & ~31ll;
      pend[p] = total;
    }
    // heavy skew seen only through a sample: one partition could hold far
    // more than its share (exact counts split heavy partitions instead)
    if (!exact_buckets && opt.force_mode != 2 && maxload > 4 * (n / nparts) + 4096) mode = (scap >= 64) ? 1 : 0;
  }
  st.mode = mode;

  uint64_t cap = next_pow2((uint64_t)std::max<double>(1024.0, std::ceil((double)est / opt.load_factor)));
  cap = std::min<uint64_t>(cap, next_pow2((uint64_t)(2 * n + 2)));
  cap = std::max<uint64_t>(cap, 1024);
  // a sample can miss the groups of a stretch of rows between two of its runs
  // (sorted or clustered rows): room for as many as two strata or the list of
  // unplaced rows hold, so that they do not cost a second pass
  constexpr uint32_t kStageSpill = 1u << 16;
  if (sampled) {
    const uint64_t missed = std::min<uint64_t>(kStageSpill, 2 * (uint64_t)(n / kSampleChunks));
    cap = std::max<uint64_t>(cap, next_pow2(missed + 2 * (uint64_t)est));
  }

  uint8_t* T = nullptr;
  TableRef G{};
  bool done = false;
  bool clean = true;  // counters still as cleared at the start
  // one read-back for the whole call (see Options::sync_checks)
  const bool deferred = !opt.sync_checks;
  bool prof_part = false, prof_agg = false;

  // position and null counters of the result rows, apart from the
  // aggregation's counts and flags in counters[0, 16); cleared with them
  unsigned int* ccount = counters + 256;
  uint32_t* chost = host + 256;
  OutPtrs O;
  std::memset(&O, 0, sizeof(O));
  O.counters = ccount;
  struct Undo {  // the outputs go back when the call does not return them
    Result& r;
    bool keep = false;
    ~Undo() { if (!keep) r.release(); }
  } undo{R};
  auto make_outputs = [&](int64_t out_rows) {
    // every column in one allocation: the data first, then all masks together
    // (one clear for them, and for a small call most of its time was the
    // allocations and clears of its columns)
    {
      auto column = [&](int type_id) {
        OutColumn c;
        c.type_id = type_id;
        c.size = out_rows;
        return c;
      };
      for (int k = 0; k < P.num_keys; ++k) R.keys.push_back(column(keys[k].type_id));
      int j = 0;
      for (auto& r : reqs) {
        std::vector<OutColumn> cols;
        for (size_t q = 0; q < r.aggs.size(); ++q) cols.push_back(column(out_types[j++]));
        R.results.push_back(cols);
      }
      const size_t rows = (size_t)std::max<int64_t>(out_rows, 1);
      const size_t mask_bytes = (rows + 511) / 512 * 64;  // as cudf pads them
      size_t at = 0;
      auto take = [&](size_t bytes) {
        const size_t o = at;
        at += (bytes + 255) & ~(size_t)255;
        return o;
      };
      std::vector<size_t> data_at, mask_at;
      auto each = [&](auto f) {
        for (int k = 0; k < P.num_keys; ++k) f(R.keys[k], keys[k].mask != nullptr);
        int o = 0;
        for (auto& cols : R.results)
          for (auto& c : cols) f(c, P.outs[o++].nullable != 0);
      };
      each([&](OutColumn& c, bool) { data_at.push_back(take(rows * type_width(c.type_id))); });
      const size_t masks = at;
      each([&](OutColumn&, bool nullable) { mask_at.push_back(nullable ? take(mask_bytes) : 0); });
      R.block_bytes = std::max<size_t>(at, 16);
      R.block = alloc.allocate(alloc.ctx, R.block_bytes, (void*)stream);
      if (!R.block) throw Error(ERR_ALLOC, "device allocation of the output columns failed");
      if (at > masks) ck(cudaMemsetAsync((uint8_t*)R.block + masks, 0, at - masks, stream), "memset masks");
      size_t i = 0;
      each([&](OutColumn& c, bool nullable) {
        c.data = (uint8_t*)R.block + data_at[i];
        c.mask = nullable ? (uint32_t*)((uint8_t*)R.block + mask_at[i]) : nullptr;
        ++i;
      });
      for (int k = 0; k < P.num_keys; ++k) {
        O.key_data[k] = R.keys[k].data;
        O.key_mask[k] = R.keys[k].mask;
      }
      j = 0;
      for (auto& cols : R.results)
        for (auto& c : cols) {
          O.out_data[j] = c.data;
          O.out_mask[j++] = c.mask;
        }
    }
  };
  int64_t out_rows = -1;

  if (mode == 2) {
    // ---- pass 1: scatter rows into hash partitions ----
    state.partitioned = true;
    int64_t total = pend.back();
    // region starts, ends and cursors (= starts): one pinned staging copy
    // into one device block
    int64_t* d_base = (int64_t*)S.get(3 * sizeof(int64_t) * nparts);
    int64_t* d_end = d_base + nparts;
    unsigned long long* d_cur = (unsigned long long*)(d_end + nparts);
    {
      if ((size_t)3 * nparts > kRegionWords) throw Error(ERR_LOGIC, "internal error: too many partitions");
      int64_t* st3 = pinned_regions();
      state.staged = true;
      std::memcpy(st3, pbase.data(), 8 * nparts);
      std::memcpy(st3 + nparts, pend.data(), 8 * nparts);
      std::memcpy(st3 + 2 * nparts, pbase.data(), 8 * nparts);
      ck(cudaMemcpyAsync(d_base, st3, 24 * (size_t)nparts, cudaMemcpyHostToDevice, stream), "h2d");
    }
    RecArgs A;
    std::memset(&A, 0, sizeof(A));
    A.nparts = nparts;
    A.end = d_end;
    A.cursor = d_cur;
    // 32-byte loads of records: the allocator gives 16-byte alignment only
    A.recs = (uint64_t*)(((uintptr_t)S.get((size_t)total * 8 * rec.words + 16) + 31) & ~(uintptr_t)31);
    A.counters = counters;
    mark("partition scratch");
    if (opt.profile) ck(cudaEventRecord(events()[0], stream), "event");
    if (!launch_rec_scatter(P, A, rec, dev.smem_optin, stream))
      throw Error(ERR_LOGIC, "internal error: no launch shape for the partition pass");
    ++st.kernels;
    ck(cudaGetLastError(), "partition launch");
    if (opt.profile) ck(cudaEventRecord(events()[4], stream), "event");

    // ---- pass 2: per-partition shared-memory aggregation ----
    // pass-2 work: one item per partition, except that a partition holding
    // far more rows than the average (a heavy key) is cut into row ranges
    // handled by several CTAs, each merging its table into the global table
    std::vector<PartItem> items;
    int64_t nsplit = 0;
    int nwagg = 0;  // leading items taken by the warp-combining launch
    {
      int64_t nrows = 0;
      for (auto r : prows) nrows += r;
      // a work item is about a partition's average share, and small enough
      // that few partitions still spread over every SM (a multiple of 64 rows:
      // pass 2 reads aligned row pairs)
      const int64_t share = nrows / std::max(1, nparts);
      int64_t chunk =
        std::max<int64_t>(32768, nparts < dev.sms ? std::min(share, nrows / (4 * (int64_t)dev.sms)) : share) & ~(int64_t)63;
      // Few partitions of up to 64Ki rows an SM: cut into as many pieces as end
      // soonest, in whole waves over the SMs, an item's table and merges counted
      // as 2Ki rows (few partitions have few groups each).  In items of 32Ki rows
      // 2M rows of 5500 groups were 42 whole partitions: six FLOAT32 sums 0.45
      // ms, now 0.30; 4M rows of 7000 groups 0.58, now 0.41.  Under a long tail
      // the partitions are far from equal and so are their pieces, up to half
      // as long again: three or more to an SM even out (7M Zipf rows of 16K
      // groups, 12 accumulators: 0.80, whole partitions 1.05, 32Ki-row items
      // 0.87; 9.5M rows 1.04 against 0.98 with 32Ki, so the line is lower).
      const bool even =
        exact_buckets && nparts < dev.sms && nrows < (long_tail ? 57344 : 65536) * (int64_t)dev.sms;
      if (even) {
        int64_t best = INT64_MAX;
        for (int64_t k = 1; k <= 16; ++k) {
          if (long_tail && nparts * k < 3 * dev.sms) continue;
          const int64_t end = (nparts * k + dev.sms - 1) / dev.sms * (share / k + 2048);
          if (end < best) best = end, chunk = std::max<int64_t>(64, share / k);
        }
      }
      // partitions that hold a hot key come first, in the launch that folds
      // the rows of one slot per warp.  A long-tailed key distribution (32
      // buckets above four times the usual one: Zipf) has keys of hundreds of
      // rows everywhere and folds everywhere (100M Zipf pairs: 3.5 ms against
      // 4.8 with the hottest partitions only), as do keys in sorted order, whose
      // rows stay together (20M rows of 5000 groups: 1.03 against 3.15).  With
      // wagg_pct given, those above that share of the average fold.
      const bool by_share = ((opt.set_mask | rule_fields) & OPT_WAGG) || !exact_buckets;
      const double heavy = opt.wagg_pct / 100.0 * ((double)nrows / std::max(1, nparts));
      // the folding launch runs by itself: partitions that stand out are cut into
      // pieces that fill the SMs (20M rows, 60K groups, one of 5%: 31 items of
      // 33Ki rows kept the other SMs waiting)
      int64_t folded = 0;
      for (int p = 0; p < nparts; ++p)
        if (long_tail || clustered || phot[p]) folded += prows[p];
      const int64_t hot_chunk =
        by_share || 2 * folded > nrows ? chunk : std::min(chunk, std::max<int64_t>(8192, folded / (2 * (int64_t)dev.sms)));
      for (int pass = 0; pass < 2; ++pass) {
        for (int p = 0; p < nparts; ++p) {
          const int64_t r = prows[p];
          const bool hot_part = !by_share && phot[p] && r > 2 * share && hot_chunk < chunk;
          const int64_t c = hot_part ? hot_chunk : chunk;
          const bool equal = even || hot_part;
          const int64_t pieces = equal ? std::max<int64_t>(1, (r + c / 2) / c) : r > 2 * c ? (r + c - 1) / c : 1;
          const bool split = exact_buckets && pieces > 1;
          const bool folds =
            by_share ? split || (double)r > heavy || opt.wagg_pct == 0 : long_tail || clustered || phot[p];
          if ((pass == 0) != folds) continue;
          if (!split) {
            // VARIANCE/STD: the second pass looks every group up in the global
            // table; with checks after each stage the groups are counted there
            items.push_back(PartItem{p, P.need_second_pass || !deferred, pbase[p], pend[p]});
            continue;
          }
          ++nsplit;
          const int64_t step = equal ? ((r + pieces - 1) / pieces + 63) & ~(int64_t)63 : c;
          for (int64_t b = 0; b < r; b += step)
            items.push_back(PartItem{p, 1, pbase[p] + b, pbase[p] + std::min(r, b + step)});
        }
        if (pass == 0) nwagg = (int)items.size();
      }
      // CTAs claim items in order: largest first within each launch, so the
      // launch does not end waiting on one long item taken last
      auto rows_of = [&](const PartItem& it) { return std::min(it.end - it.begin, prows[it.part]); };
      auto larger = [&](const PartItem& x, const PartItem& y) { return rows_of(x) > rows_of(y); };
      std::stable_sort(items.begin(), items.begin() + nwagg, larger);
      std::stable_sort(items.begin() + nwagg, items.end(), larger);
    }
    PartItem* d_items = (PartItem*)S.get(sizeof(PartItem) * items.size());
    ck(cudaMemcpyAsync(d_items, items.data(), sizeof(PartItem) * items.size(), cudaMemcpyHostToDevice, stream), "h2d");
    // a table four times the groups expected in a partition costs no probes
    // and less to reset than all of shared memory (a caller's estimate may be
    // far off: it gets the whole table)
    const int scap_p = exact_buckets ? (int)std::min<int64_t>(scap_rec, 4 * (est / nparts) + 256) & ~3
                                     : scap_rec;
    const int sfill_p = std::max(1, (int)(scap_p * 0.9));
    // groups expected to miss their partition's shared table, plus those of
    // split partitions, go to the global spill table (no more than there are:
    // its clear and its compaction cost 20 us with room for every slot of 54
    // split partitions)
    const double expect_spill = std::max(0.0, (double)est - 0.85 * (double)nparts * scap_rec);
    uint64_t spill_cap = next_pow2((uint64_t)std::max<double>(65536.0, 2.0 * expect_spill + 2.0 * std::min((double)nsplit * scap2, 1.25 * est) +
                                                                              (P.need_second_pass || !deferred ? 2.0 * est : 0.0)));
    // spill list: room for the rows of the groups expected to spill
    uint32_t spill_list = (uint32_t)std::min<uint64_t>(
      1ull << 31, next_pow2((uint64_t)std::max<double>(262144.0, 4.0 * expect_spill)));
    // rows that pass 2 writes itself (VARIANCE/STD: none, every group goes to T)
    const int64_t dcap = P.need_second_pass ? 0 : (int64_t)(est * 1.5) + (int64_t)nparts * 256 + 4096;
    for (int attempt = 0;; ++attempt) {
      T = (uint8_t*)S.get((size_t)(spill_cap + 1) * P.slot_bytes);
      A.spill_rows = (int64_t*)S.get((size_t)spill_list * sizeof(int64_t));
      A.spill_cap = spill_list;
      k_init_slots<<<dev.sms * 4, 256, 0, stream>>>(T, (int64_t)spill_cap + 1, P.slot_bytes, tmpl);
      if (attempt > 0) ck(cudaMemsetAsync(counters, 0, 16, stream), "memset");
      // [8..9] work, [10..11] groups written by pass 2, [12] spill list length, [13] list overflow
      if (attempt > 0) ck(cudaMemsetAsync(counters + 6, 0, 8 * 4, stream), "memset");
      G = TableRef{T, spill_cap - 1, P.slot_bytes, P.key_words, counters};
      // result rows for every group pass 2 writes and every slot of T; with
      // checks after each stage, pass 2 merges everything into T instead
      if (deferred) {
        out_rows = dcap + (int64_t)spill_cap + 1;
        make_outputs(out_rows);
      }
      const EmitRef D{out_rows, (unsigned long long*)(counters + 10)};
      // items of split (heavy) partitions first, with rows of one slot
      // combined per warp before their shared update; then the rest
      auto launch2 = [&](int first, int count, unsigned int* work, bool wagg) {
        if (count <= 0) return;
        RecArgs Ai = A;
        Ai.items = d_items + first;
        Ai.nitems = count;
        Ai.work = work;
        (P.key_words == 1 ? launch_rec_aggregate1 : launch_rec_aggregate2)(P, Ai, rec, G, D, O, scap_p, sfill_p, tmpl, wagg,
                                                                           stream);
        ++st.kernels;
      };
      launch2(0, nwagg, counters + 8, true);
      launch2(nwagg, (int)items.size() - nwagg, counters + 9, false);
      if (opt.profile) ck(cudaEventRecord(events()[1], stream), "event");
      // rows listed as not fitting their partition's table (none when the
      // sample sized the partitions well): one grid-stride launch that reads
      // the list length on the device
      launch_rec_spill(P, A, rec, G, dev.sms * 2, stream);
      if (!deferred) k_finish_count<<<1, 1, 0, stream>>>(P, G);  // deferred: the compaction counts it
      st.kernels += deferred ? 2 : 3;
      ck(cudaGetLastError(), "partition aggregate launch");
      if (deferred) {
        // counts and flags stay on the device until the compaction is done
        mark("partition passes launched");
        done = true;
        cap = spill_cap;
        prof_part = opt.profile;
        break;
      }
      ck(cudaMemcpyAsync(host, counters, 64, cudaMemcpyDeviceToHost, stream), "d2h");
      ck(cudaStreamSynchronize(stream), "partition sync");
      if (opt.profile && attempt == 0) {
        float ms = 0, ms1 = 0;
        ck(cudaEventElapsedTime(&ms, events()[0], events()[1]), "event time");
        ck(cudaEventElapsedTime(&ms1, events()[0], events()[4]), "event time");
        st.agg_kernel_ms += ms;
        st.scatter_ms = ms1;
      }
      mark("partition passes (synced)");
      if (host[5]) break;  // a region overflowed: fall back to the global table
      if (host[1] == 0 && host[13] == 0) {
        done = true;
        cap = spill_cap;
        break;
      }
      if (attempt >= 6) throw Error(ERR_CUDA, "hash table overflow");
      if (host[1]) spill_cap *= 8;
      if (host[13]) {
        spill_list = (uint32_t)std::min<uint64_t>((uint64_t)spill_list * 8, 1ull << 31);
        spill_cap = std::max<uint64_t>(spill_cap, next_pow2((uint64_t)host[12] * 2));
      }
      S.put(T);
      S.put(A.spill_rows);
      ++st.retries;
    }
    if (!done) {
      clean = false;
      mode = 0;
      st.mode = 0;
      ++st.retries;
      S.put(T);
      S.put(A.spill_rows);
    }
  }

  // shared stage through k_stage_aggregate: plans whose columns all have
  // closed-form updates and whose groups fit one CTA's ~220 KB table
  bool raw_stage = mode == 1 && part_ok && opt.block >= 512 && own_table && est <= (int64_t)(0.85 * scap_rec);
  bool stage_fold = false;
  StageArgs stage;
  std::memset(&stage, 0, sizeof(stage));
  if (!done && raw_stage) {
    stage.rows_per_cta = ((n + dev.sms - 1) / dev.sms + 63) & ~(int64_t)63;
    // copies of the table: as many as fit, while each still sees enough rows
    // per group to be worth folding back
    // (an odd number of four-slot buckets and of 8- or 16-byte units per copy:
    // see k_stage_aggregate)
    const int64_t budget = (int64_t)scap_rec * (P.slot_bytes + 4);
    const int64_t unit = 8 * P.key_words;
    int64_t slots = std::min<int64_t>(scap_rec, (2 * est + 16 + 3) & ~(int64_t)3);
    if ((slots / 4) % 2 == 0 && slots + 4 <= scap_rec) slots += 4;
    auto pitch_of = [&](int64_t sl) {
      const int64_t p = sl * P.slot_bytes;
      return (p / unit) % 2 ? p : p + unit;
    };
    const int64_t fit = budget / (slots * 4 + pitch_of(slots)), worth = stage.rows_per_cta / (16 * est);
    stage.replicas = (int)std::max<int64_t>(1, std::min<int64_t>(kMaxReplicas, std::min(fit, worth)));
    stage.slots = (int)(stage.replicas == 1 ? std::min<int64_t>(scap_rec, (4 * est + 64 + 3) & ~(int64_t)3) : slots);
    stage.pitch = (int)(stage.replicas == 1 ? (int64_t)stage.slots * P.slot_bytes : pitch_of(slots));
    stage.sfill = std::max(1, (int)(stage.slots * 0.9));
    // rows of one slot are folded per warp first where a key may hold a
    // sixteenth of the rows (two lanes of a warp) or rows of one key follow one
    // another, and the copies do not already keep a warp's lanes apart.  Sorted
    // rows, folded / not, ms: 21 accumulators, 4 copies 8M 0.85 / 1.05, 20M 1.78 /
    // 2.26; 8 copies 0.77 / 0.70, 1.58 / 1.40; 15 copies 0.65 / 0.65.  12 or
    // fewer, 4 copies 1.5M 0.22 / 0.32, 9 copies 0.22 / 0.26, 12-15 copies equal.
    const bool wide = P.num_accs > 16;
    stage_fold = stage.replicas < 32 && (!buckets || hot || (clustered && (!wide || stage.replicas < 8)));
    stage.spill_cap = kStageSpill;
    stage.spill_rows = (int64_t*)S.get(sizeof(int64_t) * stage.spill_cap);
    stage.counters = counters;
  }

  if (!done) {
    for (int attempt = 0;; ++attempt) {
      size_t tbytes = (size_t)(cap + 1) * P.slot_bytes;
      T = (uint8_t*)S.get(tbytes);
      k_init_slots<<<dev.sms * 8, 256, 0, stream>>>(T, (int64_t)cap + 1, P.slot_bytes, tmpl);
      if (attempt > 0 || !clean) ck(cudaMemsetAsync(counters, 0, 16 * 4, stream), "memset counters");
      G = TableRef{T, cap - 1, P.slot_bytes, P.key_words, counters};
      int block = std::min(opt.block, 512);
      if (opt.profile) ck(cudaEventRecord(events()[0], stream), "event");
      if (raw_stage) {
        if (attempt > 0) ck(cudaMemsetAsync(counters + 12, 0, 2 * 4, stream), "memset");  // spill list
        st.kernels += launch_stage(P, stage, G, tmpl, stage_fold, stream);
      } else if (mode == 1) {
        size_t sm = (size_t)scap * P.slot_bytes;
        allow_max_smem((const void*)k_aggregate<true>);
        int grid = grid_for((const void*)k_aggregate<true>, block, sm, opt.blocks_per_sm);
        grid = (int)std::min<int64_t>(grid, (n + block - 1) / block);
        k_aggregate<true><<<grid, block, sm, stream>>>(P, G, scap, sfill, tmpl);
      } else {
        int grid = grid_for((const void*)k_aggregate<false>, block, 0, opt.blocks_per_sm);
        grid = (int)std::min<int64_t>(grid, (n + block - 1) / block);
        k_aggregate<false><<<grid, block, 0, stream>>>(P, G, 1, 0, tmpl);
      }
      if (opt.profile) ck(cudaEventRecord(events()[1], stream), "event");
      if (!deferred) k_finish_count<<<1, 1, 0, stream>>>(P, G);
      st.kernels += deferred ? 2 : 3;
      ck(cudaGetLastError(), "aggregate launch");
      if (deferred) {
        prof_agg = opt.profile;
        break;
      }
      ck(cudaMemcpyAsync(host, counters, 64, cudaMemcpyDeviceToHost, stream), "count d2h");
      ck(cudaStreamSynchronize(stream), "aggregate sync");
      if (raw_stage && host[13]) {
        // more groups than the tables held: redo through the per-row kernel
        raw_stage = false;
        host[1] = 1;
      }
      if (opt.profile) {
        float ms = 0;
        ck(cudaEventElapsedTime(&ms, events()[0], events()[1]), "event time");
        st.agg_kernel_ms += ms;
      }
      if (host[1] == 0) break;
      // table overflow: the kernel stopped inserting; redo with a larger table
      if (attempt >= 6) throw Error(ERR_CUDA, "hash table overflow");
      S.put(T);
      cap *= 4;
      ++st.retries;
    }
  }
  st.capacity = (int64_t)cap;
  mark("aggregate done");
  mark("outputs");
  // deferred: outputs are sized for every slot that could hold a group
  int64_t G_n = deferred ? -1 : (int64_t)host[0];
  if (out_rows < 0) out_rows = deferred ? (int64_t)cap + 1 : G_n;
  R.num_groups = G_n;

  if (P.need_second_pass) {
    int grid = grid_for((const void*)k_var_pass, 256, 0, 0);
    k_var_pass<<<grid, 256, 0, stream>>>(P, G);
    ++st.kernels;
    ck(cudaGetLastError(), "variance pass launch");
  }

  // ---- outputs ----
  {
    if (!R.block) make_outputs(out_rows);
    if (opt.profile) ck(cudaEventRecord(events()[2], stream), "event");
    const int64_t limit = deferred ? out_rows : G_n;
    if (deferred || G_n > 0) {
      int64_t nslots = (int64_t)cap + 1;
      int grid = (int)std::min<int64_t>((nslots + 255) / 256, (int64_t)dev.sms * 8);
      k_compact<<<grid, 256, 0, stream>>>(P, T, nslots, P.slot_bytes, limit, O);
      ++st.kernels;
    }
    if (opt.profile) ck(cudaEventRecord(events()[3], stream), "event");
    ck(cudaGetLastError(), "compact launch");
    // deferred: the counts and flags come with the compaction's counters
    const int ncc = 4 + P.num_keys + P.num_outs;
    if (deferred) ck(cudaMemcpyAsync(host, counters, 4 * (256 + ncc), cudaMemcpyDeviceToHost, stream), "counts d2h");
    else ck(cudaMemcpyAsync(chost, ccount, 4 * ncc, cudaMemcpyDeviceToHost, stream), "null counts d2h");
    ck(cudaStreamSynchronize(stream), "compact sync");
    mark("compaction (synced)");
    if (deferred) {
      // an overflow anywhere (a table, a region, the result rows, a spill
      // list): redo the call with checks after every stage, or, where only a
      // sample or the caller's estimate had sized it, from the count of every row
      const bool again = host[1] || chost[1] || (mode == 2 && (host[5] || host[13])) ||
                         (raw_stage && host[13]);
      if (again) {
        R.release();
        Options o2 = opt_in;
        o2.sync_checks = !sampled && opt.groups_hint < 0;
        o2.full_sketch = 1;
        o2.groups_hint = -1;
        S.clear();
        Result again_r = aggregate_call(keys, null_policy, reqs, stream, alloc, o2, stats, state);
        if (stats) ++stats->retries;
        return again_r;
      }
      const int64_t dn = mode == 2 ? (int64_t)(host[10] | ((uint64_t)host[11] << 32)) : 0;
      G_n = (int64_t)chost[2];
      if (G_n != (int64_t)host[0] + dn + chost[3])
        throw Error(ERR_CUDA, "internal error: compaction wrote " + std::to_string(G_n) + " groups of " +
                                  std::to_string((int64_t)host[0] + dn + chost[3]));
      R.num_groups = G_n;
      for (auto& c : R.keys) c.size = G_n;
      for (auto& cols : R.results)
        for (auto& c : cols) c.size = G_n;
      if (prof_part || prof_agg) {
        float ms = 0, ms1 = 0;
        ck(cudaEventElapsedTime(&ms, events()[0], events()[1]), "event time");
        st.agg_kernel_ms += ms;
        if (prof_part) {
          ck(cudaEventElapsedTime(&ms1, events()[0], events()[4]), "event time");
          st.scatter_ms = ms1;
        }
      }
    } else if (chost[1]) {
      throw Error(ERR_CUDA, "internal error: compaction found more groups than were counted");
    }
    if (opt.profile) {
      float ms = 0;
      ck(cudaEventElapsedTime(&ms, events()[2], events()[3]), "event time");
      st.compact_ms = ms;
    }
    for (int k = 0; k < P.num_keys; ++k) R.keys[k].null_count = chost[4 + k];
    int j = 0;
    for (auto& cols : R.results)
      for (auto& c : cols) c.null_count = chost[4 + P.num_keys + j++];
  }
  if (stats) *stats = st;
  undo.keep = true;
  return R;
}
}  // namespace

Result aggregate(const std::vector<Column>& keys, int null_policy, const std::vector<Request>& reqs,
                 cudaStream_t stream, const Allocator& alloc, const Options& opt, Stats* stats)
{
  CallState state;
  auto settle = [&] {  // the thread's next call writes its pinned staging again
    if (state.staged) cudaStreamSynchronize(stream);
  };
  try {
    return aggregate_call(keys, null_policy, reqs, stream, alloc, opt, stats, state);
  } catch (const Error& e) {
    settle();
    // rows as records can take up to about twice the columns' bytes: without
    // room for them the global table, which needs no copy of the rows
    if (e.code != ERR_ALLOC || !state.partitioned) throw;
  } catch (...) {
    settle();
    throw;
  }
  Options o2 = opt;
  o2.partition = 0;
  Result R = aggregate_call(keys, null_policy, reqs, stream, alloc, o2, stats, state);
  if (stats) ++stats->retries;
  return R;
}

}  // namespace gb

namespace gb {

// Global-table aggregation whose hash table and counters live in `scratch`
// (caller-owned device memory) and whose results go to caller-owned columns:
// the path makes no device or pinned-host allocation.  Counters are read back
// with pageable copies.  Returns the number of groups.
int64_t aggregate_into_scratch(const std::vector<Column>& keys, int null_policy,
                               const std::vector<Request>& reqs, cudaStream_t stream, void* scratch,
                               size_t scratch_bytes, int64_t max_groups,
                               std::vector<OutColumn>& out_keys, std::vector<OutColumn>& out_results)
{
  Plan P;
  std::vector<int> out_types;
  build_plan(keys, null_policy, reqs, P, out_types);
  if (max_groups < 0) throw Error(ERR_LOGIC, "max_groups must be >= 0");
  if (out_keys.size() != (size_t)P.num_keys || out_results.size() != (size_t)P.num_outs)
    throw Error(ERR_LOGIC, "output column count does not match the keys and requests");
  for (int k = 0; k < P.num_keys; ++k) {
    OutColumn& o = out_keys[k];
    o.type_id = keys[k].type_id;
    if (max_groups > 0 && !o.data) throw Error(ERR_LOGIC, "output key column without a data buffer");
    if (keys[k].mask && max_groups > 0 && !o.mask) throw Error(ERR_LOGIC, "nullable output key column without a mask buffer");
    if (!keys[k].mask) o.mask = nullptr;
  }
  for (int j = 0; j < P.num_outs; ++j) {
    OutColumn& o = out_results[j];
    o.type_id = out_types[j];
    if (max_groups > 0 && !o.data) throw Error(ERR_LOGIC, "output result column without a data buffer");
    if (P.outs[j].nullable && max_groups > 0 && !o.mask) throw Error(ERR_LOGIC, "nullable output result column without a mask buffer");
    if (!P.outs[j].nullable) o.mask = nullptr;
  }
  const int64_t n = P.num_rows;
  const uint64_t cap = next_pow2((uint64_t)std::max<int64_t>(64, 2 * max_groups));
  const size_t need = 4096 + (size_t)(cap + 1) * P.slot_bytes;
  if (need > scratch_bytes)
    throw Error(ERR_LOGIC, "max_groups " + std::to_string(max_groups) + " with this plan's " +
                               std::to_string(P.slot_bytes) + "-byte slots needs " + std::to_string(need) +
                               " bytes of table; the allocation-free entry point has " +
                               std::to_string(scratch_bytes));
  unsigned int* counters = (unsigned int*)scratch;
  uint8_t* T = (uint8_t*)scratch + 4096;
  ck(cudaMemsetAsync(counters, 0, 4096, stream), "memset counters");
  for (int k = 0; k < P.num_keys; ++k)
    if (out_keys[k].mask && max_groups > 0)
      ck(cudaMemsetAsync(out_keys[k].mask, 0, (size_t)((max_groups + 31) / 32) * 4, stream), "memset mask");
  for (int j = 0; j < P.num_outs; ++j)
    if (out_results[j].mask && max_groups > 0)
      ck(cudaMemsetAsync(out_results[j].mask, 0, (size_t)((max_groups + 31) / 32) * 4, stream), "memset mask");
  uint32_t host[4 + kMaxKeyCols + kMaxOutputs];
  std::memset(host, 0, sizeof(host));
  if (n > 0) {
    DevInfo dev = dev_info();
    SlotTemplate tmpl;
    build_template(P, tmpl);
    k_init_slots<<<dev.sms * 4, 256, 0, stream>>>(T, (int64_t)cap + 1, P.slot_bytes, tmpl);
    TableRef G{T, cap - 1, P.slot_bytes, P.key_words, counters};
    int grid = grid_for((const void*)k_aggregate<false>, 512, 0, 0);
    grid = (int)std::min<int64_t>(grid, (n + 511) / 512);
    k_aggregate<false><<<grid, 512, 0, stream>>>(P, G, 1, 0, tmpl);
    k_finish_count<<<1, 1, 0, stream>>>(P, G);
    ck(cudaGetLastError(), "aggregate launch");
    ck(cudaMemcpyAsync(host, counters, 8, cudaMemcpyDeviceToHost, stream), "count d2h");
    ck(cudaStreamSynchronize(stream), "aggregate sync");
    if (host[1]) throw Error(ERR_LOGIC, "more groups than max_groups (table full)");
    if ((int64_t)host[0] > max_groups)
      throw Error(ERR_LOGIC, "more groups (" + std::to_string(host[0]) + ") than max_groups (" +
                                 std::to_string(max_groups) + ")");
    const int64_t G_n = host[0];
    if (P.need_second_pass) {
      int g2 = grid_for((const void*)k_var_pass, 256, 0, 0);
      k_var_pass<<<g2, 256, 0, stream>>>(P, G);
    }
    OutPtrs O;
    std::memset(&O, 0, sizeof(O));
    for (int k = 0; k < P.num_keys; ++k) {
      O.key_data[k] = out_keys[k].data;
      O.key_mask[k] = out_keys[k].mask;
    }
    for (int j = 0; j < P.num_outs; ++j) {
      O.out_data[j] = out_results[j].data;
      O.out_mask[j] = out_results[j].mask;
    }
    O.counters = counters;
    ck(cudaMemsetAsync(counters, 0, 512, stream), "memset");
    if (G_n > 0) {
      int64_t nslots = (int64_t)cap + 1;
      int g3 = (int)std::min<int64_t>((nslots + 255) / 256, (int64_t)dev.sms * 8);
      k_compact<<<g3, 256, 0, stream>>>(P, T, nslots, P.slot_bytes, G_n, O);
    }
    ck(cudaGetLastError(), "compact launch");
    ck(cudaMemcpyAsync(host, counters, 4 * (4 + P.num_keys + P.num_outs), cudaMemcpyDeviceToHost, stream),
       "null counts d2h");
    ck(cudaStreamSynchronize(stream), "compact sync");
    if (host[1]) throw Error(ERR_CUDA, "internal error: compaction found more groups than were counted");
    host[0] = (uint32_t)G_n;
  } else {
    ck(cudaStreamSynchronize(stream), "sync");
  }
  const int64_t groups = n > 0 ? (int64_t)host[0] : 0;
  for (int k = 0; k < P.num_keys; ++k) {
    out_keys[k].size = groups;
    out_keys[k].null_count = n > 0 ? host[4 + k] : 0;
  }
  for (int j = 0; j < P.num_outs; ++j) {
    out_results[j].size = groups;
    out_results[j].null_count = n > 0 ? host[4 + P.num_keys + j] : 0;
  }
  return groups;
}

}  // namespace gb
