// gb_record.cu -- record layout and the launchers of pass 1 and the spill pass
// (gb_record.cuh), in their own compilation unit.
#include <algorithm>
#include <cstring>

#include "gb_engine.h"
#include "gb_record.cuh"

namespace gb {

RecCol rec_col(const ValCol& c, int bit, int shift, int adv)
{
  const bool nothing = c.sum_off < 0 && c.min_off < 0 && c.max_off < 0 && c.sq_off < 0;
  const uint32_t kind = nothing               ? RK_NONE
                        : c.cat == CAT_F64    ? RK_F64
                        : c.cat == CAT_F32    ? RK_F32
                        : c.width == 8        ? RK_W64
                        : c.cat == CAT_SIGNED ? RK_S32
                                              : RK_Z32;
  const uint32_t flags = (c.cat == CAT_SIGNED ? RF_SIGNED : 0) | (c.cat == CAT_BOOL ? RF_BOOL : 0) |
                         (c.sum_op == OP_SUM_I32 ? RF_SUM32 : 0);
  const uint32_t ext = c.width < 4 ? 32 - 8 * c.width : 0;
  return RecCol{{(uint32_t)(uint16_t)c.sum_off | (uint32_t)(uint16_t)c.min_off << 16,
                 (uint32_t)(uint16_t)c.max_off | (uint32_t)(uint16_t)c.sq_off << 16,
                 (uint32_t)(uint16_t)c.nulls_off | kind << 16 | (uint32_t)shift << 24,
                 (uint32_t)adv | ext << 8 | flags << 16 | (uint32_t)bit << 24}};
}

bool record_layout(const Plan& P, RecSpec& S)
{
  std::memset(&S, 0, sizeof(S));
  if (P.num_vals > kMaxRecCols) return false;
  int key_bits = 0;
  for (int k = 0; k < P.num_keys; ++k) {
    const KeyCol& c = P.keys[k];
    key_bits = std::max(key_bits, 64 * c.word + c.shift + 8 * c.width);
    if (c.has_null_bit) key_bits = std::max(key_bits, 64 * c.null_word + c.null_shift + 1);
  }
  const int key_bytes = P.key_words == 2 ? 16 : key_bits <= 32 ? 4 : 8;
  S.keymask = key_bytes == 4 ? 0xFFFFFFFFull : ~0ull;
  for (int v = 0; v < P.num_vals; ++v) S.has_bits |= P.vals[v].mask != nullptr;
  // widest columns first, each in the first free place aligned to its width
  int order[kMaxRecCols];
  for (int v = 0; v < P.num_vals; ++v) order[v] = v;
  std::stable_sort(order, order + P.num_vals, [&](int a, int b) { return P.vals[a].width > P.vals[b].width; });
  int at[kMaxRecCols];
  for (int words : kRecSizes) {
    bool used[8 * kMaxRecWords] = {};
    for (int i = 0; i < key_bytes; ++i) used[i] = true;
    if (S.has_bits) used[8 * words - 1] = true;
    bool fits = key_bytes <= 8 * words;
    for (int j = 0; j < P.num_vals && fits; ++j) {
      const int w = P.vals[order[j]].width;
      int o = 0;
      for (; o + w <= 8 * words; o += w) {
        bool free = true;
        for (int i = 0; i < w; ++i) free = free && !used[o + i];
        if (free) break;
      }
      if (o + w > 8 * words) { fits = false; break; }
      for (int i = 0; i < w; ++i) used[o + i] = true;
      at[order[j]] = o;
    }
    if (fits) { S.words = words; break; }
  }
  if (S.words == 0) return false;
  std::stable_sort(order, order + P.num_vals, [&](int a, int b) { return at[a] < at[b]; });
  S.ncols = P.num_vals;
  int word = P.key_words - 1;
  for (int j = 0; j < P.num_vals; ++j) {
    const ValCol& c = P.vals[order[j]];
    S.src_col[j] = order[j];
    S.off[j] = at[order[j]];
    S.col[j] = rec_col(c, order[j], 8 * (S.off[j] % 8), S.off[j] / 8 - word);
    word = S.off[j] / 8;
  }
  for (int v = 0; v < P.num_vals; ++v) {
    if (P.vals[v].mask) {
      S.mask_col[S.nmask] = v;
      S.mask_bit[S.nmask++] = (uint8_t)v;
    } else {
      S.vb_const |= (uint8_t)(1u << v);
    }
  }
  const KeyCol& k = P.keys[0];
  S.key8 = P.num_keys == 1 && k.width == 8 && k.mask == nullptr && k.word == 0 && k.shift == 0 &&
           (k.cat == CAT_SIGNED || k.cat == CAT_UNSIGNED);
  return true;
}

namespace {
template <int KW, int NT, int RPT, int MINB>
void launch(const Plan& P, const RecArgs& A, const RecSpec& S, cudaStream_t stream)
{
  constexpr int T = NT * RPT;
  const size_t smem = rec_scatter_smem(T, S.words, A.nparts, S.nmask);
  const int64_t ntiles = (P.num_rows + T - 1) / T;
  auto go = [&](auto kern) {
    allow_max_smem((const void*)kern);
    const int grid = (int)std::min<int64_t>(grid_for((const void*)kern, NT, smem, MINB), ntiles);
    kern<<<grid, NT, smem, stream>>>(P, A, S);
  };
  // reservations in flight across phase C while their results fit registers
  const int per = (A.nparts + NT - 1) / NT;
  if (per <= 2) go(k_rec_scatter<KW, NT, RPT, MINB, 2>);
  else if (per <= 8) go(k_rec_scatter<KW, NT, RPT, MINB, 8>);
  else go(k_rec_scatter<KW, NT, RPT, MINB, 1>);
}
template <int KW, int NT, int MINB>
bool launch_rows(int rows, const Plan& P, const RecArgs& A, const RecSpec& S, cudaStream_t s)
{
  switch (rows) {
    case 8:
      if constexpr (KW == 1) {
        launch<KW, NT, 8, MINB>(P, A, S, s);
        return true;
      }
      return false;
    case 6: launch<KW, NT, 6, MINB>(P, A, S, s); return true;
    case 5: launch<KW, NT, 5, MINB>(P, A, S, s); return true;
    case 4: launch<KW, NT, 4, MINB>(P, A, S, s); return true;
    case 3: launch<KW, NT, 3, MINB>(P, A, S, s); return true;
    case 2: launch<KW, NT, 2, MINB>(P, A, S, s); return true;
    case 1: launch<KW, NT, 1, MINB>(P, A, S, s); return true;
    default: return false;
  }
}
template <int KW>
bool launch_shape(const RecShape& r, const Plan& P, const RecArgs& A, const RecSpec& S, cudaStream_t s)
{
  return r.ctas == 1 ? launch_rows<KW, 1024, 1>(r.rows, P, A, S, s) : launch_rows<KW, 512, 2>(r.rows, P, A, S, s);
}
}  // namespace

bool launch_rec_scatter(const Plan& P, const RecArgs& A, const RecSpec& S, int smem_optin, cudaStream_t stream)
{
  const RecShape r = rec_shape(P.key_words, S.words, A.nparts, S.nmask, smem_optin);
  return P.key_words == 1 ? launch_shape<1>(r, P, A, S, stream) : launch_shape<2>(r, P, A, S, stream);
}

void launch_rec_spill(const Plan& P, const RecArgs& A, const RecSpec& S, const TableRef& G, int grid,
                      cudaStream_t stream)
{
  k_rec_spill<<<grid, 256, 0, stream>>>(P, G, A, S);
}

}  // namespace gb
