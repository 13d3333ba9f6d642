// gb_record_agg2.cu -- pass 2 over records with two-word keys (gb_record.cuh), in its
// own compilation unit.
#include <algorithm>

#include "gb_engine.h"
#include "gb_record.cuh"

namespace gb {

void launch_rec_aggregate2(const Plan& P, const RecArgs& A, const RecSpec& S, const TableRef& G, const EmitRef& D,
                           const OutPtrs& O, int scap, int sfill, const SlotTemplate& tmpl, bool wagg, cudaStream_t stream)
{
  const size_t smem = (size_t)scap * 4 + (size_t)(scap + 1) * P.slot_bytes;  // tags, slots, the all-ones key's
  auto go = [&](auto kern) {
    allow_max_smem((const void*)kern);
    const int grid = std::min(grid_for((const void*)kern, 1024, smem, 0), A.nitems);
    kern<<<grid, 1024, smem, stream>>>(P, A, S, G, D, O, scap, sfill, tmpl);
  };
  switch (S.words) {
    case 2: wagg ? go(k_rec_aggregate<2, 2, true>) : go(k_rec_aggregate<2, 2, false>); break;
    case 4: wagg ? go(k_rec_aggregate<2, 4, true>) : go(k_rec_aggregate<2, 4, false>); break;
    case 6: wagg ? go(k_rec_aggregate<2, 6, true>) : go(k_rec_aggregate<2, 6, false>); break;
    case 8: wagg ? go(k_rec_aggregate<2, 8, true>) : go(k_rec_aggregate<2, 8, false>); break;
    default: wagg ? go(k_rec_aggregate<2, 12, true>) : go(k_rec_aggregate<2, 12, false>); break;
  }
}

}  // namespace gb
