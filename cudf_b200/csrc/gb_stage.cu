// gb_stage.cu -- launcher of the shared-stage mode (gb_stage.cuh), in its own
// compilation unit.
#include <algorithm>
#include <cstring>

#include "gb_engine.h"
#include "gb_stage.cuh"

namespace gb {

void stage_layout(const Plan& P, RecSpec& S)
{
  std::memset(&S, 0, sizeof(S));
  S.ncols = P.num_vals;
  for (int v = 0; v < P.num_vals; ++v) S.col[v] = rec_col(P.vals[v], v, 0, v > 0);
}

int launch_stage(const Plan& P, const StageArgs& A, const TableRef& G, const SlotTemplate& tmpl, bool fold,
                 cudaStream_t stream)
{
  RecSpec S;
  stage_layout(P, S);
  const size_t total = (size_t)A.replicas * A.slots;
  const size_t smem = total * 4 + (size_t)A.replicas * A.pitch + P.slot_bytes;
  const int grid = (int)((P.num_rows + A.rows_per_cta - 1) / A.rows_per_cta);
  auto go = [&](auto kern) {
    allow_max_smem((const void*)kern);
    kern<<<grid, 1024, smem, stream>>>(P, A, S, G, tmpl);
  };
  const bool few = P.num_vals <= 4;
  if (P.key_words == 1) {
    if (fold) few ? go(k_stage_aggregate<1, 4, true>) : go(k_stage_aggregate<1, 8, true>);
    else few ? go(k_stage_aggregate<1, 4, false>) : go(k_stage_aggregate<1, 8, false>);
  } else {
    if (fold) few ? go(k_stage_aggregate<2, 4, true>) : go(k_stage_aggregate<2, 8, true>);
    else few ? go(k_stage_aggregate<2, 4, false>) : go(k_stage_aggregate<2, 8, false>);
  }
  k_stage_spill<<<std::min(grid, 64), 256, 0, stream>>>(P, G, A);
  return 2;
}

}  // namespace gb
