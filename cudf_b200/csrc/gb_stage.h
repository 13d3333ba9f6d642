// gb_stage.h -- host interface of the shared-stage mode (gb_stage.cuh).
#pragma once
#include "gb_record.h"

namespace gb {

struct StageArgs {
  int64_t rows_per_cta;    // contiguous row range of a CTA (a multiple of 64)
  int32_t replicas;        // copies of the table in a CTA
  int32_t slots;           // slots of one copy (a multiple of four)
  int32_t pitch;           // bytes from one copy's slots to the next one's
  int32_t sfill;           // slots of one copy that may be claimed
  int64_t* spill_rows;     // rows that fitted no copy
  unsigned int spill_cap;
  unsigned int* counters;  // [12] spill list length, [13] its overflow
};

constexpr int kMaxReplicas = 256;

// Column descriptors over the caller's own columns, in plan order.
void stage_layout(const Plan& P, RecSpec& S);
// Aggregates the rows into G through per-CTA shared tables, then applies the
// spilled rows; returns the kernels launched.
int launch_stage(const Plan& P, const StageArgs& A, const TableRef& G, const SlotTemplate& tmpl, bool fold,
                 cudaStream_t stream);

}  // namespace gb
