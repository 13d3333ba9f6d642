// gb_record.h -- host interface of the partitioned path's row records
// (gb_record.cuh): layout, launchers.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "gb_kernels.cuh"
#include "gb_partition.cuh"
#include "gb_plan.h"
#include "gb_record_shape.h"

namespace gb {

constexpr int kMaxRecCols = 8;     // value columns of a record (one validity byte)
constexpr int kMaxRecWords = 12;   // 8-byte words of a record

// How a value column's element is read out of its word and updated.
enum RecKind : uint8_t { RK_F64 = 0, RK_F32, RK_W64, RK_S32, RK_Z32, RK_NONE };

// One value column of a record, in record order: what pass 2 needs to update
// a slot, in one 16-byte descriptor.
// (Kept packed, so that a kernel holds it in four registers.)
struct __align__(16) RecCol {
  uint32_t w[4];
  // slot byte offsets of the accumulators and the null counter, -1 when absent
  __host__ __device__ int sum() const { return (int16_t)(w[0] & 0xFFFFu); }
  __host__ __device__ int min() const { return (int16_t)(w[0] >> 16); }
  __host__ __device__ int max() const { return (int16_t)(w[1] & 0xFFFFu); }
  __host__ __device__ int sq() const { return (int16_t)(w[1] >> 16); }
  __host__ __device__ int nulls() const { return (int16_t)(w[2] & 0xFFFFu); }
  __host__ __device__ int kind() const { return (w[2] >> 16) & 0xFF; }  // RecKind
  __host__ __device__ int shift() const { return w[2] >> 24; }          // bit position inside its word
  __host__ __device__ int adv() const { return w[3] & 0xFF; }           // words since the previous column's word
  __host__ __device__ int ext() const { return (w[3] >> 8) & 0xFF; }    // narrow integers: 32 - element bits
  __host__ __device__ int flags() const { return (w[3] >> 16) & 0xFF; } // RF_*
  __host__ __device__ int bit() const { return w[3] >> 24; }            // validity bit
};
enum : uint8_t { RF_SIGNED = 1, RF_SUM32 = 2, RF_BOOL = 4 };

// The record of a row: key word(s), then the value columns widest first, each
// at a multiple of its width, and the validity byte in the top byte of the
// last word (only when a value column has a mask).  Plans whose packed key
// fits 32 bits keep it in the low half of word 0.
struct RecSpec {
  int32_t words;        // 8-byte words per record: 2, 4, 6, 8 or 12
  int32_t ncols;
  int32_t has_bits;
  int32_t pad;
  uint64_t keymask;     // bits of word 0 that belong to a one-word key
  RecCol col[kMaxRecCols];
  int32_t src_col[kMaxRecCols];  // plan value column of record column j
  int32_t off[kMaxRecCols];      // its byte offset in the record
  int32_t nmask;                 // value columns with a mask, and their validity bits
  int32_t mask_col[kMaxRecCols];
  uint8_t mask_bit[kMaxRecCols];
  uint8_t vb_const;              // validity bits of the columns without one
  int32_t key8;                  // one 8-byte integer key column without a mask: its bits are the key word
};

struct RecArgs {
  int32_t nparts;
  const int64_t* end;            // [nparts] one past the last record of each region
  unsigned long long* cursor;    // [nparts] next free record of each region
  uint64_t* recs;                // 32-byte aligned
  unsigned int* counters;        // [5] region overflow, [12] spill list length, [13] its overflow
  int64_t* spill_rows;           // pass 2: records that did not fit their shared table
  unsigned int spill_cap;
  const PartItem* items;         // pass 2 work list
  int32_t nitems;
  unsigned int* work;            // pass 2 claim counter
};

// Descriptor of a value column: validity bit, bit position in its word, words
// since the previous column's.
RecCol rec_col(const ValCol& c, int bit, int shift, int adv);
// Lays the record out; false when the plan has no record form (more than
// kMaxRecCols value columns).
bool record_layout(const Plan& P, RecSpec& S);
// Pass 1 over nparts partitions; false when no launch shape fits (see rec_shape).
bool launch_rec_scatter(const Plan& P, const RecArgs& A, const RecSpec& S, int smem_optin, cudaStream_t stream);
// Pass 2 over A's items, for one- and two-word keys; `wagg`: rows of one slot
// combined per warp first.
void launch_rec_aggregate1(const Plan& P, const RecArgs& A, const RecSpec& S, const TableRef& G, const EmitRef& D,
                           const OutPtrs& O, int scap, int sfill, const SlotTemplate& tmpl, bool wagg, cudaStream_t stream);
void launch_rec_aggregate2(const Plan& P, const RecArgs& A, const RecSpec& S, const TableRef& G, const EmitRef& D,
                           const OutPtrs& O, int scap, int sfill, const SlotTemplate& tmpl, bool wagg, cudaStream_t stream);
// Applies the listed records to the global spill table.
void launch_rec_spill(const Plan& P, const RecArgs& A, const RecSpec& S, const TableRef& G, int grid,
                      cudaStream_t stream);

}  // namespace gb
