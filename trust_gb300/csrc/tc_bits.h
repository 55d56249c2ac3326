// tc_bits.h — host interface of the block-bitmap counting path (tc_bits.cu).
#pragma once
#include "tc_internal.h"

namespace tc {

// Tables of this path: rows of more than BITS_TABLE_MIN entries; arcs whose rows are both shorter
// are left to the hash-table kernel (48, 64, 96, 128 measured within 1 % of each other on R-MAT
// 20; R-MAT 22 12.9, 12.9, 12.4, 12.3 ms).
constexpr int BITS_TABLE_MIN = 128;
// Longest row the conversion groups in shared memory; graphs with a longer one keep the hash tables.
constexpr int BITS_MAX_ROW = 8192;

struct BitsPlan {
  int nb = 0;               // blocks (of 16 columns) of the bitmap
  unsigned *ctr = nullptr;  // device counters: units, in-list entries, unit claims
  int64_t rows_c_at = 0;    // first C row among the row descriptors
  bool ranked = false;      // the columns are ranked already (bits_columns)
};

bool bits_eligible(const DevGraph3 &g, int64_t max_out_degree);
// Whether enough of the entries fall into the bitmap's columns (waits for st).
int bits_columns(trust_tc_ctx *c, const DevGraph3 &g, cudaStream_t st, BitsPlan *plan, bool *suit);
// After the scheduling pass (its pairs, counts and, for one graph, work sums) and its readback.  Only arcs
// of source rows in [row_lo, row_hi) are counted.  A tile job's A and C rows must be duplicate-free.
int bits_prepare(trust_tc_ctx *c, const DevGraph3 &g, int64_t row_lo, int64_t row_hi, const SchedPlan &plan,
                 int64_t max_out_degree, cudaStream_t st, BitsPlan *out);
int bits_launch(trust_tc_ctx *c, const BitsPlan &plan, const int32_t *adj, TcControl *ctl, cudaStream_t st);

}  // namespace tc
