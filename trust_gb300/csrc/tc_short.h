// tc_short.h — host interface of the short-row kernel (tc_short.cu).
#pragma once
#include "tc_internal.h"

namespace tc {

constexpr int SHORT_ROW_MAX = 8;

// Count the rows in [row_lo, row_hi) of a validated CSR none of whose rows is longer than
// SHORT_ROW_MAX into ctl.
int launch_short_rows(const int64_t *beg, const int32_t *adj, int64_t n, int64_t m, int64_t row_lo, int64_t row_hi,
                      TcControl *ctl, int num_sms, cudaStream_t st);

}  // namespace tc
