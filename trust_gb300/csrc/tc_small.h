// tc_small.h — host interface of the one-launch path for small graphs (tc_small.cu).
#pragma once
#include "tc_internal.h"

namespace tc {

// Faster than the general path at every size measured below these bounds: 8 KiB of bitmap per warp
// still leaves three CTAs of eight warps per SM, and up to 2^21 arcs the two paths report the same
// class sizes.
constexpr int64_t SMALL_MAX_IDS = 65536;
constexpr int64_t SMALL_MAX_ARCS = (1 << 21) - 1;

bool small_graph(int64_t n, int64_t m);
// The whole count (synchronises st, after an event in c->ev[4]); the totals, class sizes under the tuned classes
// and under the plain split, are in c->h_ctl.
int small_count(trust_tc_ctx *c, const int64_t *beg, const int32_t *adj, int64_t n, int64_t m, int64_t row_lo,
                int64_t row_hi, int check_ids, int warp_max, int cta_max, cudaStream_t st);

}  // namespace tc
