// tc_rows.cuh — device helpers shared by the counting kernels: row bounds, hash-table inserts, short rows
// matched from registers.
#pragma once
#include "tc_common.cuh"

namespace tc {

// Row start and length of v (int: m < 2^31 is enforced on the host).
__device__ __forceinline__ void row_of(const int64_t *__restrict__ beg, int v, int &b, int &d) {
  const long long lo = tc_ld_nc(beg + v), hi = tc_ld_nc(beg + v + 1);
  b = (int)lo;
  d = (int)(hi - lo);
}

__device__ __forceinline__ int ceil_log2_table(int d) {
  // smallest power of two >= 2d, at least 64 slots
  int need = max(2 * d, 64);
  return 32 - __clz(need - 1);
}

// Insert into an open-addressing table of 2^log2 slots (log2 >= 6; -1 = empty) in buckets of four: the first
// free slot from the first of bucket hash(key) on.
__device__ __forceinline__ bool set_insert(int *tab, int log2, int key) {
  const unsigned mask = (1u << log2) - 1u;
  unsigned h = tc_hash((unsigned)key, log2 - 2) << 2;
  for (unsigned it = 0; it <= mask; ++it) {
    int prev = atomicCAS(tab + h, -1, key);
    if (prev == -1 || prev == key) return true;
    h = (h + 1u) & mask;
  }
  return false;
}

// Position (0..31) of the n-th (0-based) set bit of mask; mask must have more than n set bits.
__device__ __forceinline__ int nth_set_bit(unsigned mask, int n) {
  int pos = 0;
#pragma unroll
  for (int step = 16; step >= 1; step >>= 1) {
    const int cnt = __popc(mask & ((1u << step) - 1u));
    if (n >= cnt) {
      n -= cnt;
      mask >>= step;
      pos += step;
    }
  }
  return pos;
}

// Membership of w in a row of at most G keys held in registers (-1 past the row; w >= 0).
template <int G>
__device__ __forceinline__ unsigned match_keys(int w, const int (&key)[G]) {
  bool m = false;
#pragma unroll
  for (int k = 0; k < G; ++k) m |= w == key[k];
  return m;
}

// One lane walks its own arc's target row against its vertex's keys in registers: the first eight
// entries and the next four are loaded before any is matched (most of these rows are that short),
// then four at a time with the next four in flight.  -2 marks entries past the row.
template <int G>
__device__ __forceinline__ unsigned lane_walk(const int32_t *__restrict__ row, int d, const int (&key)[G]) {
  unsigned h = 0;
  int w[8];
#pragma unroll
  for (int r = 0; r < 8; ++r) w[r] = r < d ? tc_ld_nc(row + r) : -2;
  int n0 = -2, n1 = -2, n2 = -2, n3 = -2;
  if (d > 8) {
    n0 = tc_ld_nc(row + 8);
    n1 = 9 < d ? tc_ld_nc(row + 9) : -2;
    n2 = 10 < d ? tc_ld_nc(row + 10) : -2;
    n3 = 11 < d ? tc_ld_nc(row + 11) : -2;
  }
#pragma unroll
  for (int r = 0; r < 8; ++r) h += match_keys<G>(w[r], key);
  for (int k = 8; k < d; k += 4) {
    const int m0 = k + 4 < d ? tc_ld_nc(row + k + 4) : -2, m1 = k + 5 < d ? tc_ld_nc(row + k + 5) : -2,
              m2 = k + 6 < d ? tc_ld_nc(row + k + 6) : -2, m3 = k + 7 < d ? tc_ld_nc(row + k + 7) : -2;
    h += match_keys<G>(n0, key) + match_keys<G>(n1, key) + match_keys<G>(n2, key) + match_keys<G>(n3, key);
    n0 = m0; n1 = m1; n2 = m2; n3 = m3;
  }
  return h;
}

}  // namespace tc
