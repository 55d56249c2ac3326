// tc_short.cu — large graphs whose rows all have at most 8 entries (meshes, road networks, very
// sparse random graphs), counted in row order without queues.
//
// The persistent kernel reaches such rows through the class lists, four or eight lanes per row, with
// the registers and the loop structure of its larger classes (mesh 4096 x 4096: 242 warp instructions
// per 32 arcs at 40 warps per SM).  Here a warp takes 32 consecutive rows: their offsets and entries
// are read coalesced, the rows' arcs fill the lanes without gaps, and each lane reads its arc's target
// row (at most three 16-byte pieces) and compares it with its source row's keys, which the warp
// staged in shared memory.
// Bound by the load pipe (82 % busy: every lane reads its own two offsets and row) and its latency:
// mesh 4096 x 4096 0.50 -> 0.36 ms of counting, the call 651 -> 490 us.  Rows to 8 beside longer
// ones were tried too, with the target rows' pieces dealt over the lanes: Chung-Lu 3.8 M 433 -> 412
// us but 160 -> 213 on 300,000 arcs and 120 us more on R-MAT 20, so mixed graphs keep the queues.
#include <algorithm>

#include "tc_count.h"
#include "tc_internal.h"
#include "tc_short.h"

namespace tc {

namespace {

constexpr int SH_WARPS = 8;
constexpr int SH_THREADS = 32 * SH_WARPS;
constexpr int SH_MAX = SHORT_ROW_MAX;        // entries of a row
constexpr int SH_WAVES = 4;
constexpr int SH_ARCS = 32 * SH_MAX;         // arcs of a warp's 32 rows

struct ShortArgs {
  const int64_t *beg;
  const int32_t *adj;
  int64_t n, m, row_lo, row_hi;
  TcControl *ctl;
};

// Matches of one 16-byte piece (entries at..at+3 of adj) that lie in the target row [s, s + dd).
template <int K>
__device__ __forceinline__ unsigned piece_hits(int4 w, int rel, int dd, const int (&key)[K]) {
  bool m0 = false, m1 = false, m2 = false, m3 = false;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    m0 |= w.x == key[k];
    m1 |= w.y == key[k];
    m2 |= w.z == key[k];
    m3 |= w.w == key[k];
  }
  return (unsigned)(m0 && (unsigned)rel < (unsigned)dd) + (unsigned)(m1 && (unsigned)(rel + 1) < (unsigned)dd) +
         (unsigned)(m2 && (unsigned)(rel + 2) < (unsigned)dd) + (unsigned)(m3 && (unsigned)(rel + 3) < (unsigned)dd);
}

// Entries at..at+3 (at a multiple of 4): one 16-byte load where all four lie in the array.
template <bool VEC>
__device__ __forceinline__ int4 load4(const int32_t *__restrict__ adj, unsigned at, unsigned m) {
  if (VEC && at + 3 < m) return __ldg(reinterpret_cast<const int4 *>(adj + at));
  return make_int4(at < m ? tc_ld_nc(adj + at) : -1, at + 1 < m ? tc_ld_nc(adj + at + 1) : -1,
                   at + 2 < m ? tc_ld_nc(adj + at + 2) : -1, at + 3 < m ? tc_ld_nc(adj + at + 3) : -1);
}

template <bool VEC>
__global__ void __launch_bounds__(SH_THREADS, 6) short_rows_kernel(ShortArgs p) {
  __shared__ __align__(16) int keys_all[SH_WARPS][SH_ARCS];  // row of lane l: 8 l .., -1 past its end
  __shared__ unsigned char slot_all[SH_WARPS][SH_ARCS];      // arc k: its place in keys
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int *keys = keys_all[warp];
  unsigned char *slot = slot_all[warp];
  const int64_t nwarps = (int64_t)gridDim.x * SH_WARPS;
  const int64_t tiles = (p.n + 31) >> 5;
  const unsigned m = (unsigned)p.m;  // below 2^31
  unsigned long long hits = 0, wedges = 0;
  for (int64_t t = (int64_t)blockIdx.x * SH_WARPS + warp; t < tiles; t += nwarps) {
    const int64_t v = t * 32 + lane;
    int b = 0, d = 0;
    if (v < p.n) {
      const long long lo = tc_ld_nc(p.beg + v);
      b = (int)lo;
      d = (int)(tc_ld_nc(p.beg + v + 1) - lo);
      if (d < 2 || v < p.row_lo || v >= p.row_hi) d = 0;
    }
    const bool wide = __any_sync(TC_FULL_MASK, d > 4);
    int w[SH_MAX];
#pragma unroll
    for (int j = 0; j < 4; ++j) w[j] = j < d ? tc_ld_nc(p.adj + b + j) : -1;
    if (wide) {
#pragma unroll
      for (int j = 4; j < SH_MAX; ++j) w[j] = j < d ? tc_ld_nc(p.adj + b + j) : -1;
    }
    int incl = d;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(TC_FULL_MASK, incl, o);
      if (lane >= o) incl += y;
    }
    const int tot = __shfl_sync(TC_FULL_MASK, incl, 31);
    if (tot == 0) continue;
    unsigned char *mine = slot + (incl - d);
    reinterpret_cast<int4 *>(keys)[2 * lane] = make_int4(w[0], w[1], w[2], w[3]);
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (j < d) mine[j] = (unsigned char)(8 * lane + j);
    if (wide) {
      reinterpret_cast<int4 *>(keys)[2 * lane + 1] = make_int4(w[4], w[5], w[6], w[7]);
#pragma unroll
      for (int j = 4; j < SH_MAX; ++j)
        if (j < d) mine[j] = (unsigned char)(8 * lane + j);
    }
    __syncwarp();
    unsigned h = 0, wd = 0;
    for (int k0 = 0; k0 < tot; k0 += 32) {
      const int k = k0 + lane;
      int s = 0, dd = 0, at = 0;
      if (k < tot) {
        at = slot[k];
        const int u = keys[at];
        const long long lo = tc_ld_nc(p.beg + u);
        s = (int)lo;
        dd = (int)(tc_ld_nc(p.beg + u + 1) - lo);
      }
      wd += (unsigned)dd;
      const int4 ka = reinterpret_cast<const int4 *>(keys)[at >> 3 << 1];
      if (!wide && !__any_sync(TC_FULL_MASK, dd > 4)) {  // at most four entries on both sides
        int e[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) e[j] = j < dd ? tc_ld_nc(p.adj + s + j) : -2;
#pragma unroll
        for (int j = 0; j < 4; ++j) h += e[j] == ka.x || e[j] == ka.y || e[j] == ka.z || e[j] == ka.w;
        continue;
      }
      const int pieces = dd ? (s + dd - (s & ~3) + 3) >> 2 : 0;  // 0..3
      const unsigned from = (unsigned)(s & ~3);
      const int4 none = make_int4(-1, -1, -1, -1);
      const int4 x = pieces > 0 ? load4<VEC>(p.adj, from, m) : none;
      const int4 y = pieces > 1 ? load4<VEC>(p.adj, from + 4, m) : none;
      const bool three = __any_sync(TC_FULL_MASK, pieces > 2);
      const int4 z = pieces > 2 ? load4<VEC>(p.adj, from + 8, m) : none;
      auto walk = [&](const auto &key) {
        h += piece_hits(x, (int)from - s, dd, key) + piece_hits(y, (int)from + 4 - s, dd, key);
        if (three) h += piece_hits(z, (int)from + 8 - s, dd, key);
      };
      if (wide) {
        const int4 kb = reinterpret_cast<const int4 *>(keys)[(at >> 3 << 1) + 1];
        const int key[8] = {ka.x, ka.y, ka.z, ka.w, kb.x, kb.y, kb.z, kb.w};
        walk(key);
      } else {
        const int key[4] = {ka.x, ka.y, ka.z, ka.w};
        walk(key);
      }
    }
    hits += h;
    wedges += wd;
    __syncwarp();
  }
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) {
    hits += __shfl_down_sync(TC_FULL_MASK, hits, o);
    wedges += __shfl_down_sync(TC_FULL_MASK, wedges, o);
  }
  __shared__ unsigned long long sum[2];
  if (threadIdx.x < 2) sum[threadIdx.x] = 0;
  __syncthreads();
  if (lane == 0 && hits) atomicAdd(&sum[0], hits);
  if (lane == 0 && wedges) atomicAdd(&sum[1], wedges);
  __syncthreads();
  if (threadIdx.x == 0 && sum[0]) atomicAdd(&p.ctl->count, sum[0]);
  if (threadIdx.x == 0 && sum[1]) atomicAdd(&p.ctl->wedges, sum[1]);
}

}  // namespace

int launch_short_rows(const int64_t *beg, const int32_t *adj, int64_t n, int64_t m, int64_t row_lo, int64_t row_hi,
                      TcControl *ctl, int num_sms, cudaStream_t st) {
  ShortArgs a{beg, adj, n, m, row_lo, row_hi, ctl};
  // several CTAs per resident slot: they are handed out as SMs free up, so heavy stretches of rows
  // (the first of a renumbered graph) do not set the tail
  const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, (int64_t)num_sms * 6 * SH_WAVES));
  if (((uintptr_t)adj & 15) == 0) short_rows_kernel<true><<<blocks, SH_THREADS, 0, st>>>(a);
  else short_rows_kernel<false><<<blocks, SH_THREADS, 0, st>>>(a);
  TC_NOTE_LAUNCH();
  TC_CUDA_TRY(cudaGetLastError());
  return TRUST_TC_OK;
}

}  // namespace tc
