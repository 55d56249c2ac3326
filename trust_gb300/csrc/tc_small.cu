// tc_small.cu — graphs small enough that latency is the whole cost: one launch, one synchronisation.
//
// The general path checks and classifies the rows, reads the class sizes back, launches the counting
// kernel over five class queues and reads the count back: two host round trips and about thirty
// dependent memory latencies around a few microseconds of work.  Here one kernel does all of it: a
// warp per (row, every S-th batch of 32 arcs) checks what it reads before using it as an index,
// builds the row's bitmap over all ids in shared memory (a probe is one 4-byte load, no hashing) and
// probes it, four rows at a time, eight lanes each; the last CTA to finish writes the totals
// straight into the context's pinned control block and clears the accumulators.
// Calls on GB300, general path / this one, us: R-MAT 8 (1,311 arcs) 79 / 27, R-MAT 16 ef16 (0.9 M)
// 400 / 126, K_512 191 / 79, Erdos-Renyi 60,000 / 1.9 M arcs 161 / 133.
// Small graphs are bound by the launch and the round trip (device time 12 of R-MAT 8's 28 us), R-MAT 16 by the
// L1 (75 % busy) and the issue (68 %) of its 94 M probes.  Every other round of rows goes to the warps in reverse
// order: with rows longest first a warp then gets about the same work (R-MAT 16 160 -> 142 us, R-MAT
// 16 ef32 330 -> 244).  Tried and slower: chunks of 64 arcs whatever their rows (181 us).
// Within a CTA the rows go to whichever warp is free, and a row too long for one warp (unoriented graphs, a
// dense part of a sparse graph) is left to a second launch, a CTA per piece, after a look at the first one's
// totals: general path / one warp per row / this, us: one row of 60,000 among 319,000 arcs 360 / 6800 / 362, 30 of
// them 1485 / 26,400 / 650, both directions of R-MAT 16 ef12 2510 / 4450 / 1670, K_1800 in 60,000 vertices 2930 /
// 2000 / 940, 6000 rows of 200 in random order 244 / 352 / 235; pieces from 128 arcs on instead of 512: R-MAT 16
// 146 us.
#include <algorithm>
#include <type_traits>

#include "tc_count.h"
#include "tc_internal.h"
#include "tc_small.h"

namespace tc {

namespace {

constexpr int SM_WARPS = 8;
constexpr int SM_THREADS = 32 * SM_WARPS;

struct SmallArgs {
  const int64_t *beg;
  const int32_t *adj;
  int n, m;
  int row_lo, row_hi;
  int check_ids;
  int warp_max, cta_max;
  int splits;   // warps per row
  int words;    // bitmap words per warp; the last one stays zero (entries that are no ids)
  TcControl *acc;    // device accumulators, zero between calls.  bad_offset_at: CTAs finished and, from bit 32
                     // on, units: in the first line of what the host reads
  TcControl *out;    // pinned host block
  int2 *units;       // (row, first arc) of the long rows' pieces
};

// A row of which one warp would take more than LONG_PART arcs is left to long_rows_kernel, in pieces of
// 256 arcs (a batch per warp) or a 64th of the row (each piece makes the row's bitmap again).
constexpr int LONG_PART = 512;
constexpr int LONG_TARGET = 512;  // (tested for in the first kernel too: R-MAT 16 126 -> 129 us)
__device__ __forceinline__ int unit_arcs(int d) { return (d + 16383) / 16384 * 256; }
static_assert(SMALL_MAX_UNITS >= SMALL_MAX_ARCS / 256 + SMALL_MAX_ARCS / LONG_PART, "room in the context's list");

// A row that may be indexed: begin <= end inside the arc array.  Rows out of bounds are reported by
// the warp that owns them.
__device__ __forceinline__ int checked_row(const SmallArgs &p, int v, int &b) {
  const long long lo = tc_ld_nc(p.beg + v), hi = tc_ld_nc(p.beg + v + 1);
  b = (int)lo;
  if (lo < 0 || hi < lo || hi > p.m) return -1;
  return (int)(hi - lo);
}

// Hits of the rows of 32 arcs (the lane's: s, of dd entries; 0: no arc) in the bitmap `words`; `none` is the
// index of its last word, which is zero.
template <bool BIG>
__device__ __forceinline__ unsigned probe_rows(const int32_t *__restrict__ adj, const unsigned *words, unsigned none,
                                               int s, int dd) {
  const int lane = threadIdx.x & 31;
  const int grp = lane >> 3, gl = lane & 7;
  unsigned h = 0;
  // BIG: rows of LONG_TARGET entries or more by the whole warp, eight entries per lane and step
  unsigned big = BIG ? __ballot_sync(TC_FULL_MASK, dd >= LONG_TARGET) : 0u;
  if (big) {
    do {
      const int j = __ffs(big) - 1;
      big &= big - 1;
      const int32_t *row = adj + __shfl_sync(TC_FULL_MASK, s, j);
      const int dj = __shfl_sync(TC_FULL_MASK, dd, j);
      for (int k = lane; k - lane < dj; k += 256) {
        unsigned w[8];
#pragma unroll
        for (int r = 0; r < 8; ++r) w[r] = k + 32 * r < dj ? (unsigned)tc_ld_nc(row + k + 32 * r) : 0xffffffffu;
#pragma unroll
        for (int r = 0; r < 8; ++r) h += words[min(w[r] >> 5, none)] >> (w[r] & 31u) & 1u;
      }
    } while (big);
    if (dd >= LONG_TARGET) dd = 0;
  }
  // four rows at a time, eight lanes each: 64 entries of each per step while one has more than 32 left
  // (R-MAT 16 ef16 142 -> 126 us, ef28 261 -> 227), else 32
  const bool longer = __any_sync(TC_FULL_MASK, dd > 32);
  const unsigned have = __ballot_sync(TC_FULL_MASK, dd > 0);
  for (unsigned rest = have; rest;) {
    // the grp-th remaining row
    unsigned mine = rest;
    for (int k = 0; k < grp; ++k) mine &= mine - 1;
    const int j = mine ? __ffs(mine) - 1 : 0;
    const int sj = __shfl_sync(TC_FULL_MASK, s, j);
    int dj = __shfl_sync(TC_FULL_MASK, dd, j);
    if (!mine) dj = 0;
    auto walk = [&](int k, auto steps) {
      constexpr int U = decltype(steps)::value;
      unsigned w[U];
#pragma unroll
      for (int r = 0; r < U; ++r) w[r] = k + 8 * r < dj ? (unsigned)tc_ld_nc(adj + sj + k + 8 * r) : 0xffffffffu;
#pragma unroll
      for (int r = 0; r < U; ++r) h += words[min(w[r] >> 5, none)] >> (w[r] & 31u) & 1u;
    };
    int k = gl;
    if (longer)
      for (; __any_sync(TC_FULL_MASK, k + 32 < dj); k += 64) walk(k, std::integral_constant<int, 8>());
    for (; __any_sync(TC_FULL_MASK, k < dj); k += 32) walk(k, std::integral_constant<int, 4>());
#pragma unroll
    for (int k = 0; k < 4; ++k) rest &= rest - 1;
  }
  return h;
}

// The arcs at a0 + lane of row v (d entries from b on): checked, and where the row is counted probed.
template <bool BIG>
__device__ __forceinline__ void probe_arcs(const SmallArgs &p, const unsigned *words, unsigned none, bool counted, int b,
                                           int d, int a0, int &bad, unsigned long long &hits, unsigned long long &wedges) {
  const int i = a0 + (threadIdx.x & 31);
  int s = 0, dd = 0;
  if (i < d) {
    const int u = tc_ld_nc(p.adj + b + i);
    if ((unsigned)u >= (unsigned)p.n) bad |= p.check_ids ? TC_DEV_BAD_IDS : 0;
    else if (counted) dd = max(checked_row(p, u, s), 0);
  }
  if (!counted) return;
  wedges += (unsigned)dd;
  hits += probe_rows<BIG>(p.adj, words, none, s, dd);
}

// Sum a CTA's results into the accumulators; the last CTA hands the totals over and clears them for the
// next kernel.  All threads call it.
struct SmallSums {
  unsigned long long count, wedges;
  int bad, dmax, last;
  int hist[2][TC_NUM_CLASSES];
};
__device__ __forceinline__ void clear(SmallSums &cta) {
  if (threadIdx.x < 2 * TC_NUM_CLASSES) (&cta.hist[0][0])[threadIdx.x] = 0;
  if (threadIdx.x == 0) {
    cta.count = cta.wedges = 0;
    cta.bad = cta.dmax = 0;
  }
}
__device__ __forceinline__ void finish(const SmallArgs &p, SmallSums &cta, unsigned long long hits,
                                       unsigned long long wedges, int bad, int dmax) {
  bad = __reduce_or_sync(TC_FULL_MASK, bad);
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) {
    hits += __shfl_down_sync(TC_FULL_MASK, hits, o);
    wedges += __shfl_down_sync(TC_FULL_MASK, wedges, o);
  }
  if ((threadIdx.x & 31) == 0) {
    if (hits) atomicAdd(&cta.count, hits);
    if (wedges) atomicAdd(&cta.wedges, wedges);
    if (bad) atomicOr(&cta.bad, bad);
    atomicMax(&cta.dmax, dmax);
  }
  __syncthreads();
  if (threadIdx.x < TC_NUM_CLASSES) {
    if (cta.hist[0][threadIdx.x]) atomicAdd(&p.acc->class_count[threadIdx.x], cta.hist[0][threadIdx.x]);
    if (cta.hist[1][threadIdx.x]) atomicAdd(&p.acc->class_count_alt[threadIdx.x], cta.hist[1][threadIdx.x]);
  }
  if (threadIdx.x == 0) {
    if (cta.count) atomicAdd(&p.acc->count, cta.count);
    if (cta.wedges) atomicAdd(&p.acc->wedges, cta.wedges);
    if (cta.bad) atomicOr(&p.acc->status, cta.bad);
    if (cta.dmax) atomicMax(&p.acc->max_out_degree, cta.dmax);
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) cta.last = (unsigned)atomicAdd(&p.acc->bad_offset_at, 1ull) == gridDim.x - 1;
  __syncthreads();
  if (!cta.last) return;
  __threadfence();
  static_assert(sizeof(TcControl) % 8 == 0, "copied by 8-byte words");
  const unsigned long long *src = reinterpret_cast<const unsigned long long *>(p.acc);
  for (int i = threadIdx.x; i < (int)(sizeof(TcControl) / 8); i += SM_THREADS) {
    reinterpret_cast<unsigned long long *>(p.out)[i] = __ldcg(src + i);
    reinterpret_cast<unsigned long long *>(p.acc)[i] = 0;
  }
  __threadfence_system();
}

__global__ void __launch_bounds__(SM_THREADS, 6) small_kernel(SmallArgs p) {
  extern __shared__ unsigned bitmaps[];
  __shared__ SmallSums cta;
  __shared__ int next;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned *words = bitmaps + warp * p.words;
  const unsigned none = (unsigned)p.words - 1;
  for (int i = lane; i < p.words; i += 32) words[i] = 0;
  clear(cta);
  if (threadIdx.x == 0) {
    next = SM_WARPS;
    if (blockIdx.x == 0 && (tc_ld_nc(p.beg) != 0 || tc_ld_nc(p.beg + p.n) != p.m)) cta.bad = TC_DEV_BAD_OFFSETS;
  }
  __syncthreads();
  unsigned long long hits = 0, wedges = 0;
  int bad = 0, dmax = 0;
  const int tasks = p.n * p.splits, nwarps = gridDim.x * SM_WARPS;
  // the CTA's rows, in the order of the rounds, go to its warps as they finish
  auto claim = [&]() {
    int k = 0;
    if (lane == 0) k = atomicAdd(&next, 1);
    return __shfl_sync(TC_FULL_MASK, k, 0);
  };
  for (int k = warp; k / SM_WARPS * nwarps < tasks; k = claim()) {
    const int round = k / SM_WARPS, me = blockIdx.x * SM_WARPS + k % SM_WARPS;
    const int t = round * nwarps + (round & 1 ? nwarps - 1 - me : me);
    if (t >= tasks) continue;
    const int v = t / p.splits, part = t - v * p.splits;
    int b;
    int d = checked_row(p, v, b);
    if (d < 0) {
      // Rows that overlap (invalid offsets) can hold far more arcs than the graph, but there is a row out of order
      // between any two of them: a CTA that meets one claims no more.
      if (lane == 0) atomicMax(&next, SM_WARPS * tasks);
      bad |= TC_DEV_BAD_OFFSETS;
      continue;
    }
    dmax = max(dmax, d);
    const bool counted = v >= p.row_lo && v < p.row_hi && d >= 2;
    if (part == 0 && lane < 2) {  // the row's class under the tuned classes and under the plain split
      const bool plain = lane;
      const int wm = lane ? TC_PLAIN_WARP_MAX : p.warp_max;
      int c = TC_CLASS_SKIP;
      if (counted)
        c = plain ? (d <= wm ? TC_CLASS_WARP : d <= p.cta_max ? TC_CLASS_CTA : TC_CLASS_HUGE)
                  : (d <= 4    ? TC_CLASS_G4
                     : d <= 8  ? TC_CLASS_G8
                     : d <= 16 ? TC_CLASS_G16
                     : d <= 32 ? TC_CLASS_G32
                     : d <= wm ? TC_CLASS_WARP
                     : d <= p.cta_max ? TC_CLASS_CTA
                                      : TC_CLASS_HUGE);
      atomicAdd(&cta.hist[lane][c], 1);
    }
    if (part * 32 >= d || (!counted && !p.check_ids)) continue;
    if (d > LONG_PART * p.splits) {
      if (part == 0) {
        const int per = unit_arcs(d), k = (d + per - 1) / per;
        unsigned long long at = 0;
        if (lane == 0) at = atomicAdd(&p.acc->bad_offset_at, (unsigned long long)k << 32) >> 32;
        at = __shfl_sync(TC_FULL_MASK, at, 0);
        if (at + k > SMALL_MAX_UNITS) bad |= TC_DEV_BAD_OFFSETS;  // rows that overlap
        else
          for (int j = lane; j < k; j += 32) p.units[at + j] = make_int2(v, j * per);
      }
      continue;
    }
    if (counted) {
      for (int i = lane; i < d; i += 32) {
        const unsigned w = (unsigned)tc_ld_nc(p.adj + b + i);
        if (w < (unsigned)p.n) atomicOr(words + (w >> 5), 1u << (w & 31u));
      }
      __syncwarp();
    }
    for (int a0 = part * 32; a0 < d; a0 += 32 * p.splits) probe_arcs<false>(p, words, none, counted, b, d, a0, bad, hits, wedges);
    if (counted) {
      __syncwarp();
      for (int i = lane; i < d; i += 32) {
        const unsigned w = (unsigned)tc_ld_nc(p.adj + b + i);
        if (w < (unsigned)p.n) words[w >> 5] = 0;
      }
      __syncwarp();
    }
  }
  finish(p, cta, hits, wedges, bad, dmax);
}

// The long rows' pieces, a CTA each: the row's bitmap once, its 32-arc batches dealt to the warps.
__global__ void __launch_bounds__(SM_THREADS, 6) long_rows_kernel(SmallArgs p, int n_units) {
  extern __shared__ unsigned words[];
  __shared__ SmallSums cta;
  const unsigned none = (unsigned)p.words - 1;
  for (int i = threadIdx.x; i < p.words; i += SM_THREADS) words[i] = 0;
  clear(cta);
  __syncthreads();
  unsigned long long hits = 0, wedges = 0;
  int bad = 0;
  for (int t = blockIdx.x; t < n_units; t += gridDim.x) {
    const int2 unit = p.units[t];
    int b;
    const int d = checked_row(p, unit.x, b);
    const bool counted = unit.x >= p.row_lo && unit.x < p.row_hi && d >= 2;
    if (counted) {
#pragma unroll 4
      for (int i = threadIdx.x; i < d; i += SM_THREADS) {
        const unsigned w = (unsigned)tc_ld_nc(p.adj + b + i);
        if (w < (unsigned)p.n) atomicOr(words + (w >> 5), 1u << (w & 31u));
      }
      __syncthreads();
    }
    for (int a0 = unit.y + (threadIdx.x & ~31); a0 < min(d, unit.y + unit_arcs(d)); a0 += SM_THREADS)
      probe_arcs<true>(p, words, none, counted, b, d, a0, bad, hits, wedges);
    if (counted) {
      __syncthreads();
      for (int i = threadIdx.x; i < p.words; i += SM_THREADS) words[i] = 0;
      __syncthreads();
    }
  }
  finish(p, cta, hits, wedges, bad, 0);
}

}  // namespace

bool small_graph(int64_t n, int64_t m) { return n >= 1 && n <= SMALL_MAX_IDS && m <= SMALL_MAX_ARCS; }

int small_count(trust_tc_ctx *c, const int64_t *beg, const int32_t *adj, int64_t n, int64_t m, int64_t row_lo,
                int64_t row_hi, int check_ids, int warp_max, int cta_max, cudaStream_t st) {
  if (!c->small_zeroed) {
    TC_CUDA_TRY(cudaStreamSynchronize(c->copy_stream));
    c->small_zeroed = true;
  }
  SmallArgs a;
  a.beg = beg;
  a.adj = adj;
  a.n = (int)n;
  a.m = (int)m;
  a.row_lo = (int)row_lo;
  a.row_hi = (int)row_hi;
  a.check_ids = check_ids;
  a.warp_max = warp_max;
  a.cta_max = cta_max;
  // rows of few batches: a warp each; dense graphs: several warps share a row's batches
  a.splits = (int)std::min<int64_t>(8, std::max<int64_t>(1, m / (16 * n)));
  a.words = (int)(n / 32 + 2);
  a.acc = c->d_small;
  a.out = c->h_ctl;
  a.units = c->d_small_units;
  const int64_t tasks = n * a.splits;
  const size_t smem = sizeof(unsigned) * (size_t)a.words * SM_WARPS;
  TC_CUDA_TRY(cudaFuncSetAttribute(small_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)sizeof(unsigned) * (SMALL_MAX_IDS / 32 + 2) * SM_WARPS));
  const int per_sm = (int)std::min<size_t>(6, (size_t)220 * 1024 / (smem + 1536));  // resident CTAs
  const int blocks = (int)std::min<int64_t>((tasks + SM_WARPS - 1) / SM_WARPS, (int64_t)c->num_sms * per_sm);
  small_kernel<<<blocks, SM_THREADS, smem, st>>>(a);
  note_launch();
  TC_CUDA_TRY(cudaGetLastError());
  TC_CUDA_TRY(cudaEventRecord(c->ev[4], st));
  TC_CUDA_TRY(cudaStreamSynchronize(st));
  const int n_units = (int)(c->h_ctl->bad_offset_at >> 32);
  if (n_units == 0 || c->h_ctl->status) return TRUST_TC_OK;
  const TcControl rest = *c->h_ctl;
  long_rows_kernel<<<std::min(n_units, c->num_sms * 6), SM_THREADS, sizeof(unsigned) * (size_t)a.words, st>>>(a, n_units);
  note_launch();
  TC_CUDA_TRY(cudaGetLastError());
  TC_CUDA_TRY(cudaEventRecord(c->ev[4], st));
  TC_CUDA_TRY(cudaStreamSynchronize(st));
  const TcControl pieces = *c->h_ctl;
  *c->h_ctl = rest;
  c->h_ctl->count += pieces.count;
  c->h_ctl->wedges += pieces.wedges;
  c->h_ctl->status |= pieces.status;
  return TRUST_TC_OK;
}

}  // namespace tc
