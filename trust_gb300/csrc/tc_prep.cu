// tc_prep.cu — GPU preprocessing: edge pairs -> oriented, renumbered CSR.
//
// Moves the reference's CPU preprocessing onto the GPU:
//   Preprocess/fromDirectToUndirect.cpp:53-109  compact ids, (min,max) pairs, dedupe
//   Preprocess/preprocess_outdegree.cpp:79-98   orient each edge from lower to higher degree
//   Preprocess/preprocess_outdegree.cpp:186-222 renumber (out-degree descending) and write CSR
// with two deliberate changes: ties are broken by vertex id (the reference's std::sort leaves
// them unspecified) and each row is sorted ascending (the reference writes rows unsorted, :213).
// Vertices without edges are dropped (the reference keeps a self-loop-only vertex as an isolated
// row).  Every step is a stable LSD radix sort, a scan, or an elementwise kernel.
#include <algorithm>
#include <vector>

#include "tc_internal.h"

namespace tc {

typedef unsigned long long u64;
typedef unsigned int u32;

constexpr int RS_THREADS = 256;
constexpr int RS_ITEMS = 16;
constexpr int RS_TILE = RS_THREADS * RS_ITEMS;  // keys per CTA per pass

// ------------------------------------------------------------------------------------------
// scans (exclusive, tile of 4096 per CTA, reduce-then-scan)
// ------------------------------------------------------------------------------------------
template <typename T>
__device__ T block_excl_scan(T x, T *total) {
  __shared__ T warp_tot[RS_THREADS / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  T incl = x;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    T y = __shfl_up_sync(TC_FULL_MASK, incl, off);
    if (lane >= off) incl += y;
  }
  if (lane == 31) warp_tot[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    T w = lane < RS_THREADS / 32 ? warp_tot[lane] : T(0);
    T wi = w;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      T y = __shfl_up_sync(TC_FULL_MASK, wi, off);
      if (lane >= off) wi += y;
    }
    if (lane < RS_THREADS / 32) warp_tot[lane] = wi - w;
    if (lane == RS_THREADS / 32 - 1) *total = wi;
  }
  __syncthreads();
  T r = warp_tot[warp] + incl - x;
  __syncthreads();
  return r;
}

template <typename T>
__global__ void scan_reduce_kernel(const T *__restrict__ in, int64_t n, T *__restrict__ sums) {
  __shared__ T tot;
  const int64_t base = (int64_t)blockIdx.x * RS_TILE + (int64_t)threadIdx.x * RS_ITEMS;
  T s = 0;
#pragma unroll
  for (int j = 0; j < RS_ITEMS; ++j)
    if (base + j < n) s += in[base + j];
  block_excl_scan<T>(s, &tot);
  if (threadIdx.x == 0) sums[blockIdx.x] = tot;
}

template <typename T>
__global__ void scan_down_kernel(const T *in, T *out, int64_t n, const T *__restrict__ offs) {
  __shared__ T tot;
  const int64_t base = (int64_t)blockIdx.x * RS_TILE + (int64_t)threadIdx.x * RS_ITEMS;
  T v[RS_ITEMS];
  T s = 0;
#pragma unroll
  for (int j = 0; j < RS_ITEMS; ++j) {
    v[j] = base + j < n ? in[base + j] : T(0);
    s += v[j];
  }
  T run = block_excl_scan<T>(s, &tot) + (offs ? offs[blockIdx.x] : T(0));
#pragma unroll
  for (int j = 0; j < RS_ITEMS; ++j) {
    if (base + j < n) out[base + j] = run;
    run += v[j];
  }
}

// Exclusive scan of n elements (in may equal out).  Returns the total through *total_out
// (device-to-host read, synchronising `st`) when total_out is not null.
template <typename T>
static int scan_exclusive(const T *in, T *out, int64_t n, cudaStream_t st, T *total_out) {
  if (n <= 0) {
    if (total_out) *total_out = 0;
    return TRUST_TC_OK;
  }
  T last_in = 0;
  if (total_out) TC_CUDA_TRY(cudaMemcpyAsync(&last_in, in + n - 1, sizeof(T), cudaMemcpyDeviceToHost, st));
  if (total_out) TC_CUDA_TRY(cudaStreamSynchronize(st));
  const int64_t nb = (n + RS_TILE - 1) / RS_TILE;
  T *sums = nullptr;
  if (nb > 1) {
    TC_CUDA_TRY(cudaMallocAsync((void **)&sums, sizeof(T) * nb, st));
    scan_reduce_kernel<T><<<(unsigned)nb, RS_THREADS, 0, st>>>(in, n, sums);
    TC_NOTE_LAUNCH();
    TC_CUDA_TRY(cudaGetLastError());
    int rc = scan_exclusive<T>(sums, sums, nb, st, (T *)nullptr);
    if (rc) return rc;
  }
  scan_down_kernel<T><<<(unsigned)nb, RS_THREADS, 0, st>>>(in, out, n, sums);
  TC_NOTE_LAUNCH();
  TC_CUDA_TRY(cudaGetLastError());
  if (sums) TC_CUDA_TRY(cudaFreeAsync(sums, st));
  if (total_out) {
    T last_out = 0;
    TC_CUDA_TRY(cudaMemcpyAsync(&last_out, out + n - 1, sizeof(T), cudaMemcpyDeviceToHost, st));
    TC_CUDA_TRY(cudaStreamSynchronize(st));
    *total_out = last_out + last_in;
  }
  return TRUST_TC_OK;
}

size_t scan_u32_scratch(int64_t n) {
  size_t words = 0;
  for (int64_t nb = (n + RS_TILE - 1) / RS_TILE; nb > 1; nb = (nb + RS_TILE - 1) / RS_TILE) words += (size_t)nb;
  return words;
}

int scan_exclusive_u32(const unsigned *in, unsigned *out, int64_t n, unsigned *scratch, cudaStream_t st) {
  if (n <= 0) return TRUST_TC_OK;
  const int64_t nb = (n + RS_TILE - 1) / RS_TILE;
  if (nb > 1) {
    scan_reduce_kernel<u32><<<(unsigned)nb, RS_THREADS, 0, st>>>(in, n, scratch);
    TC_NOTE_LAUNCH();
    TC_CUDA_TRY(cudaGetLastError());
    int rc = scan_exclusive_u32(scratch, scratch, nb, scratch + nb, st);
    if (rc) return rc;
  }
  scan_down_kernel<u32><<<(unsigned)nb, RS_THREADS, 0, st>>>(in, out, n, nb > 1 ? scratch : nullptr);
  TC_NOTE_LAUNCH();
  TC_CUDA_TRY(cudaGetLastError());
  return TRUST_TC_OK;
}

int scan_exclusive_i64(const int64_t *in, int64_t *out, int64_t n, cudaStream_t st, int64_t *total) {
  return scan_exclusive<int64_t>(in, out, n, st, total);
}

// ------------------------------------------------------------------------------------------
// stable LSD radix sort of u64 keys, 8-bit digits
// ------------------------------------------------------------------------------------------
// Per pass: digit counts of every tile, one scan over [digit][tile], and a scatter that first
// orders the tile in shared memory, so that the keys of one digit leave as one contiguous run (16
// keys, 128 bytes, on average) instead of single 8-byte writes.  Each warp ranks 256 consecutive
// keys with ballots and counters of its own: no atomics, and six barriers per 4096 keys instead of
// two per 256.  Bound by the load/store pipe (66 % busy: shared-memory scatter and the runs' ragged
// ends) as much as by memory (a pass moves 24 bytes per key).  268 M keys on GB300: scatter 0.98 ms
// and counts 0.26, against 1.77 and 0.28 with single writes; tiles of 6144 keys (two CTAs of 512
// threads per SM instead of three) were 2 % slower, a match instruction instead of the ballots equal.
constexpr int SORT_WARPS = 16;
constexpr int SORT_THREADS = 32 * SORT_WARPS;
constexpr int SORT_ITEMS = 8;                          // keys per lane
constexpr int SORT_TILE = SORT_THREADS * SORT_ITEMS;    // keys per CTA
constexpr size_t SORT_SMEM = sizeof(u64) * SORT_TILE;

// Edge pair i as a canonical key (min << bits | max); self-loops and ids out of range become the
// largest key, which no valid pair has (its ends would be equal).
template <bool WIDE>  // pairs are 8-byte aligned
struct PairKeys {
  const int32_t *pairs;
  u32 bound;      // exclusive id bound
  u32 shift_mul;  // 2^bits
  u64 invalid;    // 2^(2 bits) - 1
  __device__ __forceinline__ u64 operator()(int64_t i) const {
    int u, v;
    if (WIDE) {
      const int2 p = __ldg(reinterpret_cast<const int2 *>(pairs) + i);
      u = p.x;
      v = p.y;
    } else {
      u = __ldg(pairs + 2 * i);
      v = __ldg(pairs + 2 * i + 1);
    }
    const u32 lo = min((u32)u, (u32)v), hi = max((u32)u, (u32)v);  // (negative ids are above any bound)
    return lo != hi && hi < bound ? (u64)lo * shift_mul + hi : invalid;
  }
};
struct PlainKeys {
  const u64 *keys;
  __device__ __forceinline__ u64 operator()(int64_t i) const { return keys[i]; }
};

// 8-bit digit at a shift that is a multiple of 8.
__device__ __forceinline__ u32 digit_at(u64 k, int byte) {
  return __byte_perm((u32)k, (u32)(k >> 32), (u32)byte) & 255u;
}

template <class In>
__global__ void __launch_bounds__(SORT_THREADS) sort_hist_kernel(In in, int64_t n, int byte, u32 *__restrict__ counts,
                                                                 u32 ntiles) {
  __shared__ u32 h[2][256];  // two copies: half the conflicts on a popular digit
  for (int i = threadIdx.x; i < 512; i += SORT_THREADS) (&h[0][0])[i] = 0;
  __syncthreads();
  const int64_t base = (int64_t)blockIdx.x * SORT_TILE;
  const int have = (int)min((int64_t)SORT_TILE, n - base);
  u32 *mine = h[threadIdx.x & 1];
  u64 k[SORT_ITEMS];
#pragma unroll
  for (int j = 0; j < SORT_ITEMS; ++j) k[j] = in(base + min(j * SORT_THREADS + (int)threadIdx.x, have - 1));
#pragma unroll
  for (int j = 0; j < SORT_ITEMS; ++j)
    if (j * SORT_THREADS + (int)threadIdx.x < have) atomicAdd(mine + digit_at(k[j], byte), 1u);
  __syncthreads();
  for (int d = threadIdx.x; d < 256; d += SORT_THREADS) counts[(size_t)d * ntiles + blockIdx.x] = h[0][d] + h[1][d];
}

// LOW: write the low 32 bits under `low_mask` only (the last pass of the arc sort writes the CSR's
// neighbour array itself).
template <class In, bool LOW>
__global__ void __launch_bounds__(SORT_THREADS, 3) sort_scatter_kernel(In in, void *__restrict__ out, int64_t n, int byte,
                                                                       const u32 *__restrict__ offs, u32 ntiles,
                                                                       u32 low_mask) {
  extern __shared__ __align__(16) u64 sorted[];
  __shared__ unsigned short cnt[SORT_WARPS][256];  // then: first place in the tile of the warp's keys of a digit
  __shared__ u32 gbase[256];                       // a digit's place in the output, minus its place in the tile
  __shared__ u32 wtot[8];
  static_assert(SORT_THREADS >= 256, "a thread per digit");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned lt = tc_lanemask_lt();
  for (int i = threadIdx.x; i < SORT_WARPS * 128; i += SORT_THREADS) reinterpret_cast<u32 *>(cnt)[i] = 0;
  const int64_t base = (int64_t)blockIdx.x * SORT_TILE;
  const int have = (int)min((int64_t)SORT_TILE, n - base);
  const int first = warp * (32 * SORT_ITEMS) + lane;
  u64 key[SORT_ITEMS];
  u32 rank[SORT_ITEMS / 2];  // two 16-bit ranks each
#pragma unroll
  for (int j = 0; j < SORT_ITEMS; ++j) key[j] = in(base + min(first + 32 * j, have - 1));
  u32 my_gbase = 0;
  if (threadIdx.x < 256) my_gbase = offs[(size_t)threadIdx.x * ntiles + blockIdx.x];
  __syncthreads();
#pragma unroll
  for (int j = 0; j < SORT_ITEMS; ++j) {
    const bool valid = first + 32 * j < have;
    const u32 d = digit_at(key[j], byte);
    unsigned peers = __ballot_sync(TC_FULL_MASK, valid);
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      const bool one = d & (1u << b);
      const unsigned set = __ballot_sync(TC_FULL_MASK, one);
      peers &= one ? set : ~set;
    }
    const u32 before = __popc(peers & lt);
    const u32 seen = cnt[warp][d];
    if (j & 1) rank[j / 2] |= (seen + before) << 16;
    else rank[j / 2] = seen + before;
    __syncwarp();
    if (valid && before == 0) cnt[warp][d] = (unsigned short)(seen + __popc(peers));
    __syncwarp();
  }
  __syncthreads();
  u32 tot = 0, incl = 0;
  if (threadIdx.x < 256) {  // digit threadIdx.x: totals over the warps, then over the digits
#pragma unroll
    for (int w = 0; w < SORT_WARPS; ++w) tot += cnt[w][threadIdx.x];
    incl = tot;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const u32 y = __shfl_up_sync(TC_FULL_MASK, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) wtot[warp] = incl;
  }
  __syncthreads();
  if (threadIdx.x < 256) {
    u32 s = incl - tot;
    for (int w = 0; w < warp; ++w) s += wtot[w];
    gbase[threadIdx.x] = my_gbase - s;
#pragma unroll
    for (int w = 0; w < SORT_WARPS; ++w) {
      const u32 c = cnt[w][threadIdx.x];
      cnt[w][threadIdx.x] = (unsigned short)s;
      s += c;
    }
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < SORT_ITEMS; ++j)
    if (first + 32 * j < have)
      sorted[cnt[warp][digit_at(key[j], byte)] + (j & 1 ? rank[j / 2] >> 16 : rank[j / 2] & 0xffffu)] = key[j];
  __syncthreads();
#pragma unroll
  for (int j = 0; j < SORT_ITEMS; ++j) {
    const int i = j * SORT_THREADS + (int)threadIdx.x;
    if (i < have) {
      const u64 k = sorted[i];
      const u32 at = gbase[digit_at(k, byte)] + (u32)i;
      if (LOW) reinterpret_cast<int32_t *>(out)[at] = (int32_t)((u32)k & low_mask);
      else reinterpret_cast<u64 *>(out)[at] = k;
    }
  }
}

static u32 sort_tiles(int64_t n) { return (u32)((n + SORT_TILE - 1) / SORT_TILE); }

// counts of one pass, and the scan's scratch after them (u32 words)
static size_t sort_scratch(int64_t n) { return 256 * (size_t)sort_tiles(n) + scan_u32_scratch(256 * (int64_t)sort_tiles(n)); }

template <class In, bool LOW = false>
static int sort_pass(In in, void *out, int64_t n, int shift, u32 *scratch, cudaStream_t st, u32 low_mask = 0) {
  const u32 nt = sort_tiles(n);
  u32 *counts = scratch;
  TC_CUDA_TRY(cudaFuncSetAttribute(sort_scatter_kernel<In, LOW>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)SORT_SMEM));
  sort_hist_kernel<<<nt, SORT_THREADS, 0, st>>>(in, n, shift / 8, counts, nt);
  TC_NOTE_LAUNCH();
  TC_CUDA_TRY(cudaGetLastError());
  int rc = scan_exclusive_u32(counts, counts, 256 * (int64_t)nt, scratch + 256 * (size_t)nt, st);
  if (rc) return rc;
  sort_scatter_kernel<In, LOW><<<nt, SORT_THREADS, SORT_SMEM, st>>>(in, out, n, shift / 8, counts, nt, low_mask);
  TC_NOTE_LAUNCH();
  TC_CUDA_TRY(cudaGetLastError());
  return TRUST_TC_OK;
}

// Sort n (< 2^32) keys by bits [lo, lo + bits) (lo a multiple of 8) through two buffers; *sorted is the one that holds
// the result.
static int sort_bits(u64 *keys, u64 *tmp, int64_t n, int lo, int bits, u32 *scratch, cudaStream_t st, u64 **sorted) {
  u64 *src = keys, *dst = tmp;
  for (int b = 0; b < bits && n > 1; b += 8) {
    int rc = sort_pass(PlainKeys{src}, dst, n, lo + b, scratch, st);
    if (rc) return rc;
    std::swap(src, dst);
  }
  *sorted = src;
  return TRUST_TC_OK;
}

static int bits_for(int64_t x) {  // bits needed to represent values in [0, x]
  int b = 1;
  while (b < 63 && ((int64_t)1 << b) <= x) ++b;
  return b;
}

// ------------------------------------------------------------------------------------------
// pipeline kernels
// ------------------------------------------------------------------------------------------
#define GRID_STRIDE(i, n) \
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < (n); i += (int64_t)gridDim.x * blockDim.x)

// First of a run of equal keys, invalid pairs (the largest key) left out.
__device__ __forceinline__ bool unique_at(const u64 *__restrict__ keys, int64_t i, int64_t n, u64 invalid, u64 *key) {
  if (i >= n) return false;
  const u64 k = keys[i];
  *key = k;
  return k != invalid && (i == 0 || keys[i - 1] != k);
}

__global__ void __launch_bounds__(RS_THREADS) unique_count_kernel(const u64 *__restrict__ keys, int64_t n, u64 invalid,
                                                                  u32 *__restrict__ counts) {
  __shared__ u32 tot;
  if (threadIdx.x == 0) tot = 0;
  __syncthreads();
  const int64_t base = (int64_t)blockIdx.x * RS_TILE;
  u32 c = 0;
#pragma unroll
  for (int r = 0; r < RS_ITEMS; ++r) {
    u64 k;
    c += unique_at(keys, base + r * RS_THREADS + threadIdx.x, n, invalid, &k);
  }
  c = __reduce_add_sync(TC_FULL_MASK, c);
  if ((threadIdx.x & 31) == 0) atomicAdd(&tot, c);
  __syncthreads();
  if (threadIdx.x == 0) counts[blockIdx.x] = tot;
}

// Unique keys in order, and the degrees of both ends.  The keys are sorted by their smaller end, so
// a warp adds each run of it with one atomic; the larger ends are spread over the graph.
__global__ void __launch_bounds__(RS_THREADS) unique_write_kernel(const u64 *__restrict__ keys, int64_t n, u64 invalid,
                                                                  int bits, const u32 *__restrict__ offs,
                                                                  u64 *__restrict__ out, u32 *__restrict__ deg) {
  __shared__ u32 wcnt[RS_ITEMS][RS_THREADS / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned lt = tc_lanemask_lt();
  const int64_t base = (int64_t)blockIdx.x * RS_TILE;
  u64 key[RS_ITEMS];
  unsigned flags = 0, ballots[RS_ITEMS];
#pragma unroll
  for (int r = 0; r < RS_ITEMS; ++r) {
    key[r] = invalid;
    const bool u = unique_at(keys, base + r * RS_THREADS + threadIdx.x, n, invalid, &key[r]);
    ballots[r] = __ballot_sync(TC_FULL_MASK, u);
    if (u) flags |= 1u << r;
    if (lane == 0) wcnt[r][warp] = __popc(ballots[r]);
  }
  __syncthreads();
  // exclusive scan of the 16 x 8 warp counts, in key order, by the first warp (four each)
  if (warp == 0) {
    u32 *w = &wcnt[0][0];
    u32 v[4], s = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      v[j] = w[4 * lane + j];
      s += v[j];
    }
    u32 incl = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const u32 y = __shfl_up_sync(TC_FULL_MASK, incl, o);
      if (lane >= o) incl += y;
    }
    u32 run = incl - s + offs[blockIdx.x];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      w[4 * lane + j] = run;
      run += v[j];
    }
  }
  __syncthreads();
  const u64 low = ((u64)1 << bits) - 1;
#pragma unroll
  for (int r = 0; r < RS_ITEMS; ++r) {
    const bool u = flags >> r & 1;
    const u32 a = (u32)(key[r] >> bits);
    if (u) {
      out[wcnt[r][warp] + __popc(ballots[r] & lt)] = key[r];
      atomicAdd(deg + (u32)(key[r] & low), 1u);
    }
    // runs of the smaller end among the warp's 32 keys (duplicates carry their run's end too)
    const u32 prev = __shfl_up_sync(TC_FULL_MASK, a, 1);
    const unsigned heads = __ballot_sync(TC_FULL_MASK, lane == 0 || a != prev);
    if (heads >> lane & 1) {
      const unsigned after = lane == 31 ? 0u : heads & ~(lt | (1u << lane));
      const unsigned run = (after ? (1u << (__ffs(after) - 1)) - 1u : 0xffffffffu) & ~lt;
      const u32 c = __popc(ballots[r] & run);
      if (c) atomicAdd(deg + a, c);
    }
  }
}

__global__ void present_kernel(const u32 *__restrict__ deg, int64_t n, u32 *flags) {
  GRID_STRIDE(i, n) { flags[i] = deg[i] > 0; }
}

// Orient every edge from its lower to its higher end by (degree, id); keys hold the smaller id
// first, so equal degrees keep the order.  Out-degrees on the way, by id or, with cid, by compacted id.
__global__ void orient_kernel(u64 *__restrict__ e, const u32 *__restrict__ n_edges, int bits,
                              const u32 *__restrict__ deg, const u32 *__restrict__ cid, u32 *__restrict__ od) {
  const u64 low = ((u64)1 << bits) - 1;
  const int64_t ne = *n_edges, stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < ne; i += 4 * stride) {
    u64 k[4];
    u32 da[4], db[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) k[r] = i + r * stride < ne ? e[i + r * stride] : 0;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      da[r] = __ldg(deg + (u32)(k[r] >> bits));
      db[r] = __ldg(deg + (u32)(k[r] & low));
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      if (i + r * stride >= ne) break;
      const u64 a = k[r] >> bits, b = k[r] & low;
      if (da[r] > db[r]) e[i + r * stride] = b << bits | a;
      const u32 source = (u32)(da[r] > db[r] ? b : a);
      atomicAdd(od + (cid ? __ldg(cid + source) : source), 1u);
    }
  }
}

__global__ void max_kernel(const u32 *__restrict__ x, int64_t n, u32 *mx) {
  u32 m = 0;
  GRID_STRIDE(i, n) { m = max(m, x[i]); }
  m = __reduce_max_sync(TC_FULL_MASK, m);
  if ((threadIdx.x & 31) == 0 && m) atomicMax(mx, m);
}

// Present vertices in id order, keyed for the renumbering (out-degree, descending).
__global__ void renumber_key_kernel(const u32 *__restrict__ deg, const u32 *__restrict__ od, const u32 *__restrict__ cid,
                                    int64_t id_bound, bool od_compact, u32 odmax, u64 *vkeys) {
  GRID_STRIDE(x, id_bound) {
    if (deg[x]) vkeys[cid[x]] = ((u64)(odmax - od[od_compact ? cid[x] : x]) << 32) | (u64)x;
  }
}

// New ids in that order, and the new rows' lengths (entry n: 0).
__global__ void newid_kernel(const u64 *__restrict__ vkeys, int64_t n, u32 odmax, u32 *__restrict__ newid,
                             int64_t *__restrict__ len) {
  GRID_STRIDE(p, n + 1) {
    if (p == n) {
      len[p] = 0;
    } else {
      const u64 k = vkeys[p];
      newid[k & 0xffffffffu] = (u32)p;
      len[p] = odmax - (u32)(k >> 32);
    }
  }
}

// Original order kept: the new ids are cid, the rows' lengths the out-degrees of present vertices.
__global__ void kept_len_kernel(const u32 *__restrict__ deg, const u32 *__restrict__ od, const u32 *__restrict__ cid,
                                int64_t id_bound, bool od_compact, int64_t n, int64_t *__restrict__ len) {
  GRID_STRIDE(x, id_bound) {
    if (deg[x]) len[cid[x]] = od[od_compact ? cid[x] : x];
    if (x == 0) len[n] = 0;
  }
}

__global__ void relabel_kernel(u64 *__restrict__ e, int64_t ne, int bits, int nbits, const u32 *__restrict__ newid) {
  const u64 low = ((u64)1 << bits) - 1;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < ne; i += 4 * stride) {
    u64 k[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) k[r] = i + r * stride < ne ? e[i + r * stride] : 0;
#pragma unroll
    for (int r = 0; r < 4; ++r)
      k[r] = (u64)__ldg(newid + (u32)(k[r] >> bits)) << nbits | __ldg(newid + (u32)(k[r] & low));
#pragma unroll
    for (int r = 0; r < 4; ++r)
      if (i + r * stride < ne) e[i + r * stride] = k[r];
  }
}

static int grid_for(int64_t n) { return (int)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, 152 * 32)); }

// ------------------------------------------------------------------------------------------
// host pipeline
// ------------------------------------------------------------------------------------------
struct DevBufs {
  std::vector<void *> ptrs;
  cudaStream_t st;
  ~DevBufs() {
    for (void *p : ptrs) cudaFreeAsync(p, st);
  }
  template <typename T>
  int get(T **p, int64_t count) {
    *p = nullptr;
    cudaError_t e = cudaMallocAsync((void **)p, sizeof(T) * (size_t)std::max<int64_t>(count, 1), st);
    if (e != cudaSuccess) return cuda_status(e);
    ptrs.push_back(*p);
    return TRUST_TC_OK;
  }
};

// seg_out[g] = compacted id of the first vertex at or after original id seg_in[g] (the present
// vertices before it), or n for seg_in[g] >= id_bound
__global__ void seg_map_kernel(const u32 *__restrict__ cid, int64_t id_bound, int64_t n,
                               const int64_t *__restrict__ seg_in, int64_t nseg, int64_t *seg_out) {
  GRID_STRIDE(g, nseg) {
    const int64_t x = seg_in[g];
    seg_out[g] = x >= id_bound ? n : (x <= 0 ? 0 : (int64_t)cid[x]);
  }
}

// keep_order: new ids are the compacted ids (original order kept, isolated vertices dropped)
// instead of the out-degree-descending renumbering; with d_seg_in / d_seg_out (nseg entries, on
// the device) the original-id boundaries of segments are mapped to the new ids.
int build_csr_device(const int32_t *d_pairs, int64_t np, int64_t id_bound, int64_t **d_beg_out,
                     int32_t **d_adj_out, int64_t *n_out, int64_t *m_out, cudaStream_t st, bool keep_order,
                     const int64_t *d_seg_in, int64_t nseg, int64_t *d_seg_out) {
  if (np < 0 || id_bound < 1 || id_bound >= ((int64_t)1 << 31)) return TRUST_TC_E_ARG;
  if (np >= ((int64_t)1 << 32) - 1) return TRUST_TC_E_TOO_LARGE;
  DevBufs B;
  B.st = st;
  int rc;
  u64 *keys, *tmp;
  u32 *scratch, *small, *deg, *cid, *od, *newid;
  const int bits = bits_for(id_bound - 1);
  const int64_t ntile = std::max<int64_t>((np + RS_TILE - 1) / RS_TILE, 1);
  // Ids far apart (more of them than edges have ends): out-degrees by compacted id, so that one less array
  // of id_bound entries is mapped, cleared and read: 1000 pairs with ids below 2^31 75 -> 54 ms, below 2^28
  // 10.1 -> 7.4.  Otherwise by id: no gather per edge.
  const bool sparse_ids = id_bound > 2 * np;
  const int64_t n_most = std::min(id_bound, 2 * np);
  const int64_t od_count = sparse_ids ? n_most : id_bound;
  const size_t words = std::max(std::max(sort_scratch(np), (size_t)ntile + 1 + scan_u32_scratch(ntile + 1)),
                                std::max(sort_scratch(n_most), scan_u32_scratch(id_bound + 1)));
  if ((rc = B.get(&keys, np)) || (rc = B.get(&tmp, np)) || (rc = B.get(&scratch, (int64_t)words)) ||
      (rc = B.get(&small, 4)) || (rc = B.get(&deg, id_bound)) || (rc = B.get(&cid, id_bound + 1)) ||
      (rc = B.get(&od, od_count)))
    return rc;
  // 1. canonical (min,max) keys, sorted (the first pass reads the pairs); invalid pairs sort last
  const u64 invalid = ((u64)1 << (2 * bits)) - 1;
  u64 *cur = keys, *other = tmp;
  if (np > 0) {
    rc = ((uintptr_t)d_pairs & 7) == 0
             ? sort_pass(PairKeys<true>{d_pairs, (u32)id_bound, 1u << bits, invalid}, cur, np, 0, scratch, st)
             : sort_pass(PairKeys<false>{d_pairs, (u32)id_bound, 1u << bits, invalid}, cur, np, 0, scratch, st);
    if (rc) return rc;
    if ((rc = sort_bits(cur, other, np, 8, 2 * bits - 8, scratch, st, &cur))) return rc;
    other = cur == keys ? tmp : keys;
  }
  // 2. unique edges and degrees
  TC_CUDA_TRY(cudaMemsetAsync(deg, 0, sizeof(u32) * id_bound, st));
  TC_CUDA_TRY(cudaMemsetAsync(od, 0, sizeof(u32) * (size_t)std::max<int64_t>(od_count, 1), st));
  TC_CUDA_TRY(cudaMemsetAsync(scratch, 0, sizeof(u32) * (size_t)(ntile + 1), st));
  unique_count_kernel<<<(unsigned)ntile, RS_THREADS, 0, st>>>(cur, np, invalid, scratch);
  TC_NOTE_LAUNCH();
  TC_CUDA_TRY(cudaGetLastError());
  if ((rc = scan_exclusive_u32(scratch, scratch, ntile + 1, scratch + ntile + 1, st))) return rc;
  u64 *e = other;  // unique edges live there from here on
  unique_write_kernel<<<(unsigned)ntile, RS_THREADS, 0, st>>>(cur, np, invalid, bits, scratch, e, deg);
  TC_NOTE_LAUNCH();
  TC_CUDA_TRY(cudaGetLastError());
  // 3. compacted ids (vertices without edges dropped); orientation by (degree, id)
  TC_CUDA_TRY(cudaMemcpyAsync(small, scratch + ntile, sizeof(u32), cudaMemcpyDeviceToDevice, st));
  TC_CUDA_TRY(cudaMemsetAsync(small + 2, 0, sizeof(u32), st));
  present_kernel<<<grid_for(id_bound), 256, 0, st>>>(deg, id_bound, cid);
  TC_NOTE_LAUNCH();
  TC_CUDA_TRY(cudaMemsetAsync(cid + id_bound, 0, sizeof(u32), st));
  TC_CUDA_TRY(cudaGetLastError());
  if ((rc = scan_exclusive_u32(cid, cid, id_bound + 1, scratch, st))) return rc;
  TC_CUDA_TRY(cudaMemcpyAsync(small + 1, cid + id_bound, sizeof(u32), cudaMemcpyDeviceToDevice, st));
  orient_kernel<<<grid_for((np + 3) / 4), 256, 0, st>>>(e, small, bits, deg, sparse_ids ? cid : nullptr, od);
  TC_NOTE_LAUNCH();
  max_kernel<<<grid_for((od_count + 7) / 8), 256, 0, st>>>(od, od_count, small + 2);
  TC_NOTE_LAUNCH();
  TC_CUDA_TRY(cudaGetLastError());
  u32 h[3] = {0, 0, 0};  // edges, vertices, largest out-degree
  TC_CUDA_TRY(cudaMemcpyAsync(h, small, sizeof h, cudaMemcpyDeviceToHost, st));
  TC_CUDA_TRY(cudaStreamSynchronize(st));
  const int64_t nu = h[0], n = h[1];
  const u32 odmax = h[2];
  if (d_seg_in && nseg > 0) {
    seg_map_kernel<<<grid_for(nseg), 256, 0, st>>>(cid, id_bound, n, d_seg_in, nseg, d_seg_out);
    TC_NOTE_LAUNCH();
  }
  int64_t *beg = nullptr;
  int32_t *adj = nullptr;
  TC_CUDA_TRY(cudaMalloc((void **)&beg, sizeof(int64_t) * (size_t)(n + 1)));
  cudaError_t ea = cudaMalloc((void **)&adj, sizeof(int32_t) * (size_t)std::max<int64_t>(nu, 1));
  if (ea != cudaSuccess) {
    cudaFree(beg);
    return cuda_status(ea);
  }
  auto finish = [&]() -> int {
    // 4. renumber: out-degree descending, ties by id (a stable sort from id order)
    if (keep_order) {
      newid = cid;
      kept_len_kernel<<<grid_for(id_bound), 256, 0, st>>>(deg, od, cid, id_bound, sparse_ids, n, beg);
      TC_NOTE_LAUNCH();
    } else {
      u64 *vkeys, *vtmp;
      if ((rc = B.get(&vkeys, n)) || (rc = B.get(&vtmp, n))) return rc;
      newid = cid;  // each vertex's entry is replaced by its new id
      renumber_key_kernel<<<grid_for(id_bound), 256, 0, st>>>(deg, od, cid, id_bound, sparse_ids, odmax, vkeys);
      TC_NOTE_LAUNCH();
      TC_CUDA_TRY(cudaGetLastError());
      if ((rc = sort_bits(vkeys, vtmp, n, 32, bits_for(odmax), scratch, st, &vkeys))) return rc;
      newid_kernel<<<grid_for(n + 1), 256, 0, st>>>(vkeys, n, odmax, newid, beg);
      TC_NOTE_LAUNCH();
    }
    TC_CUDA_TRY(cudaGetLastError());
    if ((rc = scan_exclusive_i64(beg, beg, n + 1, st, nullptr))) return rc;
    // 5. arcs by (source, target); the last pass writes the neighbour array
    if (nu > 0) {
      const int nbits = bits_for(std::max<int64_t>(n - 1, 1));
      relabel_kernel<<<grid_for((nu + 3) / 4), 256, 0, st>>>(e, nu, bits, nbits, newid);
      TC_NOTE_LAUNCH();
      TC_CUDA_TRY(cudaGetLastError());
      const int last = (2 * nbits - 1) / 8 * 8;
      u64 *arcs = e;
      if ((rc = sort_bits(e, cur, nu, 0, last, scratch, st, &arcs))) return rc;
      if ((rc = sort_pass<PlainKeys, true>(PlainKeys{arcs}, adj, nu, last, scratch, st,
                                           (u32)(((u64)1 << nbits) - 1))))
        return rc;
    }
    return cuda_status(cudaStreamSynchronize(st));
  };
  if ((rc = finish())) {
    cudaFree(beg);
    cudaFree(adj);
    return rc;
  }
  *d_beg_out = beg;
  *d_adj_out = adj;
  *n_out = n;
  *m_out = nu;
  return TRUST_TC_OK;
}

}  // namespace tc

// ---- the n x n hash partition on the GPU ---------------------------------------------------
// Tile (i,j) of Preprocess/partition.cpp:72-121: the rows of vertices v = i (mod p) as local row
// v / p, restricted to entries w = j (mod p), stored as w / p; rows stay sorted.  A warp per
// row: one ballot per part and 32 entries, lane j keeps part j's count (pass 1) or cursor (pass 2).
__global__ void part_count_kernel(const int64_t *__restrict__ beg, const int32_t *__restrict__ adj, int64_t n,
                                  int p, int64_t stride, int64_t *__restrict__ cnt) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t v = warp; v < n; v += nwarps) {
    const int64_t b = beg[v], e = beg[v + 1];
    int64_t mine = 0;
    for (int64_t k0 = b; k0 < e; k0 += 32) {
      const bool valid = k0 + lane < e;
      const int jw = valid ? (int)(adj[k0 + lane] % p) : -1;
      for (int j = 0; j < p; ++j) {
        const unsigned msk = __ballot_sync(TC_FULL_MASK, jw == j);
        if (lane == j) mine += __popc(msk);
      }
    }
    if (lane < p) cnt[(int64_t)((v % p) * p + lane) * stride + v / p] = mine;
  }
}

__global__ void part_fill_kernel(const int64_t *__restrict__ beg, const int32_t *__restrict__ adj, int64_t n, int p,
                                 int64_t stride, const int64_t *__restrict__ off, const int64_t *__restrict__ tbase,
                                 int32_t *__restrict__ out) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t v = warp; v < n; v += nwarps) {
    const int64_t b = beg[v], e = beg[v + 1];
    if (b == e) continue;
    const int i = (int)(v % p);
    // lane j: where part j's entries of this row go (tile base + row offset)
    int64_t pos = lane < p ? tbase[i * p + lane] + off[(int64_t)(i * p + lane) * stride + v / p] : 0;
    for (int64_t k0 = b; k0 < e; k0 += 32) {
      const bool valid = k0 + lane < e;
      const int w = valid ? adj[k0 + lane] : 0;
      const int jw = valid ? w % p : -1;
      for (int j = 0; j < p; ++j) {
        const unsigned msk = __ballot_sync(TC_FULL_MASK, jw == j);
        const int64_t cur = __shfl_sync(TC_FULL_MASK, pos, j);
        if (jw == j) out[cur + __popc(msk & ((1u << lane) - 1u))] = w / p;
        if (lane == j) pos += __popc(msk);
      }
    }
  }
}

namespace tc {

int partition_device(const int64_t *beg, const int32_t *adj, int64_t n, int64_t m, int p, Tile *tiles, int64_t **d_beg,
                     int32_t **d_adj) {
  if (n < 1 || m < 0 || p < 1 || p > 32) return TRUST_TC_E_ARG;
  cudaStream_t st = 0;
  const int64_t stride = (n + p - 1) / p + 1;  // rows of part 0, plus the end offset
  const size_t T = (size_t)p * p;
  int64_t *cnt = nullptr, *tbase = nullptr;
  int32_t *out = nullptr;
  TC_CUDA_TRY(cudaMalloc((void **)&cnt, sizeof(int64_t) * T * (size_t)stride));
  auto fail = [&](int rc) {
    cudaFree(cnt);
    cudaFree(tbase);
    cudaFree(out);
    return rc;
  };
  auto cu = [&](cudaError_t e) { return e == cudaSuccess ? TRUST_TC_OK : cuda_status(e); };
  int rc = cu(cudaMemsetAsync(cnt, 0, sizeof(int64_t) * T * (size_t)stride, st));
  if (rc) return fail(rc);
  const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>((n * 32 + 255) / 256, 152 * 64));
  part_count_kernel<<<blocks, 256, 0, st>>>(beg, adj, n, p, stride, cnt);
  TC_NOTE_LAUNCH();
  if ((rc = cu(cudaGetLastError()))) return fail(rc);
  std::vector<int64_t> hbase(T + 1, 0);
  int64_t all = 0;
  for (size_t t = 0; t < T; ++t) {
    const int i = (int)(t / p);
    const int64_t rows = n > i ? (n - i + p - 1) / p : 0;
    int64_t total = 0;
    if ((rc = scan_exclusive_i64(cnt + t * stride, cnt + t * stride, rows + 1, st, &total))) return fail(rc);
    tiles[t].rows = rows;
    tiles[t].m = total;
    all += total;
    hbase[t + 1] = (hbase[t] + total + 63) & ~(int64_t)63;
  }
  if (all != m) return fail(TRUST_TC_E_DEVICE);
  if ((rc = cu(cudaMalloc((void **)&tbase, sizeof(int64_t) * (T + 1))))) return fail(rc);
  if ((rc = cu(cudaMalloc((void **)&out, sizeof(int32_t) * (size_t)std::max<int64_t>(hbase[T], 1))))) return fail(rc);
  if ((rc = cu(cudaMemcpy(tbase, hbase.data(), sizeof(int64_t) * (T + 1), cudaMemcpyHostToDevice)))) return fail(rc);
  part_fill_kernel<<<blocks, 256, 0, st>>>(beg, adj, n, p, stride, cnt, tbase, out);
  TC_NOTE_LAUNCH();
  if ((rc = cu(cudaGetLastError())) || (rc = cu(cudaStreamSynchronize(st)))) return fail(rc);
  cudaFree(tbase);
  for (size_t t = 0; t < T; ++t) {
    tiles[t].beg = cnt + t * stride;
    tiles[t].adj = out + hbase[t];
  }
  *d_beg = cnt;
  *d_adj = out;
  return TRUST_TC_OK;
}

}  // namespace tc

extern "C" int trust_tc_build_csr_device(trust_tc_ctx *ctx, const int32_t *d_pairs, int64_t npairs,
                                         int64_t id_bound, int64_t **d_begin, int32_t **d_adj, int64_t *n,
                                         int64_t *m) {
  if (!d_begin || !d_adj || !n || !m || (npairs > 0 && !d_pairs)) return TRUST_TC_E_ARG;
  *d_begin = nullptr;
  *d_adj = nullptr;
  if (ctx) TC_CUDA_TRY(cudaSetDevice(ctx->device));
  return tc::build_csr_device(d_pairs, npairs, id_bound, d_begin, d_adj, n, m, (cudaStream_t)0, false, nullptr, 0,
                              nullptr);
}

extern "C" int trust_tc_build_batch_device(trust_tc_ctx *ctx, const int32_t *d_pairs, int64_t npairs,
                                           const int64_t *graph_vbeg, int64_t num_graphs, int64_t **d_begin,
                                           int32_t **d_adj, int64_t *n, int64_t *m, int64_t *graph_vbeg_out) {
  if (!d_begin || !d_adj || !n || !m || (npairs > 0 && !d_pairs) || num_graphs < 1 || !graph_vbeg ||
      !graph_vbeg_out || graph_vbeg[0] != 0)
    return TRUST_TC_E_ARG;
  for (int64_t g = 0; g < num_graphs; ++g)
    if (graph_vbeg[g] > graph_vbeg[g + 1]) return TRUST_TC_E_ARG;
  *d_begin = nullptr;
  *d_adj = nullptr;
  if (ctx) TC_CUDA_TRY(cudaSetDevice(ctx->device));
  const int64_t nseg = num_graphs + 1;
  int64_t *d_seg = nullptr;
  TC_CUDA_TRY(cudaMalloc((void **)&d_seg, sizeof(int64_t) * 2 * (size_t)nseg));
  cudaError_t e = cudaMemcpy(d_seg, graph_vbeg, sizeof(int64_t) * (size_t)nseg, cudaMemcpyHostToDevice);
  int rc = e == cudaSuccess ? TRUST_TC_OK : tc::cuda_status(e);
  if (!rc)
    rc = tc::build_csr_device(d_pairs, npairs, std::max<int64_t>(graph_vbeg[num_graphs], 1), d_begin, d_adj, n, m,
                              (cudaStream_t)0, true, d_seg, nseg, d_seg + nseg);
  if (!rc) {
    e = cudaMemcpy(graph_vbeg_out, d_seg + nseg, sizeof(int64_t) * (size_t)nseg, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) rc = tc::cuda_status(e);
  }
  cudaFree(d_seg);
  return rc;
}

extern "C" void trust_tc_free_device(void *p) {
  if (p) cudaFree(p);
}

extern "C" int trust_tc_copy(void *dst, const void *src, size_t bytes) {
  if (!bytes) return TRUST_TC_OK;
  if (!dst || !src) return TRUST_TC_E_ARG;
  TC_CUDA_TRY(cudaMemcpy(dst, src, bytes, cudaMemcpyDefault));
  return TRUST_TC_OK;
}
