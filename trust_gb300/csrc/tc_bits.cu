// tc_bits.cu — block-bitmap rows: the direction split's counting path on skewed graphs.
//
// After the direction split an arc (v,u) is counted by streaming the shorter of its two rows
// against a table of the longer one.  On skewed graphs nearly all of that work lies in rows whose
// entries are a small set of popular columns, so this path renumbers the columns by popularity
// (in-degree) and stores every row as 16-column blocks: one 32-bit entry (block << 17 | bit mask)
// per block present, popular blocks first.  The table of a row is then a plain bitmap in shared
// memory, indexed by block: a lookup is one 16-bit load with no hashing, no key compare and no
// collision, and one AND + popcount settles up to 16 probes.  R-MAT 20 ef16: 0.46 entries per
// probe (a = 0.57), 0.26 (a = 0.70).  Columns beyond the bitmap ("tail" entries, the unpopular
// ones) stay plain ids after the row's blocks and are looked up in a small hash set.
//
// A tile job (tables from tile A, arcs of B, probe rows from C) is counted the same way with the rows of A
// and of C converted under one column order: A's long rows are probed by the C rows of their arcs, C's
// long rows by the A rows of the arcs moved to them (R-MAT 21 as 2 x 2 tiles 24.1 -> 17.4 ms per call).
//
// The rows must be duplicate-free (the split already requires it), so |N+(v) ∩ N+(u)| is the same
// number from either side and in any column numbering.
#include <algorithm>

#include "tc_bits.h"
#include "tc_count.h"
#include "tc_internal.h"
#include "tc_rows.cuh"

namespace tc {

namespace {

typedef unsigned int u32;

// ---- column popularity -----------------------------------------------------------------------
// In-degrees of a sample of the arcs: 32 of every 512 consecutive ones.  The order only decides which
// columns get the popular blocks, never the count, and a sixteenth of the arcs gives the same order
// where it matters (R-MAT 20, all arcs / a quarter / a sixteenth: 0.28 / 0.09 / 0.03 ms; the atomics on
// popular columns bound it.  R-MAT 24 a = 0.70, a quarter / a sixteenth: 44.2 / 43.7 ms per call).
constexpr int POP_SAMPLE = 16;
__global__ void indeg_kernel(const int32_t *__restrict__ adj, int64_t m, u32 *__restrict__ indeg) {
  const int64_t groups = (m + 32 * POP_SAMPLE - 1) / (32 * POP_SAMPLE);
  const int64_t stride = (int64_t)gridDim.x * blockDim.x >> 5;
  for (int64_t g = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; g < groups; g += 4 * stride) {
    int u[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int64_t i = (g + r * stride) * 32 * POP_SAMPLE + (threadIdx.x & 31);
      u[r] = i < m ? tc_ld_nc(adj + i) : -1;
    }
#pragma unroll
    for (int r = 0; r < 4; ++r)
      if (u[r] >= 0) atomicAdd(indeg + u[r], 1u);
  }
}

// Popularity bucket, most popular first: 8 buckets per doubling of the in-degree.
__device__ __forceinline__ int pop_bucket(u32 x) {
  if (x == 0) return 255;
  const int e = 31 - __clz(x);
  const int mant = e >= 3 ? (int)(x >> (e - 3)) & 7 : (int)(x << (3 - e)) & 7;
  return 254 - min(254, e * 8 + mant);
}

constexpr int RK_TILE = 4096;

__global__ void __launch_bounds__(256) rank_hist_kernel(const u32 *__restrict__ indeg, int64_t n, u32 *__restrict__ counts,
                                                        u32 ntiles) {
  __shared__ u32 h[256];
  h[threadIdx.x] = 0;
  __syncthreads();
  const int64_t base = (int64_t)blockIdx.x * RK_TILE;
  for (int r = 0; r < RK_TILE / 256; ++r) {
    const int64_t i = base + r * 256 + threadIdx.x;
    const int b = i < n ? pop_bucket(indeg[i]) : 256;
    const unsigned peers = __match_any_sync(TC_FULL_MASK, b);
    if (b < 256 && (peers & tc_lanemask_lt()) == 0) atomicAdd(&h[b], (u32)__popc(peers));
  }
  __syncthreads();
  counts[(size_t)threadIdx.x * ntiles + blockIdx.x] = h[threadIdx.x];
}

// rank[w] = position of column w, popular buckets first (any order inside a bucket and tile).  seen (or
// null): sampled entries whose column has a rank below `direct`, and all of them.
__global__ void __launch_bounds__(256) rank_scatter_kernel(const u32 *__restrict__ indeg, int64_t n,
                                                           const u32 *__restrict__ offs, u32 ntiles,
                                                           u32 *__restrict__ rank, u32 direct, u32 *seen) {
  __shared__ u32 cur[256];
  cur[threadIdx.x] = offs[(size_t)threadIdx.x * ntiles + blockIdx.x];
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int64_t base = (int64_t)blockIdx.x * RK_TILE;
  u32 in = 0, all = 0;
  for (int r = 0; r < RK_TILE / 256; ++r) {
    const int64_t i = base + r * 256 + threadIdx.x;
    const u32 entries = i < n ? indeg[i] : 0u;
    const int b = i < n ? pop_bucket(entries) : 256;
    const unsigned peers = __match_any_sync(TC_FULL_MASK, b);
    const int leader = __ffs(peers) - 1;
    u32 at = 0;
    if (b < 256 && lane == leader) at = atomicAdd(&cur[b], (u32)__popc(peers));
    at = __shfl_sync(TC_FULL_MASK, at, leader);
    at += __popc(peers & tc_lanemask_lt());
    if (b < 256) rank[i] = at;
    if (at < direct) in += entries;
    all += entries;
  }
  if (!seen) return;
  in = __reduce_add_sync(TC_FULL_MASK, in);
  all = __reduce_add_sync(TC_FULL_MASK, all);
  if (lane == 0 && in) atomicAdd(seen, in);
  if (lane == 0 && all) atomicAdd(seen + 1, all);
}

// ---- rows to blocks --------------------------------------------------------------------------
// Row v owns entries from row_start(v): 16-byte aligned, room for its d entries and the zero
// entries that pad its blocks to a multiple of four (m + 6 n entries in all).
__host__ __device__ __forceinline__ u32 row_start(int64_t beg, int64_t v) { return (u32)((beg + 6 * v + 3) & ~3ll); }

// Place of a row's e-th block (of nd4 * 4, padding included).  Blocks are laid out in chunks of 32,
// transposed: eight lanes read a chunk with one 16-byte load each, and the c-th 16-bit lookups of
// the eight then go to consecutive blocks, whose words share few banks where a row is dense.
__device__ __forceinline__ int entry_place(int e, int nd4) {
  const int lanes = min(8, nd4 - (e >> 5 << 3)), r = e & 31;
  return (e & ~31) + (lanes == 8 ? (r & 7) * 4 + (r >> 3) : (r % lanes) * 4 + r / lanes);
}

constexpr int BITS_WARP_ROW = 512;  // rows up to this are converted by a warp, above by a CTA

// Rows of at most 32 entries: a warp takes 32 consecutive rows, packs as many whole rows as fit
// its lanes, and groups the lanes of a row that fall into one block with a match.  Longer rows are
// listed (longs: warp rows from the front, CTA rows from the back).
__global__ void __launch_bounds__(256) bits_short_kernel(const int64_t *__restrict__ beg, const int32_t *__restrict__ adj,
                                                         int64_t n, const u32 *__restrict__ rank, int nb,
                                                         u32 base_at, u32 *__restrict__ ent, int4 *__restrict__ desc,
                                                         int *__restrict__ longs, u32 *__restrict__ nlongs) {
  const int lane = threadIdx.x & 31;
  const unsigned lt = tc_lanemask_lt();
  const unsigned upto = 0xffffffffu >> (31 - lane);
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t v0 = warp * 32; v0 < n; v0 += nwarps * 32) {
    const int64_t v = v0 + lane;
    int b = 0, d = 0;
    if (v < n) {
      const long long lo = tc_ld_nc(beg + v);
      b = (int)lo;
      d = (int)(tc_ld_nc(beg + v + 1) - lo);
      if (d == 0) desc[v] = make_int4(0, 0, 0, 0);
    }
    const unsigned w1 = __ballot_sync(TC_FULL_MASK, d > 32 && d <= BITS_WARP_ROW);
    const unsigned w2 = __ballot_sync(TC_FULL_MASK, d > BITS_WARP_ROW);
    if (w1 | w2) {
      u32 at1 = 0, at2 = 0;
      if (lane == 0) {
        if (w1) at1 = atomicAdd(nlongs, (u32)__popc(w1));
        if (w2) at2 = atomicAdd(nlongs + 1, (u32)__popc(w2));
      }
      at1 = __shfl_sync(TC_FULL_MASK, at1, 0);
      at2 = __shfl_sync(TC_FULL_MASK, at2, 0);
      if (w1 >> lane & 1) longs[at1 + __popc(w1 & lt)] = (int)v;
      if (w2 >> lane & 1) longs[n - 1 - (int64_t)(at2 + __popc(w2 & lt))] = (int)v;
    }
    const int sd = d <= 32 ? d : 0;
    int incl = sd;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(TC_FULL_MASK, incl, o);
      if (lane >= o) incl += y;
    }
    const int excl = incl - sd;
    const int tot = __shfl_sync(TC_FULL_MASK, incl, 31);
    for (int base = 0; base < tot;) {
      const bool in = sd > 0 && excl >= base && incl <= base + 32;
      const unsigned inm = __ballot_sync(TC_FULL_MASK, in);
      const unsigned starts = __reduce_or_sync(TC_FULL_MASK, in ? 1u << (excl - base) : 0u);
      const int wend = __reduce_max_sync(TC_FULL_MASK, in ? incl : 0);
      const bool valid = lane < wend - base;
      const int own = valid ? nth_set_bit(inm, __popc(starts & upto) - 1) : 0;
      const int bj = __shfl_sync(TC_FULL_MASK, b, own);
      const int ex = __shfl_sync(TC_FULL_MASK, excl, own) - base;
      const int dj = __shfl_sync(TC_FULL_MASK, sd, own);
      const u32 w = valid ? rank[tc_ld_nc(adj + bj + (lane - ex))] : 0u;
      const u32 blk = w >> 4;
      const bool direct = valid && blk < (u32)nb, tail = valid && !direct;
      const u32 key = direct ? ((u32)own << 16 | blk) : 0x80000000u | (u32)lane;
      const unsigned peers = __match_any_sync(TC_FULL_MASK, key);
      const u32 mask = __reduce_or_sync(peers, 1u << (w & 15u));
      const unsigned lead = __ballot_sync(TC_FULL_MASK, direct && (peers & lt) == 0);
      const unsigned tails = __ballot_sync(TC_FULL_MASK, tail);
      if (valid) {
        const unsigned mine = (dj == 32 ? 0xffffffffu : ((1u << dj) - 1u)) << ex;
        const int nd = __popc(lead & mine), pad = (nd + 3) & ~3;
        const u32 s = base_at + row_start(bj, v0 + own);
        if (lead >> lane & 1) ent[s + entry_place(__popc(lead & mine & lt), pad >> 2)] = blk << 17 | mask;
        if (tail) ent[s + pad + __popc(tails & mine & lt)] = w;
        if (lane == ex) {
          for (int k = nd; k < pad; ++k) ent[s + entry_place(k, pad >> 2)] = 0;
          desc[v0 + own] = make_int4((int)s, pad, __popc(tails & mine), dj);
        }
      }
      base = wend;
    }
  }
}

// Grouping table of a long row: slots (block << 17 | mask), 0 = empty; T = a power of two >= 2 d.
// The lower half is indexed by the block itself (popular blocks come out in order, so that a warp
// reading the row later touches neighbouring words of a table), the upper half by a hash of the
// other blocks; a row has at most T/2 blocks, so the upper half never overflows.
__device__ __forceinline__ void group_insert(u32 *tab, int T, u32 w) {
  const u32 blk = w >> 4, bit = 1u << (w & 15u), e = blk << 17;
  const u32 half = (u32)T >> 1;
  u32 h = blk < half ? blk : half + ((blk * 0x9E3779B1u >> 12) & (half - 1));
  for (int it = 0; it < T; ++it) {
    const u32 prev = atomicCAS(tab + h, 0u, e | bit);
    if (prev == 0u) return;
    if ((prev ^ e) < 0x10000u) {
      atomicOr(tab + h, bit);
      return;
    }
    h = half + ((h + 1) & (half - 1));
  }
}

__device__ __forceinline__ int group_slots(int d) {
  int T = 64;
  while (T < 2 * d) T <<= 1;
  return T;
}

// A warp per row of 33..BITS_WARP_ROW entries.
__global__ void __launch_bounds__(256) bits_warp_kernel(const int64_t *__restrict__ beg, const int32_t *__restrict__ adj,
                                                        const u32 *__restrict__ rank, int nb, u32 base_at,
                                                        u32 *__restrict__ ent, int4 *__restrict__ desc,
                                                        const int *__restrict__ longs,
                                                        const u32 *__restrict__ nlongs) {
  __shared__ u32 tabs[8][2 * BITS_WARP_ROW];
  u32 *tab = tabs[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const unsigned lt = tc_lanemask_lt();
  const u32 nl = nlongs[0];
  const u32 nwarps = gridDim.x * 8;
  for (u32 i = blockIdx.x * 8 + (threadIdx.x >> 5); i < nl; i += nwarps) {
    const int v = longs[i];
    const long long lo = tc_ld_nc(beg + v);
    const int d = (int)(tc_ld_nc(beg + v + 1) - lo);
    const int T = group_slots(d);
    for (int k = lane; k < T; k += 32) tab[k] = 0;
    __syncwarp();
    int nt = 0;
    for (int k = lane; k < d; k += 32) {
      const u32 w = rank[tc_ld_nc(adj + lo + k)];
      if (w >> 4 < (u32)nb) group_insert(tab, T, w);
      else ++nt;
    }
    nt = __reduce_add_sync(TC_FULL_MASK, nt);
    __syncwarp();
    const u32 s = base_at + row_start(lo, v);
    int nd = 0;
    for (int k = lane; k < T; k += 32) nd += tab[k] != 0;
    nd = __reduce_add_sync(TC_FULL_MASK, nd);
    const int pad = (nd + 3) & ~3;
    int put = 0;
    for (int k = lane; k < T; k += 32) {
      const u32 e = tab[k];
      const unsigned bm = __ballot_sync(TC_FULL_MASK, e != 0);
      if (e) ent[s + entry_place(put + __popc(bm & lt), pad >> 2)] = e;
      put += __popc(bm);
    }
    if (lane < pad - nd) ent[s + entry_place(nd + lane, pad >> 2)] = 0;
    if (nt) {
      int at = 0;
      for (int k0 = 0; k0 < d; k0 += 32) {
        const u32 w = k0 + lane < d ? rank[tc_ld_nc(adj + lo + k0 + lane)] : 0u;
        const bool tail = w >> 4 >= (u32)nb;
        const unsigned bm = __ballot_sync(TC_FULL_MASK, tail);
        if (tail) ent[s + pad + at + __popc(bm & lt)] = w;
        at += __popc(bm);
      }
    }
    if (lane == 0) desc[v] = make_int4((int)s, pad, nt, d);
    __syncwarp();
  }
}

// A CTA per longer row (up to BITS_MAX_ROW entries).
__global__ void __launch_bounds__(512) bits_cta_kernel(const int64_t *__restrict__ beg, const int32_t *__restrict__ adj,
                                                       int64_t n, const u32 *__restrict__ rank, int nb, u32 base_at,
                                                       u32 *__restrict__ ent, int4 *__restrict__ desc,
                                                       const int *__restrict__ longs, const u32 *__restrict__ nlongs) {
  extern __shared__ u32 tab[];
  __shared__ int wcnt[17];
  __shared__ int ntail;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned lt = tc_lanemask_lt();
  const u32 nl = nlongs[1];
  for (u32 i = blockIdx.x; i < nl; i += gridDim.x) {
    const int v = longs[n - 1 - (int64_t)i];
    const long long lo = tc_ld_nc(beg + v);
    const int d = (int)(tc_ld_nc(beg + v + 1) - lo);
    const int T = group_slots(d);
    for (int k = threadIdx.x; k < T; k += 512) tab[k] = 0;
    if (threadIdx.x == 0) ntail = 0;
    __syncthreads();
    for (int k = threadIdx.x; k < d; k += 512) {
      const u32 w = rank[tc_ld_nc(adj + lo + k)];
      if (w >> 4 < (u32)nb) group_insert(tab, T, w);
    }
    __syncthreads();
    // each warp owns T/16 consecutive slots: count, scan over the warps, write
    const int seg = T >> 4, k0 = warp * seg;
    int c = 0;
    for (int k = lane; k < seg; k += 32) c += tab[k0 + k] != 0;
    c = __reduce_add_sync(TC_FULL_MASK, c);
    if (lane == 0) wcnt[warp] = c;
    __syncthreads();
    int at = 0, nd = 0;
    for (int k = 0; k < 16; ++k) {
      if (k < warp) at += wcnt[k];
      nd += wcnt[k];
    }
    const int pad = (nd + 3) & ~3;
    const u32 s = base_at + row_start(lo, v);
    for (int k = lane; k < seg; k += 32) {  // seg >= 64
      const u32 e = tab[k0 + k];
      const unsigned bm = __ballot_sync(TC_FULL_MASK, e != 0);
      if (e) ent[s + entry_place(at + __popc(bm & lt), pad >> 2)] = e;
      at += __popc(bm);
    }
    if ((int)threadIdx.x < pad - nd) ent[s + entry_place(nd + threadIdx.x, pad >> 2)] = 0;
    for (int k = threadIdx.x; k < d; k += 512) {
      const u32 w = rank[tc_ld_nc(adj + lo + k)];
      if (w >> 4 >= (u32)nb) ent[s + pad + atomicAdd(&ntail, 1)] = w;
    }
    __syncthreads();
    if (threadIdx.x == 0) desc[v] = make_int4((int)s, pad, ntail, d);
    __syncthreads();  // wcnt, ntail and the table are free again
  }
}

// ---- work units ------------------------------------------------------------------------------
// A table row t (d > table_min) is probed by the rows of its out-neighbours u with d(u) <= d(t)
// (kept arcs) and of the sources of the arcs moved to it (its in-list).  Its list - out-row, then
// in-list - is cut into units of about `target` probes (an in-list row counts half the table row: it
// is shorter), of at least 64 list positions.  In-list space is reserved here with one atomic per
// warp; cnt[t] becomes the in-list's start.  A tile job's tables lie in two CSRs: its A rows (side 0)
// have the rows of B as their out-lists (beg_list) and no in-lists, its C rows (side 1) only in-lists.
struct Unit {
  int t, lo, hi, len_a;
  u32 a0, b0;
  int side, pad;
};

__global__ void __launch_bounds__(256) bits_units_kernel(const int64_t *__restrict__ beg,
                                                         const int64_t *__restrict__ beg_list, int64_t n, int64_t row_lo,
                                                         int64_t row_hi, int table_min, u32 *__restrict__ cnt,
                                                         const unsigned long long *__restrict__ wsum, u32 *ctr,
                                                         unsigned long long target, Unit *__restrict__ units, int side) {
  const int lane = threadIdx.x & 31;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t v0 = (int64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31); v0 < n; v0 += stride) {
    const int64_t v = v0 + lane;
    int d = 0;
    if (v < n) d = (int)(tc_ld_nc(beg + v + 1) - tc_ld_nc(beg + v));
    const bool table = d > table_min;
    if (!__any_sync(TC_FULL_MASK, table)) continue;
    const u32 nb = table && cnt ? cnt[v] : 0u;
    long long b = 0;
    int na = 0;
    if (table && beg_list && v >= row_lo && v < row_hi) {
      b = tc_ld_nc(beg_list + v);
      na = (int)(tc_ld_nc(beg_list + v + 1) - b);
    }
    const u32 len = nb + (u32)na;
    int k = 0;
    if (len) {
      // (without work sums the out-list's rows count half the table row too)
      const unsigned long long w = (wsum ? wsum[v] : (unsigned long long)na * (unsigned)d / 2) +
                                   (unsigned long long)nb * (unsigned)d / 2;
      const unsigned long long kk = max((w + target - 1) / target, 1ull);
      k = (int)min(kk, (unsigned long long)((len + 63) / 64));
    }
    // warp-wide exclusive sums of in-list lengths and units
    u32 sb = nb;
    int sk = k;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const u32 y = __shfl_up_sync(TC_FULL_MASK, sb, o);
      const int z = __shfl_up_sync(TC_FULL_MASK, sk, o);
      if (lane >= o) {
        sb += y;
        sk += z;
      }
    }
    u32 ab = 0, ak = 0;
    if (lane == 31) {
      if (sb) ab = atomicAdd(ctr + 1, sb);
      if (sk) ak = atomicAdd(ctr, (u32)sk);
    }
    ab = __shfl_sync(TC_FULL_MASK, ab, 31) + sb - nb;
    ak = __shfl_sync(TC_FULL_MASK, ak, 31) + (u32)(sk - k);
    if (table && cnt) cnt[v] = ab;
    const u32 per = k ? (len + k - 1) / k : 0;
    for (int j = 0; j < k; ++j)
      units[ak + j] = Unit{(int)v, (int)min((u32)j * per, len), (int)min((u32)(j + 1) * per, len), na, (u32)b, ab, side, 0};
  }
}

// ---- counting --------------------------------------------------------------------------------
constexpr int TAIL_SLOTS = 2048;             // hash slots of a table's tail ids
constexpr int TAIL_CAP = TAIL_SLOTS / 2;     // tail ids per pass over the unit

__device__ __forceinline__ u32 tail_hash(u32 w) { return w * 0x9E3779B1u >> (32 - 11); }

struct BitsArgs {
  const int32_t *adj, *adj_b;
  const int4 *desc, *desc_c;  // rows of A and of C (one graph: the same)
  const u32 *ent;
  const Unit *units;
  u32 *ctr;  // [0] units, [2] claim head
  int nb;    // blocks of the bitmap
  TcControl *ctl;
};

// Persistent: a CTA claims units and builds the unit's bitmap (plain 16-bit stores: a row has one
// entry per block).  Its warps claim the list's positions in batches of up to 32 (fewer towards the
// end of the unit), a lane holding one partner row; the partner ids are loaded two batches ahead
// and the row descriptors one.  The whole 128-block steps of a row are walked by the warp; what is
// left of every row (up to four 32-block chunks) goes to a work list in shared memory that the
// warp's four 8-lane groups drain, so that rows of any length keep the lanes busy.
// Bound by the shared-memory and load pipe (R-MAT 22 a = 0.70: 71 % busy, 2.8 wavefronts per 16-bit
// lookup of 32 lanes) and, on graphs whose rows exceed the L2 (R-MAT 22: 19 GB of DRAM reads in
// 7.3 ms), by the latency of the row loads.  The kernel takes 0.91 ms of R-MAT 20 ef16 and 32.4 of R-MAT 24
// a = 0.70; the calls, against the two hash passes it replaces, 5.7 -> 2.4 ms and 170 -> 44.
__device__ __forceinline__ u32 match4(const unsigned short *tab, uint4 e) {
  const unsigned char *t = reinterpret_cast<const unsigned char *>(tab);
  const u32 x0 = *reinterpret_cast<const unsigned short *>(t + (e.x >> 16)) & e.x;
  const u32 x1 = *reinterpret_cast<const unsigned short *>(t + (e.y >> 16)) & e.y;
  const u32 x2 = *reinterpret_cast<const unsigned short *>(t + (e.z >> 16)) & e.z;
  const u32 x3 = *reinterpret_cast<const unsigned short *>(t + (e.w >> 16)) & e.w;
  return __popc(__byte_perm(x0, x1, 0x5410)) + __popc(__byte_perm(x2, x3, 0x5410));
}

__device__ __forceinline__ uint4 piece(const uint4 *row, int k, int n) {
  return k < n ? __ldg(row + k) : make_uint4(0, 0, 0, 0);
}

__device__ __forceinline__ u32 tail_has(const int *tail, u32 w) {
  u32 h = tail_hash(w);
  int x = tail[h];
  while (x != -1 && x != (int)w) {
    h = (h + 1) & (TAIL_SLOTS - 1);
    x = tail[h];
  }
  return x == (int)w;
}

template <int THREADS, int MINB>
__global__ void __launch_bounds__(THREADS, MINB) bits_count_kernel(BitsArgs p) {
  constexpr int NW = THREADS / 32;
  extern __shared__ __align__(16) unsigned char smem[];
  unsigned short *tab = reinterpret_cast<unsigned short *>(smem);
  int *tail = reinterpret_cast<int *>(smem + 2 * (size_t)p.nb);
  __shared__ uint2 rows_all[NW][128];
  __shared__ Unit su[2];
  __shared__ int4 sd[2];
  __shared__ int next_batch;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int gl = lane & 7, grp = lane >> 3;
  uint2 *rows = rows_all[warp];
  const unsigned lt = tc_lanemask_lt();
  const u32 n_units = p.ctr[0];
  for (int i = threadIdx.x; i < p.nb / 8; i += THREADS) reinterpret_cast<uint4 *>(tab)[i] = make_uint4(0, 0, 0, 0);
  for (int i = threadIdx.x; i < TAIL_SLOTS; i += THREADS) tail[i] = -1;
  auto claim = [&](int at) {
    const u32 x = atomicAdd(p.ctr + 2, 1u);
    if (x < n_units) {
      su[at] = p.units[x];
      sd[at] = (su[at].side ? p.desc_c : p.desc)[su[at].t];
    } else {
      su[at].t = -1;
    }
  };
  if (threadIdx.x == THREADS - 1) claim(0);
  unsigned long long hits = 0;
  for (int cur = 0;; cur ^= 1) {
    __syncthreads();
    if (su[cur].t < 0) break;
    const int lo = su[cur].lo, hi = su[cur].hi, len_a = su[cur].len_a;
    const int32_t *list_a = p.adj + su[cur].a0, *list_b = p.adj_b + su[cur].b0 - len_a;
    const int4 td = sd[cur];
    const u32 ts = (u32)td.x;
    if (threadIdx.x == THREADS - 1) claim(cur ^ 1);
    for (int i = threadIdx.x; i < td.y; i += THREADS) {
      const u32 e = p.ent[ts + i];
      if (e & 0xffffu) tab[e >> 17] = (unsigned short)e;
    }
    for (int t0 = 0; t0 == 0 || t0 < td.z; t0 += TAIL_CAP) {
      const int tn = min(td.z - t0, TAIL_CAP);
      for (int i = threadIdx.x; i < tn; i += THREADS) {
        const int w = (int)p.ent[ts + td.y + t0 + i];
        u32 h = tail_hash((u32)w);
        for (int it = 0; it < TAIL_SLOTS && atomicCAS(tail + h, -1, w) != -1; ++it) h = (h + 1) & (TAIL_SLOTS - 1);
      }
      if (threadIdx.x == 0) next_batch = lo;
      __syncthreads();
      // claim a batch and load its partner ids (-1: no position); ~id on the in-list side
      auto claim_ids = [&](int &id, bool &in_a) -> bool {
        int at = 0, bs = 0;
        if (lane == 0) {
          bs = min(32, max(4, (hi - *(volatile int *)&next_batch) / (2 * NW)));
          at = atomicAdd(&next_batch, bs);
        }
        at = __shfl_sync(TC_FULL_MASK, at, 0);
        bs = __shfl_sync(TC_FULL_MASK, bs, 0);
        id = -1;
        const int i = at + lane;
        if (lane < bs && i < hi) {
          in_a = i < len_a;
          id = tc_ld_nc((in_a ? list_a : list_b) + i);
        }
        return at < hi;
      };
      auto fetch = [&](int id, bool in_a) -> int4 {
        if (id < 0) return make_int4(0, 0, 0, 0);
        int4 q = __ldg((in_a ? p.desc_c : p.desc) + id);
        if (in_a && q.w > td.w) q = make_int4(0, 0, 0, 0);  // counted from that row's side
        return q;
      };
      u32 acc = 0;
      int id = -1;
      bool side = false;
      bool more = claim_ids(id, side);
      int4 qn = fetch(id, side);
      bool later = more && claim_ids(id, side);
      while (more) {
        const int4 q = qn;
        more = later;
        if (later) {
          qn = fetch(id, side);
          later = claim_ids(id, side);
        }
        if (t0 == 0) {
          const int c4 = q.y >> 2;
          const int rem = c4 & 31;
          unsigned lm = __ballot_sync(TC_FULL_MASK, c4 >= 32);
          while (lm) {
            const int j = __ffs(lm) - 1;
            lm &= lm - 1;
            const uint4 *r = reinterpret_cast<const uint4 *>(p.ent + (u32)__shfl_sync(TC_FULL_MASK, q.x, j)) + lane;
            int steps = __shfl_sync(TC_FULL_MASK, c4, j) >> 5;
            for (; steps >= 2; steps -= 2, r += 64) {
              const uint4 e0 = __ldg(r), e1 = __ldg(r + 32);
              acc += match4(tab, e0) + match4(tab, e1);
            }
            if (steps) acc += match4(tab, __ldg(r));
          }
          const int nch = (rem + 7) >> 3;  // 0..4
          const unsigned b0 = __ballot_sync(TC_FULL_MASK, nch & 1), b1 = __ballot_sync(TC_FULL_MASK, nch & 2),
                         b2 = __ballot_sync(TC_FULL_MASK, nch & 4);
          const int n = __popc(b0) + 2 * __popc(b1) + 4 * __popc(b2);
          if (n) {
            const int at = __popc(b0 & lt) + 2 * __popc(b1 & lt) + 4 * __popc(b2 & lt);
            const u32 s = (u32)q.x + 4u * (u32)(c4 - rem);
#pragma unroll
            for (int j = 0; j < 4; ++j)
              if (j < nch) rows[at + j] = make_uint2(s + 32u * j, (u32)(rem - 8 * j));
            __syncwarp();
            for (int i = grp; i - grp < n; i += 8) {
              const uint2 ra = i < n ? rows[i] : make_uint2(0, 0), rb = i + 4 < n ? rows[i + 4] : make_uint2(0, 0);
              const uint4 ea = piece(reinterpret_cast<const uint4 *>(p.ent + ra.x), gl, (int)ra.y);
              const uint4 eb = piece(reinterpret_cast<const uint4 *>(p.ent + rb.x), gl, (int)rb.y);
              acc += match4(tab, ea) + match4(tab, eb);
            }
            __syncwarp();
          }
        }
        if (tn > 0) {  // tail ids against the hash set
          const unsigned km = __ballot_sync(TC_FULL_MASK, q.z > 0);
          const int n = __popc(km);
          if (n) {
            if (q.z > 0) rows[__popc(km & lt)] = make_uint2((u32)(q.x + q.y), (u32)q.z);
            __syncwarp();
            for (int i = 0; i < n; i += 8) {
              const uint2 ra = i + grp < n ? rows[i + grp] : make_uint2(0, 0);
              const uint2 rb = i + 4 + grp < n ? rows[i + 4 + grp] : make_uint2(0, 0);
              const int nm = __reduce_max_sync(TC_FULL_MASK, max((int)ra.y, (int)rb.y));
              for (int k = gl; k - gl < nm; k += 8) {
                const bool va = k < (int)ra.y, vb = k < (int)rb.y;
                const u32 wa = va ? __ldg(p.ent + ra.x + k) : 0u, wb = vb ? __ldg(p.ent + rb.x + k) : 0u;
                if (va) acc += tail_has(tail, wa);
                if (vb) acc += tail_has(tail, wb);
              }
            }
            __syncwarp();
          }
        }
      }
      hits += acc;
      __syncthreads();
      if (tn > 0) {
        for (int i = threadIdx.x; i < TAIL_SLOTS; i += THREADS) tail[i] = -1;
        __syncthreads();
      }
    }
    for (int i = threadIdx.x; i < td.y; i += THREADS) {
      const u32 e = p.ent[ts + i];
      if (e & 0xffffu) tab[e >> 17] = 0;
    }
  }
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) hits += __shfl_down_sync(TC_FULL_MASK, hits, o);
  if (lane == 0 && hits) atomicAdd(&p.ctl->count, hits);
}

// 256 threads, five CTAs per SM.  Measured on R-MAT 22 / R-MAT 25 ef32 (call, ms): 512 threads x 3
// 15.7 / 538, 256 x 5 12.3 / 423, 256 x 6 with 40 registers 12.5 / 432, 256 x 4 13.0 / 456; the bitmap
// of 8192, 13,312, 16,384 (four CTAs) blocks 12.3 / 423, 12.3 / 415, 12.8 / 427.
constexpr int BITS_THREADS = 256;
constexpr int BITS_MINB = 5;
constexpr int BITS_MAX_BLOCKS = 13312;  // bitmap of 212,992 columns, 26 KiB; at most 32,767 (entry format)

int blocks_for(int64_t work, int64_t per, int num_sms, int most_per_sm) {
  return (int)std::max<int64_t>(1, std::min<int64_t>((work + per - 1) / per, (int64_t)num_sms * most_per_sm));
}

}  // namespace

static bool one_csr(const DevGraph3 &g) { return g.begA == g.begC && g.adjA == g.adjC; }

bool bits_eligible(const DevGraph3 &g, int64_t max_out_degree) {
  const int64_t words = g.mA + 6 * g.rows + 12 + (one_csr(g) ? 0 : g.mC + 6 * g.rowsC + 12);
  return max_out_degree > BITS_TABLE_MIN && max_out_degree <= BITS_MAX_ROW && words < ((int64_t)1 << 32);
}

// The scratch block of both steps: in-degrees, ranks, rank histogram and its scan, counters (units, in-list
// entries, claims, warp rows and CTA rows of either CSR, then sampled entries), row lists.
namespace {
struct Columns {
  u32 *indeg, *rank, *counts, *scratch, *ctr;
  int *longs;
  int64_t cols;
  u32 ntiles;
  int nb;
};
constexpr int CTR_SEEN = 8;
}  // namespace

static bool is_tile(const DevGraph3 &g) { return g.begA != g.begB || g.adjA != g.adjB || !one_csr(g); }

static int columns_of(trust_tc_ctx *c, const DevGraph3 &g, Columns *k) {
  k->cols = is_tile(g) ? g.boundA : g.rows;
  k->nb = (int)std::min<int64_t>((((k->cols + 15) / 16) + 7) & ~7ll, BITS_MAX_BLOCKS);
  k->ntiles = (u32)((k->cols + RK_TILE - 1) / RK_TILE);
  const size_t nn = (size_t)k->cols, hist = 256 * (size_t)k->ntiles, scan = scan_u32_scratch(256 * (int64_t)k->ntiles);
  const size_t rows = (size_t)std::max(g.rows, one_csr(g) ? 0 : g.rowsC);
  int rc = ensure((void **)&c->d_bits_cols, &c->bits_cols_cap, sizeof(u32) * (2 * nn + rows + hist + scan + 16));
  if (rc) return rc;
  k->indeg = c->d_bits_cols;
  k->rank = k->indeg + nn;
  k->counts = k->rank + nn;
  k->scratch = k->counts + hist;
  k->ctr = k->scratch + scan;
  k->longs = reinterpret_cast<int *>(k->ctr + 16);
  return TRUST_TC_OK;
}

// Rank the columns by popularity.
static int rank_columns(trust_tc_ctx *c, const DevGraph3 &g, const Columns &k, bool count_seen, cudaStream_t st) {
  int rc;
  TC_CUDA_TRY(cudaMemsetAsync(k.indeg, 0, sizeof(u32) * (size_t)k.cols, st));
  TC_CUDA_TRY(cudaMemsetAsync(k.ctr, 0, sizeof(u32) * 16, st));
  indeg_kernel<<<blocks_for(g.mA, 1024, c->num_sms, 16), 256, 0, st>>>(g.adjA, g.mA, k.indeg);
  note_launch();
  if (!one_csr(g)) {
    indeg_kernel<<<blocks_for(g.mC, 1024, c->num_sms, 16), 256, 0, st>>>(g.adjC, g.mC, k.indeg);
    note_launch();
  }
  rank_hist_kernel<<<k.ntiles, 256, 0, st>>>(k.indeg, k.cols, k.counts, k.ntiles);
  TC_CUDA_TRY(cudaGetLastError());
  note_launch();
  if ((rc = scan_exclusive_u32(k.counts, k.counts, 256 * (int64_t)k.ntiles, k.scratch, st))) return rc;
  rank_scatter_kernel<<<k.ntiles, 256, 0, st>>>(k.indeg, k.cols, k.counts, k.ntiles, k.rank, 16u * (u32)k.nb,
                                                count_seen ? k.ctr + CTR_SEEN : nullptr);
  TC_CUDA_TRY(cudaGetLastError());
  note_launch();
  return TRUST_TC_OK;
}

// A bitmap over 212,992 of many columns of about equal popularity leaves most entries to the tails'
// hash sets, one load and lookup each.  Share of the sampled entries in the bitmap, and ms with block bitmaps /
// hash passes, Erdos-Renyi of 600,000 vertices 0.62, 46 / 56; 800,000 0.51, 43 / 42; 1 M 0.41, 64 / 57; 4 M 0.14,
// 110 / 77.  Skewed graphs: R-MAT 24 with a = 0.45 0.67, 53 / 67, with a = 0.70 0.98, 44 / 170.
constexpr double BITS_MIN_SEEN = 0.5;

int bits_columns(trust_tc_ctx *c, const DevGraph3 &g, cudaStream_t st, BitsPlan *plan, bool *suit) {
  Columns k;
  int rc = columns_of(c, g, &k);
  if (rc) return rc;
  *suit = true;
  if ((double)k.cols * BITS_MIN_SEEN <= 16.0 * k.nb) return TRUST_TC_OK;  // whatever their popularity
  if ((rc = rank_columns(c, g, k, true, st))) return rc;
  u32 seen[2];
  TC_CUDA_TRY(cudaMemcpyAsync(seen, k.ctr + CTR_SEEN, sizeof seen, cudaMemcpyDeviceToHost, st));
  TC_CUDA_TRY(cudaStreamSynchronize(st));
  *suit = (double)seen[0] >= BITS_MIN_SEEN * (double)seen[1];
  plan->ranked = true;
  return TRUST_TC_OK;
}

// Enqueue the conversion and the work units (after the scheduling pass and its readback).
int bits_prepare(trust_tc_ctx *c, const DevGraph3 &g, int64_t row_lo, int64_t row_hi, const SchedPlan &plan,
                 int64_t max_out_degree, cudaStream_t st, BitsPlan *out) {
  const bool tile = is_tile(g);
  const bool two = !one_csr(g);  // rows of two CSRs are converted
  // units: every table at least one, and one more per `target` probes: about eight units per resident
  // CTA, so the last ones end together, but not so small that a unit's set-up shows (R-MAT 18: 1.63 ms
  // at 2^18 probes, 1.81 at 2^20; R-MAT 25: 426 and 415)
  const unsigned long long target = std::min<unsigned long long>(
      std::max<unsigned long long>(plan.w_min / (unsigned long long)(c->num_sms * BITS_MINB * 8), 1ull << 16), 1ull << 20);
  // list positions are at most 2 mB: a unit per table and per 64 of them
  const int64_t max_units = (g.mA + (tile ? g.mC : 0)) / (BITS_TABLE_MIN + 1) + 2 * g.mB / 64 + 2;
  const int64_t rows_c = two ? g.rowsC : 0;
  const u32 base_c = (u32)((g.mA + 6 * g.rows + 11) & ~3ll);
  const size_t words = two ? (size_t)base_c + (size_t)(g.mC + 6 * g.rowsC + 8) : (size_t)(g.mA + 6 * g.rows + 8);
  Columns k;
  int rc = columns_of(c, g, &k);
  if (rc) return rc;
  if ((rc = ensure((void **)&c->d_bits_desc, &c->bits_desc_cap, sizeof(int4) * (size_t)(g.rows + rows_c)))) return rc;
  if ((rc = ensure((void **)&c->d_bits_ent, &c->bits_ent_cap, sizeof(u32) * words))) return rc;
  if ((rc = ensure((void **)&c->d_bits_units, &c->bits_units_cap, sizeof(Unit) * (size_t)max_units))) return rc;
  if ((rc = ensure((void **)&c->d_split_adj, &c->split_adj_cap, sizeof(int32_t) * (size_t)std::max<int64_t>(g.mB, 1))))
    return rc;
  if (!out->ranked && (rc = rank_columns(c, g, k, false, st))) return rc;
  u32 *const rank = k.rank, *const ctr = k.ctr;
  int *const longs = k.longs;
  const int nb = k.nb;
  int4 *desc = reinterpret_cast<int4 *>(c->d_bits_desc);
  int4 *desc_c = two ? desc + g.rows : desc;
  Unit *units = reinterpret_cast<Unit *>(c->d_bits_units);
  auto convert = [&](const int64_t *beg, const int32_t *adj, int64_t n, u32 base, int4 *d, u32 *nlongs) -> int {
    bits_short_kernel<<<blocks_for(n, 256, c->num_sms, 32), 256, 0, st>>>(beg, adj, n, rank, nb, base, c->d_bits_ent, d,
                                                                          longs, nlongs);
    bits_warp_kernel<<<c->num_sms * 7, 256, 0, st>>>(beg, adj, rank, nb, base, c->d_bits_ent, d, longs, nlongs);
    note_launch(2);
    TC_CUDA_TRY(cudaGetLastError());
    if (max_out_degree > BITS_WARP_ROW) {
      int T = 64;
      while (T < 2 * max_out_degree) T <<= 1;
      const int smem = 4 * T;
      TC_CUDA_TRY(
          cudaFuncSetAttribute(bits_cta_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 4 * 2 * BITS_MAX_ROW));
      bits_cta_kernel<<<c->num_sms * std::min(4, (int)(200 * 1024 / (smem + 2048))), 512, smem, st>>>(
          beg, adj, n, rank, nb, base, c->d_bits_ent, d, longs, nlongs);
      note_launch();
      TC_CUDA_TRY(cudaGetLastError());
    }
    return TRUST_TC_OK;
  };
  if ((rc = convert(g.begA, g.adjA, g.rows, 0, desc, ctr + 3))) return rc;
  if (two && (rc = convert(g.begC, g.adjC, g.rowsC, base_c, desc_c, ctr + 5))) return rc;
  const auto cut = [&](const int64_t *beg, const int64_t *beg_list, int64_t n, u32 *cnt, const unsigned long long *wsum,
                       int side) {
    bits_units_kernel<<<blocks_for(n, 256, c->num_sms, 16), 256, 0, st>>>(beg, beg_list, n, row_lo, row_hi,
                                                                          BITS_TABLE_MIN, cnt, wsum, ctr, target, units,
                                                                          side);
    note_launch();
  };
  if (tile) {
    cut(g.begA, g.begB, g.rows, nullptr, nullptr, 0);
    cut(g.begC, nullptr, g.rowsC, c->d_split_cnt, nullptr, 1);
  } else {
    cut(g.begA, g.begA, g.rows, c->d_split_cnt, c->d_split_wsum, 0);
  }
  TC_CUDA_TRY(cudaGetLastError());
  if ((rc = split_fill_u32(c, g.mB, c->d_split_cnt, st))) return rc;
  out->nb = nb;
  out->ctr = ctr;
  out->rows_c_at = two ? g.rows : 0;
  return TRUST_TC_OK;
}

int bits_launch(trust_tc_ctx *c, const BitsPlan &plan, const int32_t *adj, TcControl *ctl, cudaStream_t st) {
  BitsArgs a{};
  a.adj = adj;
  a.adj_b = c->d_split_adj;
  a.desc = reinterpret_cast<const int4 *>(c->d_bits_desc);
  a.desc_c = a.desc + plan.rows_c_at;
  a.ent = c->d_bits_ent;
  a.units = reinterpret_cast<const Unit *>(c->d_bits_units);
  a.ctr = plan.ctr;
  a.nb = plan.nb;
  a.ctl = ctl;
  const auto kernel = bits_count_kernel<BITS_THREADS, BITS_MINB>;
  const size_t smem = 2 * (size_t)plan.nb + 4 * TAIL_SLOTS;
  TC_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   2 * BITS_MAX_BLOCKS + 4 * TAIL_SLOTS));
  TC_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
  int per_sm = 0;
  TC_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, BITS_THREADS, smem));
  kernel<<<c->num_sms * std::max(per_sm, 1), BITS_THREADS, smem, st>>>(a);
  note_launch();
  TC_CUDA_TRY(cudaGetLastError());
  return TRUST_TC_OK;
}

}  // namespace tc
