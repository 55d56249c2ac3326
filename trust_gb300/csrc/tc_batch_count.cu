// tc_batch_count.cu — the persistent counting kernel of batches (many graphs, one launch).
//
// Rows arrive in the degree-class queues of tc_batch.cu, every row knows its graph, and a graph's
// ids are one range, usually of a few thousand: so a row's table is a bitmap over its graph's ids
// wherever that fits the warp's shared memory (a probe is one 4-byte load, no hashing), with hashed
// bit filters or hash tables for larger graphs.  Batch rows are short (4096 graphs: 13 entries per
// probed row), so what counts is the instructions around the probes: the rows of a warp's arcs are
// dealt in chunks to 8-lane groups instead of being flattened entry by entry.
// 4096 graphs, 380 M arcs, on GB300: bound by instruction issue (72 % busy); 116 -> about 75 warp
// instructions per 32 probes, the run 19.1 -> 13.9 ms (three CTAs per SM instead of four: 16.0).
#include <algorithm>

#include "tc_batch_count.h"
#include "tc_rows.cuh"

namespace tc {

namespace {

// Ids of one graph: [base, base + range).
struct IdSpace {
  int base;
  unsigned range;
};

// ---- row sets: set.of(lane of the arc).has(entry); no entry (-1) is in no set --------------------
struct HashSet {
  const int *tab;
  int log2;
  __device__ __forceinline__ const HashSet &of(int /*owner*/) const { return *this; }
  __device__ __forceinline__ int has(int key) const {
    if (key < 0) return 0;
    const unsigned bmask = (1u << (log2 - 2)) - 1u;
    unsigned b = tc_hash((unsigned)key, log2 - 2);
    for (unsigned it = 0; it <= bmask; ++it) {
      const int4 q = *reinterpret_cast<const int4 *>(tab + (b << 2));
      if (q.x == key || q.y == key || q.z == key || q.w == key) return 1;
      if ((q.x | q.y | q.z | q.w) < 0) return 0;  // an empty slot ends the search
      b = (b + 1u) & bmask;
    }
    return 0;
  }
};

// The row's bitmap over its graph's ids.
struct BitSet {
  const unsigned *words;
  IdSpace sp;
  __device__ __forceinline__ const BitSet &of(int /*owner*/) const { return *this; }
  __device__ __forceinline__ int has(int w) const {
    const unsigned x = (unsigned)(w - sp.base);
    return x < sp.range ? (int)(words[x >> 5] >> (x & 31u) & 1u) : 0;
  }
};

// The rows of a warp's 32/G vertices (G = 16, 32) as bit filters of `wpv` words each.  EXACT: the
// graph's ids fit the words, the filter is the row's bitmap.  Otherwise an entry is hashed to one bit
// and a set bit is confirmed against the row's keys (`keys`: the warp's 32 row entries, -1 where
// none): 16 or 32 keys in 2048 bits or more pass by chance less than once in 60 probes.
template <int G, bool EXACT>
struct GroupFilter {
  unsigned *words;
  const int *keys;
  int wpv;
  IdSpace sp;
  __device__ __forceinline__ unsigned bit_of(unsigned x) const {
    return EXACT ? x : __umulhi(x * 0x9E3779B1u, (unsigned)wpv << 5);
  }
  __device__ __forceinline__ GroupFilter of(int owner) const {
    const int g = owner / G;
    return GroupFilter{words + g * wpv, keys + g * G, wpv, sp};
  }
  __device__ __forceinline__ int has(int w) const {
    const unsigned x = (unsigned)(w - sp.base);
    if (EXACT ? x >= sp.range : w < 0) return 0;
    const unsigned b = bit_of(x);
    const unsigned in = words[b >> 5] >> (b & 31u) & 1u;
    if (EXACT) return (int)in;
    if (!in) return 0;
    for (int i = 0; i < G; ++i)
      if (keys[i] == w) return 1;
    return 0;
  }
};

// Probe every wedge of the arcs held one per lane: the arc's target row start `s` (int: m < 2^31)
// and length `dd` (0 if idle).  The whole 96-entry steps of long rows are walked by the warp; what is
// left of every row, up to three chunks of 32 entries, goes to a list of chunks (`wl`, 96 bytes of
// shared memory per warp: lane of the arc << 2 | chunk) that the warp's four 8-lane groups drain two
// at a time, so eight loads per lane are in flight and a probe costs no search for its row.  All 32
// lanes call it.
constexpr int WL_BYTES = 96;
template <class Set>
__device__ __forceinline__ void probe_chunks(const int32_t *__restrict__ adj, int s, int dd, unsigned char *wl,
                                             const Set &set, unsigned long long &hits) {
  const int lane = threadIdx.x & 31, grp = lane >> 3, gl = lane & 7;
  const unsigned lt = tc_lanemask_lt();
  unsigned h = 0;
  const int steps = (int)((unsigned)dd / 96u), rem = dd - 96 * steps, r0 = s + 96 * steps;
  unsigned lm = __ballot_sync(TC_FULL_MASK, steps > 0);
  while (lm) {
    const int j = __ffs(lm) - 1;
    lm &= lm - 1;
    const int32_t *row = adj + __shfl_sync(TC_FULL_MASK, s, j) + lane;
    const auto mine = set.of(j);
    for (int f = __shfl_sync(TC_FULL_MASK, steps, j); f > 0; --f, row += 96) {
      const int w0 = tc_ld_nc(row), w1 = tc_ld_nc(row + 32), w2 = tc_ld_nc(row + 64);
      h += mine.has(w0) + mine.has(w1) + mine.has(w2);
    }
  }
  // chunks of rows of at most 16 entries first: two rounds of 8 entries do for them
  const bool brief = rem > 0 && rem <= 16;
  const int nch = brief ? 0 : (rem + 31) >> 5;  // 0..3
  const unsigned bs = __ballot_sync(TC_FULL_MASK, brief), b0 = __ballot_sync(TC_FULL_MASK, nch & 1),
                 b1 = __ballot_sync(TC_FULL_MASK, nch & 2);
  const int ns = __popc(bs), n = ns + __popc(b0) + 2 * __popc(b1);
  if (n) {
    const int at = ns + __popc(b0 & lt) + 2 * __popc(b1 & lt);
    if (brief) wl[__popc(bs & lt)] = (unsigned char)(lane << 2);
#pragma unroll
    for (int j = 0; j < 3; ++j)
      if (j < nch) wl[at + j] = (unsigned char)(lane << 2 | j);
    const int most = (min(32, __reduce_max_sync(TC_FULL_MASK, rem)) + 7) >> 3;  // rounds of a long chunk
    __syncwarp();
    for (int i = grp; i - grp < n; i += 8) {
      const int rounds = i - grp + 8 <= ns ? min(most, 2) : most;
      const int ca = i < n ? wl[i] : 0, cb = i + 4 < n ? wl[i + 4] : 0;
      const int oa = ca >> 2, ob = cb >> 2, ea = (ca & 3) << 5, eb = (cb & 3) << 5;
      int la = __shfl_sync(TC_FULL_MASK, rem, oa) - ea, lb = __shfl_sync(TC_FULL_MASK, rem, ob) - eb;
      const int32_t *pa = adj + __shfl_sync(TC_FULL_MASK, r0, oa) + ea + gl;
      const int32_t *pb = adj + __shfl_sync(TC_FULL_MASK, r0, ob) + eb + gl;
      la = i < n ? la - gl : 0;
      lb = i + 4 < n ? lb - gl : 0;
      int wa[4], wb[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        wa[r] = wb[r] = -1;
        if (r < rounds) {
          if (8 * r < la) wa[r] = tc_ld_nc(pa + 8 * r);
          if (8 * r < lb) wb[r] = tc_ld_nc(pb + 8 * r);
        }
      }
      const auto sa = set.of(oa), sb = set.of(ob);
#pragma unroll
      for (int r = 0; r < 4; ++r)
        if (r < rounds) h += sa.has(wa[r]) + sb.has(wb[r]);
    }
    __syncwarp();
  }
  hits += h;
}

// ---- rows of at most 8 entries: each lane walks its own arc's target row against its vertex's keys
// held in registers -------------------------------------------------------------------------------
constexpr int LANE_ROW = 128;  // longer target rows are walked by the whole warp

template <int G>
__device__ __forceinline__ void probe_short(const int32_t *__restrict__ adj, int s, int dd, int u, unsigned long long &hits) {
  const int lane = threadIdx.x & 31;
  unsigned lm = __ballot_sync(TC_FULL_MASK, dd >= LANE_ROW);
  while (lm) {
    const int j = __ffs(lm) - 1;
    lm &= lm - 1;
    const int32_t *row = adj + __shfl_sync(TC_FULL_MASK, s, j);
    const int dj = __shfl_sync(TC_FULL_MASK, dd, j);
    int key[G];
#pragma unroll
    for (int k = 0; k < G; ++k) key[k] = __shfl_sync(TC_FULL_MASK, u, (j & ~(G - 1)) + k);
    for (int k = lane; k < dj; k += 32) hits += match_keys<G>(tc_ld_nc(row + k), key);
  }
  int key[G];
#pragma unroll
  for (int k = 0; k < G; ++k) key[k] = __shfl_sync(TC_FULL_MASK, u, (lane & ~(G - 1)) + k);
  hits += lane_walk<G>(adj + s, dd < LANE_ROW ? dd : 0, key);
}

// ---- the kernel ------------------------------------------------------------------------------------
struct BlockShared {
  unsigned long long count;
  unsigned long long wedges;
  int item;
  int next_batch;
};

__device__ __forceinline__ const int *class_list(const BatchCountArgs &p, int c) { return p.lists + p.ctl->class_off[c]; }

__device__ __forceinline__ IdSpace graph_space(const BatchCountArgs &p, int g) {
  const int b = (int)tc_ld_nc(p.graph_vbeg + g);
  return IdSpace{b, (unsigned)((int)tc_ld_nc(p.graph_vbeg + g + 1) - b)};
}

// Per-graph attribution: every lane keeps the hits of the graph its warp is working on; when the
// warp moves to another graph the warp's sum goes to that graph's counter with one atomic.
struct GraphAcc {
  int cur;
  unsigned long long h, total;
};

__device__ __forceinline__ void acc_flush(const BatchCountArgs &p, GraphAcc &a) {
  unsigned long long s = a.h;
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) s += __shfl_xor_sync(TC_FULL_MASK, s, off);
  if ((threadIdx.x & 31) == 0 && a.cur >= 0 && s) atomicAdd(p.graph_counts + a.cur, s);
  a.h = 0;
}

__device__ __forceinline__ void acc_take(const BatchCountArgs &p, GraphAcc &a, int g, unsigned long long hits) {  // warp-uniform g
  if (g != a.cur) {
    acc_flush(p, a);
    a.cur = g;
  }
  a.h += hits;
  a.total += hits;
}

// One vertex handled by a whole CTA; `tab` is shared memory (CTA class) or a global spill table.
// Warps claim 32-arc batches.
template <class Set>
__device__ __forceinline__ void cta_arcs(const BatchCountArgs &p, const Set &set, int b, int d, BlockShared &bs,
                                         unsigned char *wl, unsigned long long &hits, unsigned long long &wedges) {
  const int lane = threadIdx.x & 31;
  for (;;) {
    int at = 0;
    if (lane == 0) at = atomicAdd(&bs.next_batch, 32);
    at = __shfl_sync(TC_FULL_MASK, at, 0);
    if (at >= d) break;
    int s = 0, dd = 0;
    if (at + lane < d) row_of(p.beg, tc_ld_nc(p.adj + b + at + lane), s, dd);
    wedges += (unsigned)dd;
    probe_chunks(p.adj, s, dd, wl, set, hits);
  }
  __syncthreads();
}

__device__ void cta_vertex(const BatchCountArgs &p, int v, int *tab, bool smem_table, IdSpace sp, BlockShared &bs,
                           unsigned char *wl, unsigned long long &hits, unsigned long long &wedges) {
  int b, d;
  row_of(p.beg, v, b, d);
  if (threadIdx.x == 0) bs.next_batch = 0;
  if (smem_table && sp.range - 1u < 8u * (unsigned)p.table_bytes) {  // a bitmap over the graph's ids
    unsigned *words = reinterpret_cast<unsigned *>(tab);
    for (int i = threadIdx.x; i < (int)((sp.range + 31u) >> 5); i += blockDim.x) words[i] = 0;
    __syncthreads();
    int foreign = 0;  // (buffers refilled with arcs that leave their graph)
    for (int i = threadIdx.x; i < d; i += blockDim.x) {
      const unsigned x = (unsigned)(tc_ld_nc(p.adj + b + i) - sp.base);
      if (x < sp.range) atomicOr(words + (x >> 5), 1u << (x & 31u));
      else foreign = 1;
    }
    if (!__syncthreads_or(foreign)) {
      cta_arcs(p, BitSet{words, sp}, b, d, bs, wl, hits, wedges);
      return;
    }
  }
  const int log2 = ceil_log2_table(d), T = 1 << log2;
  // (buffers refilled with rows longer than the batch was made for)
  if (smem_table ? T > p.table_bytes / 4 : log2 > p.huge_log2) {
    if (threadIdx.x == 0) atomicOr(&p.ctl->status, TC_DEV_TABLE_FULL);
    return;
  }
  for (int i = threadIdx.x; i < T; i += blockDim.x) tab[i] = -1;
  __syncthreads();
  bool ok = true;
  for (int i = threadIdx.x; i < d; i += blockDim.x) ok &= set_insert(tab, log2, tc_ld_nc(p.adj + b + i));
  if (!ok) atomicOr(&p.ctl->status, TC_DEV_TABLE_FULL);
  __syncthreads();
  cta_arcs(p, HashSet{tab, log2}, b, d, bs, wl, hits, wedges);
}

// One vertex per warp, more than 32 entries: 32-arc rounds on the warp's table, a bitmap over the
// graph's ids where the warp's words hold one, else a hash table.  The words are zero on entry and
// on return.
__device__ __forceinline__ void warp_vertex(const BatchCountArgs &p, int v, int *warp_tab, IdSpace sp, unsigned char *wl,
                                            unsigned long long &hits, unsigned long long &wedges) {
  const int lane = threadIdx.x & 31;
  int b, d;
  row_of(p.beg, v, b, d);
  auto arcs = [&](const auto &set) {
    for (int a0 = 0; a0 < d; a0 += 32) {
      int s = 0, dd = 0;
      if (a0 + lane < d) row_of(p.beg, tc_ld_nc(p.adj + b + a0 + lane), s, dd);
      wedges += (unsigned)dd;
      probe_chunks(p.adj, s, dd, wl, set, hits);
    }
    __syncwarp();
  };
  if (sp.range - 1u < 32u * (unsigned)p.warp_words) {
    unsigned *words = reinterpret_cast<unsigned *>(warp_tab);
    bool foreign = false;
    for (int i = lane; i < d; i += 32) {
      const unsigned x = (unsigned)(tc_ld_nc(p.adj + b + i) - sp.base);
      if (x < sp.range) atomicOr(words + (x >> 5), 1u << (x & 31u));
      else foreign = true;
    }
    foreign = __any_sync(TC_FULL_MASK, foreign);
    __syncwarp();
    if (!foreign) arcs(BitSet{words, sp});
    for (int i = lane; i < d; i += 32) {
      const unsigned x = (unsigned)(tc_ld_nc(p.adj + b + i) - sp.base);
      if (x < sp.range) words[x >> 5] = 0;
    }
    __syncwarp();
    if (!foreign) return;
  }
  const int log2 = ceil_log2_table(d), T = 1 << log2;
  if (T > p.warp_words) {  // (as above)
    if (lane == 0) atomicOr(&p.ctl->status, TC_DEV_TABLE_FULL);
    return;
  }
  for (int i = lane; i < T; i += 32) warp_tab[i] = -1;
  __syncwarp();
  bool ok = true;
  for (int i = lane; i < d; i += 32) ok &= set_insert(warp_tab, log2, tc_ld_nc(p.adj + b + i));
  if (!ok) atomicOr(&p.ctl->status, TC_DEV_TABLE_FULL);
  __syncwarp();
  arcs(HashSet{warp_tab, log2});
  for (int i = lane; i < T; i += 32) warp_tab[i] = 0;
  __syncwarp();
}

// The warp's 32/G vertices (lane: its row entry u or -1, that entry's row (s, dd)).  G >= 16: the
// filter words are zero on entry and on return; the region's last 32 words hold the keys.  Without
// BITMAPS (the graphs' ids do not fit the words) 16-entry rows are walked as shorter ones are, and 32-entry rows
// take a hash table, left as it is: filters there let entries pass that cost a search of the keys (one graph
// of 2 M vertices and 16 M arcs 0.59 -> 0.46 ms, 200 of 60,000 and 1.8 M arcs 7.1 -> 6.8).
constexpr int HASH32_LOG2 = 8;
template <int G, bool BITMAPS>
__device__ __forceinline__ void group_vertices(const BatchCountArgs &p, int u, int s, int dd, int *wtab, IdSpace sp,
                                               unsigned char *wl, unsigned long long &hits) {
  if constexpr (G <= 8 || (G == 16 && !BITMAPS)) {
    probe_short<G>(p.adj, s, dd, u, hits);
  } else if constexpr (!BITMAPS) {  // one vertex of up to 32 entries
    const int lane = threadIdx.x & 31;
    int4 *slots = reinterpret_cast<int4 *>(wtab);
    slots[lane] = slots[lane + 32] = make_int4(-1, -1, -1, -1);
    __syncwarp();
    if (u >= 0) set_insert(wtab, HASH32_LOG2, u);
    __syncwarp();
    probe_chunks(p.adj, s, dd, wl, HashSet{wtab, HASH32_LOG2}, hits);
    __syncwarp();
  } else {
    const int lane = threadIdx.x & 31;
    unsigned *words = reinterpret_cast<unsigned *>(wtab);
    int *keys = wtab + p.warp_words - 32;
    const int wpv = (p.warp_words - 32) / (32 / G);
    const unsigned x = (unsigned)(u - sp.base);
    auto run = [&](const auto &f) {
      unsigned *mine = words + (lane / G) * wpv;
      const unsigned b = f.bit_of(x);
      if (u >= 0) atomicOr(mine + (b >> 5), 1u << (b & 31u));
      __syncwarp();
      probe_chunks(p.adj, s, dd, wl, f, hits);
      if (u >= 0) mine[b >> 5] = 0;
      __syncwarp();
    };
    if (sp.range - 1u < 32u * (unsigned)wpv && !__any_sync(TC_FULL_MASK, u >= 0 && x >= sp.range)) {
      run(GroupFilter<G, true>{words, keys, wpv, sp});
    } else {
      keys[lane] = u;
      run(GroupFilter<G, false>{words, keys, wpv, sp});
    }
  }
}

// Pipeline state of one group for one vertex: the list entry and its graph, its row, this lane's row
// entry and that entry's row.
struct GroupStage {
  int v, g, b, d, u, s, dd;
};

// Drain one group class.  Each warp claims `chunk` steps of 32/G vertices.  Loads run three steps
// ahead: while step t is probed, step t+1's target rows, step t+2's row entries and step t+3's row
// bounds are in flight.
template <int G, bool BITMAPS>
__device__ void drain_groups(const BatchCountArgs &p, int c, int *warp_tab, unsigned char *wl, GraphAcc &acc,
                             unsigned long long &wedges) {
  constexpr int GPW = 32 / G;
  const int lane = threadIdx.x & 31;
  const int grp = lane / G, gl = lane & (G - 1);
  const int n_items = p.ctl->class_count[c];
  const int *list = class_list(p, c);
  const int claim = p.chunk * GPW;
  auto ld_v = [&](int item, int t1) { return item < t1 ? list[item] : -1; };
  auto ld_row = [&](GroupStage &x) {
    x.b = x.d = 0;
    x.g = -1;
    if (x.v >= 0) {
      row_of(p.beg, x.v, x.b, x.d);
      x.g = tc_ld_nc(p.graph_of + x.v);
    }
  };
  auto ld_elem = [&](GroupStage &x) { x.u = gl < x.d ? tc_ld_nc(p.adj + x.b + gl) : -1; };
  auto ld_target = [&](GroupStage &x) {
    x.s = x.dd = 0;
    if (x.u >= 0) row_of(p.beg, x.u, x.s, x.dd);
  };
  for (;;) {
    int t0 = 0;
    if (lane == 0) t0 = atomicAdd(&p.ctl->class_next[c], claim);
    t0 = __shfl_sync(TC_FULL_MASK, t0, 0);
    if (t0 >= n_items) break;
    const int t1 = min(t0 + claim, n_items);
    GroupStage s0, s1, s2;
    s0.v = ld_v(t0 + grp, t1);
    s1.v = ld_v(t0 + GPW + grp, t1);
    s2.v = ld_v(t0 + 2 * GPW + grp, t1);
    ld_row(s0);
    ld_row(s1);
    ld_elem(s0);
    ld_target(s0);
    ld_elem(s1);
    ld_row(s2);
    int space_of = -1;
    IdSpace sp{0, 0};
    for (int t = t0; t < t1; t += GPW) {
      GroupStage s3;
      s3.v = ld_v(t + 3 * GPW + grp, t1);
      ld_target(s1);  // row entries of t+1 arrived during the previous step
      ld_elem(s2);
      ld_row(s3);
      // one pass per graph present in this step (almost always one), the other groups' vertices
      // masked out, so every hit of a pass belongs to that pass's graph
      unsigned pending = __ballot_sync(TC_FULL_MASK, s0.g >= 0);
      while (pending) {
        const int gx = __shfl_sync(TC_FULL_MASK, s0.g, __ffs(pending) - 1);
        const bool mine = s0.g == gx;
        if (gx != space_of) {
          sp = graph_space(p, gx);
          space_of = gx;
        }
        const int dd = mine ? s0.dd : 0;
        unsigned long long hits = 0;
        wedges += (unsigned)dd;
        group_vertices<G, BITMAPS>(p, mine ? s0.u : -1, s0.s, dd, warp_tab, sp, wl, hits);
        acc_take(p, acc, gx, hits);
        pending &= ~__ballot_sync(TC_FULL_MASK, mine);
      }
      s0 = s1;
      s1 = s2;
      s2 = s3;
    }
  }
}

template <int MAXT, int MINB, bool BITMAPS>
__global__ void __launch_bounds__(MAXT, MINB) batch_count_kernel(BatchCountArgs p) {
  extern __shared__ int smem[];
  __shared__ BlockShared bs;
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  unsigned char *wl = reinterpret_cast<unsigned char *>(smem) + p.table_bytes + warp * WL_BYTES;
  if (threadIdx.x == 0) bs.count = bs.wedges = 0;
  unsigned long long wedges = 0;
  GraphAcc acc{-1, 0, 0};

  // CTA-granularity vertices, largest class first
  for (int c = TC_CLASS_HUGE; c >= TC_CLASS_CTA; --c) {
    const int n_items = p.ctl->class_count[c];
    if (n_items == 0) continue;
    if (c == TC_CLASS_HUGE && (int)blockIdx.x >= p.huge_blocks) continue;
    const int *list = class_list(p, c);
    int *tab = (c == TC_CLASS_HUGE) ? p.huge_tables + (size_t)blockIdx.x * ((size_t)1 << p.huge_log2) : smem;
    for (;;) {
      __syncthreads();
      if (threadIdx.x == 0) bs.item = atomicAdd(&p.ctl->class_next[c], 1);
      __syncthreads();
      const int t = bs.item;
      if (t >= n_items) break;
      const int v = list[t], g = p.graph_of[v];
      unsigned long long hits = 0;
      cta_vertex(p, v, tab, c == TC_CLASS_CTA, graph_space(p, g), bs, wl, hits, wedges);
      acc_take(p, acc, g, hits);
    }
  }
  __syncthreads();

  // warp and sub-warp granularity
  int *warp_tab = smem + warp * p.warp_words;
  for (int i = lane; i < p.warp_words; i += 32) warp_tab[i] = 0;
  __syncwarp();
  {
    const int n_items = p.ctl->class_count[TC_CLASS_WARP];
    const int *list = class_list(p, TC_CLASS_WARP);
    const int claim = max(1, p.chunk / 8);
    for (;;) {
      int t0 = 0;
      if (lane == 0) t0 = atomicAdd(&p.ctl->class_next[TC_CLASS_WARP], claim);
      t0 = __shfl_sync(TC_FULL_MASK, t0, 0);
      if (t0 >= n_items) break;
      const int t1 = min(t0 + claim, n_items);
      for (int t = t0; t < t1; ++t) {
        const int v = list[t], g = p.graph_of[v];
        unsigned long long hits = 0;
        warp_vertex(p, v, warp_tab, graph_space(p, g), wl, hits, wedges);
        acc_take(p, acc, g, hits);
      }
    }
  }
  drain_groups<32, BITMAPS>(p, TC_CLASS_G32, warp_tab, wl, acc, wedges);
  drain_groups<16, BITMAPS>(p, TC_CLASS_G16, warp_tab, wl, acc, wedges);
  drain_groups<8, BITMAPS>(p, TC_CLASS_G8, warp_tab, wl, acc, wedges);
  drain_groups<4, BITMAPS>(p, TC_CLASS_G4, warp_tab, wl, acc, wedges);
  acc_flush(p, acc);

  unsigned long long hits = acc.total;
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) {
    hits += __shfl_down_sync(TC_FULL_MASK, hits, off);
    wedges += __shfl_down_sync(TC_FULL_MASK, wedges, off);
  }
  if (lane == 0 && hits) atomicAdd(&bs.count, hits);
  if (lane == 0 && wedges) atomicAdd(&bs.wedges, wedges);
  __syncthreads();
  if (threadIdx.x == 0 && bs.count) atomicAdd(&p.ctl->count, bs.count);
  if (threadIdx.x == 0 && bs.wedges) atomicAdd(&p.ctl->wedges, bs.wedges);
}

// Two register budgets: up to 1024 threads per CTA, or <= 256 with four CTAs resident per SM (with
// five the kernel spills: 17.7 against 15.4 ms per run of 4096 graphs).
const void *kernel_for(int threads, bool bitmaps) {
  if (threads <= 256)
    return bitmaps ? (const void *)batch_count_kernel<256, 4, true> : (const void *)batch_count_kernel<256, 4, false>;
  return bitmaps ? (const void *)batch_count_kernel<1024, 1, true> : (const void *)batch_count_kernel<1024, 1, false>;
}

size_t smem_for(size_t table_bytes, int threads) { return table_bytes + (size_t)WL_BYTES * (threads / 32); }

}  // namespace

static int shared_limits(const void *fn, int *per_sm, int *reserved, int *most) {
  int dev = 0, optin = 0;
  TC_CUDA_TRY(cudaGetDevice(&dev));
  TC_CUDA_TRY(cudaDeviceGetAttribute(per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev));
  TC_CUDA_TRY(cudaDeviceGetAttribute(reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev));
  TC_CUDA_TRY(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  cudaFuncAttributes at;
  TC_CUDA_TRY(cudaFuncGetAttributes(&at, fn));
  *reserved += (int)at.sharedSizeBytes;  // per CTA beside the dynamic part
  *most = optin - (int)at.sharedSizeBytes;
  return TRUST_TC_OK;
}

int batch_count_warp_words(int *words) {
  int per_sm = 0, reserved = 0, most = 0;
  int rc = shared_limits(kernel_for(256, true), &per_sm, &reserved, &most);
  if (rc) return rc;
  *words = (per_sm / 4 - reserved - 8 * WL_BYTES) / (8 * 4) & ~3;
  return TRUST_TC_OK;
}

int batch_count_occupancy(int threads, bool bitmaps, size_t table_bytes, int *blocks_per_sm) {
  const void *fn = kernel_for(threads, bitmaps);
  const int smem = (int)smem_for(table_bytes, threads);
  int per_sm = 0, reserved = 0, most = 0;
  int rc = shared_limits(fn, &per_sm, &reserved, &most);
  if (rc) return rc;
  if (smem > most) {
    *blocks_per_sm = 0;
    return TRUST_TC_OK;
  }
  // (the query honours the carveout an earlier batch has set)
  TC_CUDA_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
  TC_CUDA_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
  TC_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, fn, threads, smem));
  // What the resident CTAs leave of the SM's memory is L1 (500 graphs of 20,000 vertices 0.62 -> 0.48 ms, four
  // of 2 M vertices 1.14 -> 0.65).
  const int pct = (int)(100.0 * *blocks_per_sm * (smem + reserved) / per_sm) + 1;
  TC_CUDA_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, std::min(pct, 100)));
  return TRUST_TC_OK;
}

int launch_batch_count(const BatchCountArgs &a, int blocks, int threads, bool bitmaps, cudaStream_t st) {
  BatchCountArgs p = a;
  void *params[] = {&p};
  TC_CUDA_TRY(cudaLaunchKernel(kernel_for(threads, bitmaps), dim3((unsigned)blocks), dim3((unsigned)threads), params,
                               smem_for((size_t)a.table_bytes, threads), st));
  TC_NOTE_LAUNCH();
  return TRUST_TC_OK;
}

}  // namespace tc
