"""The work this library is used for, as measurable cases.

A case names an entry point (``op``), a graph family and its sizes:

  count        count_csr over a CSR resident on the GPU, with a Context the program keeps
  count_host   count_csr over a CSR in pinned host memory (copy in, count, read the count)
  build        build_csr: edge pairs on the GPU -> oriented, renumbered CSR
  batch        Batch.run: thousands of graphs counted by one captured launch
  tiles        count_tiles: the n x n tile loop for graphs larger than the device

Graphs are drawn here with plain torch from the seed alone: R-MAT (skewed, web / social like),
Chung-Lu (power law, little clustering), triangulated meshes with holes, Erdos-Renyi and
preferential attachment.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import trust_gb300 as T
from trust_gb300 import batch as B

CHUNK = 1 << 26  # pairs drawn at a time, so that drawing needs little memory


# ---- edge pairs --------------------------------------------------------------------------------

def _gen(seed: int) -> torch.Generator:
    return torch.Generator(device="cuda").manual_seed(seed)


def _rmat(scale: int, npairs: int, a: float, seed: int) -> torch.Tensor:
    """R-MAT pairs with quadrant probabilities (a, b, b, 0.05), b = (0.95 - a) / 2."""
    g = _gen(seed)
    b = (0.95 - a) / 2
    out = torch.empty((npairs, 2), dtype=torch.int32, device="cuda")
    for at in range(0, npairs, CHUNK):
        k = min(CHUNK, npairs - at)
        u = torch.zeros(k, dtype=torch.int32, device="cuda")
        v = torch.zeros(k, dtype=torch.int32, device="cuda")
        for _ in range(scale):
            r = torch.rand(k, device="cuda", generator=g)
            down = r >= a + b
            right = ((r >= a) & (r < a + b)) | (r >= a + 2 * b)
            u.mul_(2).add_(down)
            v.mul_(2).add_(right)
        out[at:at + k, 0] = u
        out[at:at + k, 1] = v
    return out


def _chung_lu(n: int, npairs: int, gamma: float, w_max: float, seed: int) -> torch.Tensor:
    """Endpoint pairs drawn in proportion to w_i = (1 + i / i0)^(-1 / (gamma - 1)), the largest
    expected degree about w_max."""
    g = _gen(seed)
    i = torch.arange(n, dtype=torch.float64, device="cuda")
    lo, hi = 1e-6, float(n)
    for _ in range(40):  # i0 by bisection: w_max / sum(w) of the 2 npairs endpoints is w_max
        i0 = math.sqrt(lo * hi)
        s = float(((1 + i / i0) ** (-1 / (gamma - 1))).sum())
        if 2 * npairs / s > w_max:
            lo = i0
        else:
            hi = i0
    cdf = ((1 + i / i0) ** (-1 / (gamma - 1))).cumsum(0)
    cdf /= cdf[-1].clone()
    r = torch.rand((npairs, 2), dtype=torch.float64, device="cuda", generator=g)
    return torch.searchsorted(cdf, r.view(-1)).clamp_(max=n - 1).to(torch.int32).view(npairs, 2)


def _mesh(side: int, seed: int) -> torch.Tensor:
    """side x side grid with one diagonal per cell, its direction drawn per cell, 2 % of the edges
    missing; vertices numbered row by row."""
    g = _gen(seed)
    ids = torch.arange(side * side, dtype=torch.int32, device="cuda").view(side, side)
    flip = torch.rand((side - 1, side - 1), device="cuda", generator=g) < 0.5
    p = torch.where(flip, ids[:-1, 1:], ids[:-1, :-1]).reshape(-1)
    q = torch.where(flip, ids[1:, :-1], ids[1:, 1:]).reshape(-1)
    e = torch.cat([torch.stack([ids[:, :-1].reshape(-1), ids[:, 1:].reshape(-1)], 1),
                   torch.stack([ids[:-1].reshape(-1), ids[1:].reshape(-1)], 1), torch.stack([p, q], 1)])
    keep = torch.rand(e.shape[0], device="cuda", generator=g) >= 0.02
    return e[keep].contiguous()


def _er(n: int, npairs: int, seed: int) -> torch.Tensor:
    return torch.randint(0, n, (npairs, 2), dtype=torch.int32, device="cuda", generator=_gen(seed))


def _attach(n: torch.Tensor, d: torch.Tensor, base: torch.Tensor, g: torch.Generator) -> torch.Tensor:
    """Preferential attachment for several graphs at once (n vertices, d edges per vertex, first
    vertex id `base` each): an edge's far end copies a uniformly drawn earlier endpoint."""
    edges = n * d
    first = torch.cumsum(edges, 0) - edges
    graph = torch.repeat_interleave(torch.arange(n.numel(), device="cuda"), edges)
    e = torch.arange(int(edges.sum()), device="cuda") - first[graph]   # edge number inside its graph
    dg = d[graph]
    src = e // dg
    earlier = 2 * src * dg                                             # endpoints before this vertex
    pos = (torch.rand(e.numel(), dtype=torch.float64, device="cuda", generator=g) * earlier).long()
    pos = torch.where(earlier > 0, torch.minimum(pos, earlier - 1), torch.zeros_like(pos))
    draw = pos.clone()
    odd = (pos & 1).bool()
    while bool(odd.any()):                                             # a far end: look where it points
        at = odd.nonzero(as_tuple=True)[0]
        nxt = draw[first[graph[at]] + (pos[at] >> 1)]
        pos[at] = nxt
        odd = torch.zeros_like(odd)
        odd[at] = (nxt & 1).bool()
    dst = (pos >> 1) // dg
    return torch.stack([src + base[graph], dst + base[graph]], 1).to(torch.int32)


def _batch_sizes(case: dict, seed: int):
    """Sizes of the batch's graphs: vertices log-uniform in [50, nmax], even graphs Erdos-Renyi of
    average degree 4..64, odd ones preferential attachment of 2..16 edges per vertex."""
    r = np.random.RandomState(seed & 0x7FFFFFFF)
    k = case["graphs"]
    n = np.exp(r.uniform(math.log(50), math.log(case["nmax"]), k)).astype(np.int64)
    par = np.where(np.arange(k) % 2 == 0, r.randint(4, 65, k), r.randint(2, 17, k))
    return n, par


def _batch(case: dict, seed: int):
    n, par = _batch_sizes(case, seed)
    vbeg = np.zeros(n.size + 1, dtype=np.int64)
    vbeg[1:] = np.cumsum(n)
    g = _gen(seed)
    dev = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()  # noqa: E731
    even = np.arange(n.size) % 2 == 0
    ne, pe, be = dev(n[even]), dev(par[even]), dev(vbeg[:-1][even])
    cnt = ne * pe // 2
    graph = torch.repeat_interleave(torch.arange(ne.numel(), device="cuda"), cnt)
    r = torch.rand((graph.numel(), 2), dtype=torch.float64, device="cuda", generator=g)
    ng = ne[graph][:, None]
    er = (torch.minimum((r * ng).long(), ng - 1) + be[graph][:, None]).to(torch.int32)
    del r, graph, ng
    parts = [er]
    if (~even).any():
        parts.append(_attach(dev(n[~even]), dev(par[~even]), dev(vbeg[:-1][~even]), g))
    return torch.cat(parts), vbeg


def _npairs(case: dict) -> int:
    if case["graph"] == "mesh":
        s = case["side"]
        return int(0.98 * (2 * s * (s - 1) + (s - 1) ** 2))
    if case["graph"] == "batch":
        n, par = _batch_sizes(case, 1)
        return int(np.where(np.arange(n.size) % 2 == 0, n * par // 2, n * par).sum())
    return case["pairs"]


def _pairs(case: dict, seed: int):
    """(pairs, exclusive id bound).  A build case is one graph as different programs would store it:
    the seed numbers its vertices and turns its edges at random, so n and m stay what they are."""
    kind = case["graph"]
    if case["op"] == "build":
        p, bound = _pairs(dict(case, op="count"), 1)
        g = _gen(seed)
        ids = torch.randperm(bound, device="cuda", generator=g).to(torch.int32)
        for at in range(0, p.shape[0], CHUNK):
            part = p[at:at + CHUNK]
            turn = torch.rand(part.shape[0], device="cuda", generator=g) < 0.5
            q = ids[part.long()]
            part[:, 0] = torch.where(turn, q[:, 1], q[:, 0])
            part[:, 1] = torch.where(turn, q[:, 0], q[:, 1])
        return p, bound
    if kind == "rmat":
        return _rmat(case["scale"], case["pairs"], case["a"], seed), 1 << case["scale"]
    if kind == "chung_lu":
        return _chung_lu(case["n"], case["pairs"], case["gamma"], case["w_max"], seed), case["n"]
    if kind == "mesh":
        return _mesh(case["side"], seed), case["side"] ** 2
    return _er(case["n"], case["pairs"], seed), case["n"]


# ---- the cases ---------------------------------------------------------------------------------

def listed():
    return [
        # a program that counts many small graphs one call at a time: latency and launches
        dict(name="count_rmat8", op="count", graph="rmat", scale=8, pairs=2011, a=0.57),
        # the plain method's small configuration: R-MAT 16, edge factor 16
        dict(name="count_rmat16", op="count", graph="rmat", scale=16, pairs=16 << 16, a=0.57),
        # an ordinary skewed graph
        dict(name="count_rmat20", op="count", graph="rmat", scale=20, pairs=16 << 20, a=0.57),
        # a sparse power-law graph with little clustering (3.8 M vertices, 16.5 M edges)
        dict(name="count_chung_lu_3.8m", op="count", graph="chung_lu", n=3_800_000, pairs=16_500_000, gamma=2.5,
             w_max=800.0),
        # a finite-element like mesh: short rows only
        dict(name="count_mesh4096", op="count", graph="mesh", side=4096),
        # strongly skewed, 268 M pairs
        dict(name="count_rmat24_a070", op="count", graph="rmat", scale=24, pairs=16 << 24, a=0.70),
        # the largest: a billion pairs in device memory
        dict(name="count_rmat25_ef32", op="count", graph="rmat", scale=25, pairs=32 << 25, a=0.57),
        # the graph comes from a loader in pinned host memory
        dict(name="host_chung_lu_3.8m", op="count_host", graph="chung_lu", n=3_800_000, pairs=16_500_000, gamma=2.5,
             w_max=800.0),
        # preprocessing: an ordinary and a large edge list
        dict(name="build_rmat20", op="build", graph="rmat", scale=20, pairs=16 << 20, a=0.57),
        dict(name="build_rmat24", op="build", graph="rmat", scale=24, pairs=16 << 24, a=0.57),
        # 4096 graphs of 50..50,000 vertices in one launch
        dict(name="batch4096", op="batch", graph="batch", graphs=4096, nmax=50_000),
        # the tile loop of a graph that would not fit
        dict(name="tiles_rmat21_2x2", op="tiles", graph="rmat", scale=21, pairs=16 << 21, a=0.57, parts=2),
    ]


def _log(rng, lo: float, hi: float) -> float:
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _draw_graph(rng, most: float) -> dict:
    """A graph of 1e3 to `most` pairs."""
    kind = rng.choice(["rmat", "rmat", "rmat", "chung_lu", "mesh", "er"])
    pairs = int(_log(rng, 1e3, most))
    if kind == "rmat":
        ef = _log(rng, 4, 40)
        scale = max(6, min(25, round(math.log2(pairs / ef))))
        return dict(graph="rmat", scale=scale, pairs=pairs, a=round(rng.uniform(0.45, 0.70), 3))
    if kind == "mesh":
        return dict(graph="mesh", side=max(16, int(math.sqrt(min(pairs, 5e7) / 3))))
    n = max(64, int(pairs / _log(rng, 2, 24)))
    if kind == "er":
        return dict(graph="er", n=n, pairs=min(pairs, 200_000_000))
    return dict(graph="chung_lu", n=n, pairs=min(pairs, 100_000_000), gamma=round(rng.uniform(2.1, 3.0), 3),
                w_max=float(max(8, int(min(math.sqrt(pairs), _log(rng, 30, 2000))))))


def draw(rng):
    op = rng.choice(["count", "count", "count", "count", "count_host", "build", "build", "batch", "tiles"])
    if op == "batch":
        return dict(op="batch", graph="batch", graphs=int(_log(rng, 16, 4096)), nmax=int(_log(rng, 500, 50_000)))
    if op == "tiles":
        scale = rng.randint(10, 20)
        return dict(op="tiles", graph="rmat", scale=scale, pairs=int(_log(rng, 4, 24) * (1 << scale)),
                    a=round(rng.uniform(0.45, 0.65), 3), parts=rng.randint(2, 3))
    return dict(op=op, **_draw_graph(rng, {"count": 4e8, "count_host": 3e7, "build": 2.6e8}[op]))


# ---- one case ----------------------------------------------------------------------------------

def prepare(case, seed):
    op = case["op"]
    s = {"op": op}
    if op == "batch":
        pairs, vbeg = _batch(case, seed)
        beg, adj, gv = B.build_batch(pairs, vbeg)
        del pairs
        s["ctx"] = T.Context()
        s["batch"] = B.Batch(beg, adj, gv, ctx=s["ctx"])
        return s
    pairs, bound = _pairs(case, seed)
    if op == "build":
        s.update(pairs=pairs, bound=bound)
        return s
    beg, adj = T.build_csr(pairs, bound)
    del pairs
    if op == "count_host":
        s["pinned"] = (beg.cpu().pin_memory(), adj.cpu().pin_memory())  # kept: numpy views them
        s["beg"], s["adj"] = (x.numpy() for x in s["pinned"])
        s["ctx"] = T.Context()
        return s
    s.update(beg=beg, adj=adj)
    if op == "tiles":
        s["parts"] = case["parts"]
    else:
        s["ctx"] = T.Context()
    return s


def _counted(r):
    return {"triangles": r.triangles, "vertices": r.vertices, "edges": r.edges, "max_out_degree": r.max_out_degree}


def run(state):
    op = state["op"]
    if op in ("count", "count_host"):
        return _counted(T.count_csr(state["beg"], state["adj"], ctx=state["ctx"]))
    if op == "build":
        beg, adj = T.build_csr(state["pairs"], state["bound"])
        return {"beg": beg, "adj": adj}
    if op == "batch":
        counts, _ = state["batch"].run()
        return {"counts": counts.view(np.int64)}
    r = T.count_tiles(state["beg"], state["adj"], state["parts"])
    return {"triangles": r.triangles, "vertices": r.vertices, "edges": r.edges}


def work(case):
    """Bytes: a count reads the CSR once (4 per arc, 8 per row), a build reads 8 per pair and writes
    the CSR; arcs and rows are estimated from the pairs.  A count's probes are integer table lookups
    and compares, not floating-point work."""
    pairs = _npairs(case)
    kind = case["graph"]
    if kind == "rmat":
        ids = 1 << case["scale"]
        arcs, rows = 0.93 * pairs, ids * min(0.95, 0.36 + 0.012 * pairs / ids)
    elif kind == "mesh":
        arcs, rows = pairs, case["side"] ** 2
    elif kind == "batch":
        arcs, rows = pairs, float(_batch_sizes(case, 1)[0].sum())
    else:
        arcs, rows = pairs, case["n"] * (1 - math.exp(-2 * pairs / case["n"]))
    csr = 4 * arcs + 8 * rows
    return {"bytes": csr + (8 * pairs if case["op"] == "build" else 0), "flops": 0}


# ---- the same results in plain torch -----------------------------------------------------------

def _exact_csr(pairs: torch.Tensor, bound: int, keep_order: bool = False):
    """Drop self-loops and duplicates, orient from lower to higher (degree, id), number the vertices
    that have edges by out-degree (descending, ties by id), rows ascending."""
    p = pairs.long()
    lo, hi = p.min(1).values, p.max(1).values
    key = torch.unique((lo * bound + hi)[lo != hi])
    lo, hi = key // bound, key % bound
    deg = torch.bincount(torch.cat([lo, hi]), minlength=bound)
    present = deg > 0
    n = int(present.sum())
    swap = (deg[lo] > deg[hi])  # ties: the smaller id first, and lo < hi already
    src, dst = torch.where(swap, hi, lo), torch.where(swap, lo, hi)
    if keep_order:
        new = torch.cumsum(present, 0) - 1
    else:
        od = torch.bincount(src, minlength=bound)
        rank = torch.argsort(torch.where(present, -od, torch.ones_like(od)), stable=True)
        new = torch.empty_like(rank)
        new[rank] = torch.arange(bound, device="cuda")
    arc = torch.sort(new[src] * n + new[dst]).values
    beg = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    if n:
        beg[1:] = torch.cumsum(torch.bincount(arc // n, minlength=n), 0)
    return beg, arc % max(n, 1), arc, new


def _exact_hits(beg, adj, arc, limit: float):
    """Per arc (v, u): how many w of the shorter of the two rows lie in the other; None when that
    takes more than `limit` lookups."""
    n, m = beg.numel() - 1, adj.numel()
    d = beg[1:] - beg[:-1]
    v = torch.repeat_interleave(torch.arange(n, device="cuda"), d)
    short = torch.where(d[adj] <= d[v], adj, v)
    other = torch.where(d[adj] <= d[v], v, adj)
    cost = d[short]
    if float(cost.sum()) > limit:
        return None, v
    hits = torch.zeros(m, dtype=torch.int64, device="cuda")
    ends = torch.cumsum(cost, 0)
    at = 0
    while at < m:
        done = int(ends[at - 1]) if at else 0
        to = max(at + 1, int(torch.searchsorted(ends, done + (1 << 27), right=True)))
        c = cost[at:to]
        arcs = torch.repeat_interleave(torch.arange(at, to, device="cuda"), c)
        k = torch.arange(arcs.numel(), device="cuda") - (ends[at:to] - c - done)[arcs - at]
        q = other[arcs] * n + adj[beg[short[arcs]] + k]
        found = arc[torch.searchsorted(arc, q).clamp_(max=m - 1)] == q
        hits.index_add_(0, arcs[found], torch.ones(int(found.sum()), dtype=torch.int64, device="cuda"))
        at = to
    return hits, v


def exact(case, seed):
    if _npairs(case) > 40_000_000:
        return None
    if case["op"] == "batch":
        pairs, vbeg = _batch(case, seed)
        beg, adj, arc, _ = _exact_csr(pairs, int(vbeg[-1]), keep_order=True)
        # an arc's graph, from its original id: rows keep their order, so count present ids
        deg = torch.bincount(pairs[pairs[:, 0] != pairs[:, 1]].long().reshape(-1), minlength=int(vbeg[-1]))
        cum = torch.cat([torch.zeros(1, dtype=torch.int64, device="cuda"), torch.cumsum(deg > 0, 0)])
        gv = cum[torch.from_numpy(vbeg).cuda()]
        hits, v = _exact_hits(beg, adj, arc, 3e9)
        if hits is None:
            return None
        graph = torch.searchsorted(gv, v, right=True) - 1
        counts = torch.zeros(vbeg.size - 1, dtype=torch.int64, device="cuda").index_add_(0, graph, hits)
        return {"counts": counts}
    pairs, bound = _pairs(case, seed)
    beg, adj, arc, _ = _exact_csr(pairs, bound)
    if case["op"] == "build":
        return {"beg": beg, "adj": adj.to(torch.int32)}
    hits, _ = _exact_hits(beg, adj, arc, 3e9)
    if hits is None:
        return None
    out = {"triangles": int(hits.sum()), "vertices": beg.numel() - 1, "edges": adj.numel()}
    if case["op"] != "tiles":
        out["max_out_degree"] = int((beg[1:] - beg[:-1]).max()) if beg.numel() > 1 else 0
    return out
