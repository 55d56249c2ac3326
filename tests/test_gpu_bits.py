"""The block-bitmap counting path (tc_bits.cu) at the sizes where it can go wrong, against the
oracle's forward-intersection counter: rows at the table bound and at the bounds of the row
conversion's kernels, bitmaps narrower and wider than the graph, tail ids over several passes."""
import numpy as np
import pytest

import trust_gb300 as T
from oracle import oracle as O

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _csr(rows, n):
    beg = np.zeros(n + 1, dtype=np.int64)
    for v, r in rows.items():
        beg[v + 1] = len(r)
    beg = np.cumsum(beg)
    adj = np.zeros(int(beg[-1]), dtype=np.int32)
    for v, r in rows.items():
        adj[beg[v]:beg[v + 1]] = r
    return beg, adj


def _check(beg, adj, lo=None, hi=None):
    db, da = torch.from_numpy(beg).cuda(), torch.from_numpy(adj).cuda()
    expect = O.count_forward_sorted_range(beg, adj, 0, beg.size - 1, 2, 8)
    d = np.diff(beg)
    src = np.repeat(np.arange(d.size), d)
    sel = d[src] >= 2
    with T.Context() as ctx:
        for _ in range(2):
            r = T.count_csr(db, da, ctx=ctx, direction_split=1)
            assert r.triangles == expect and r.direction_split == 1
            assert r.wedges == int(np.minimum(d[adj], d[src])[sel].sum())
        n = beg.size - 1
        cut = [0, n // 3, n // 2 + 1, n]
        parts = [T.count_csr(db, da, ctx=ctx, direction_split=1, row_range=(a, b)).triangles
                 for a, b in zip(cut[:-1], cut[1:])]
        assert sum(parts) == expect
        assert T.count_csr(db, da, ctx=ctx, direction_split=1, schedule=T.SCHED_TUNED).triangles == expect
        assert T.count_csr(db, da, ctx=ctx, schedule=T.SCHED_PLAIN).triangles == expect


@pytest.mark.parametrize("n", [129, 130, 131, 200, 513, 514, 700, 1100])
def test_complete_graphs(n):
    """Row v = v+1..n-1: rows of every length up to n-1 (128 / 129: the table bound; 32 / 33 and
    512 / 513: the conversion kernels' bounds)."""
    rows = {v: np.arange(v + 1, n) for v in range(n)}
    _check(*_csr(rows, n))


@pytest.mark.parametrize("scale,ef,a", [(10, 64, 0.57), (13, 48, 0.45), (15, 24, 0.7), (17, 16, 0.57)])
def test_rmat(scale, ef, a):
    b = (0.95 - a) / 2
    beg, adj = T.build_csr(T.gen_rmat(scale, ef, a, b, b, seed=scale), 1 << scale)
    _check(beg.cpu().numpy(), adj.cpu().numpy())


@pytest.mark.parametrize("n,hubs,row", [(300_000, 40, 300), (600_000, 30, 1500), (500_000, 12, 3000),
                                        (400_000, 3, 8192)])
def test_tails(n, hubs, row):
    """Rows whose columns mostly lie beyond the bitmap (one reader each): tails of one and of several
    passes; the hubs also point at each other and share some columns."""
    rng = np.random.default_rng(n + hubs)
    rows = {}
    shared = rng.choice(np.arange(hubs, n), size=row // 4, replace=False)
    for h in range(hubs):
        mine = rng.choice(np.arange(hubs, n), size=row - shared.size - (hubs - 1 - h), replace=False)
        rows[h] = np.unique(np.concatenate([np.arange(h + 1, hubs), shared, mine]))[:row]
    for v in range(hubs, n, 7):  # many short rows: popular columns and a few of their own
        rows[v] = np.unique(rng.integers(hubs, n, size=rng.integers(1, 5)))
    beg, adj = _csr(rows, n)
    _check(beg, adj)


@pytest.mark.parametrize("row", [8192, 8193])
def test_longest_row(row):
    """One row of 8192 entries (the longest the conversion groups) and of 8193 (the hash tables)."""
    n = 20_000
    rng = np.random.default_rng(row)
    rows = {0: np.sort(rng.choice(np.arange(1, n), size=row, replace=False))}
    for v in range(1, 3000):
        rows[v] = np.unique(rng.integers(v + 1, n, size=rng.integers(1, 300)))
    _check(*_csr(rows, n))


def _slice_count(beg, adj, lo, hi):
    """The counted quantity over source rows [lo, hi), rows in any order and with repeated entries."""
    row = lambda v: adj[beg[v]:beg[v + 1]].tolist()  # noqa: E731
    return sum(w in s for v in range(lo, hi) if beg[v + 1] - beg[v] >= 2 for s in (set(row(v)),)
               for u in row(v) for w in row(u))


@pytest.mark.parametrize("long_row", [129, 20])
@pytest.mark.parametrize("schedule", [T.SCHED_LEARNED, T.SCHED_TUNED])
def test_slices_with_duplicates_outside(long_row, schedule):
    """A slice of increasing rows whose arcs lead to rows outside it with a repeated entry (kept arcs: the
    slice's row is the longer; moved arcs: the repeating row is) counts with multiplicity."""
    n = 500
    rows = {0: np.concatenate([[5, 7, 100], np.arange(200, 200 + long_row - 3)]),
            1: np.array([7, 100, 101]),
            100: np.array([5, 5, 7]), 101: np.concatenate([[7, 7], np.arange(130, 330), [330] * 2])}
    for v in range(110, 300):
        rows[v] = np.array([v + 5, v + 9])
    beg, adj = _csr(rows, n)
    db, da = torch.from_numpy(beg).cuda(), torch.from_numpy(adj).cuda()
    with T.Context() as ctx:
        cuts = (0, 1, 2, 105, n)
        parts = [T.count_csr(db, da, ctx=ctx, direction_split=1, schedule=schedule, row_range=(a, b))
                 for a, b in zip(cuts[:-1], cuts[1:])]
        assert [r.triangles for r in parts] == [_slice_count(beg, adj, a, b) for a, b in zip(cuts[:-1], cuts[1:])]
        assert all(r.direction_split == 0 for r in parts)
        assert sum(r.triangles for r in parts) == O.count_forward(beg, adj)


@pytest.mark.parametrize("where", ["first", "second", "last", "none"])
@pytest.mark.parametrize("pad", [0, 1, 2, 3])
def test_slice_check_sees_every_row(where, pad):
    """One repeated or descending entry anywhere outside the slice keeps it unsplit; rows that end on a
    larger entry than the next row starts with, empty rows and one-entry rows do not."""
    n = 3000
    rng = np.random.default_rng(pad)
    rows = {v: np.unique(rng.integers(0, n, size=rng.integers(0, 9))) for v in range(pad, n - pad)}
    rows[n // 2] = np.arange(300)
    at = {"first": min(v for v in rows if len(rows[v]) > 2), "last": max(v for v in rows if len(rows[v]) > 2)}
    at["second"] = min(v for v in rows if len(rows[v]) > 2 and v > at["first"])
    if where != "none":
        rows[at[where]] = rows[at[where]][[0, 2, 1]] if where == "second" else rows[at[where]][[0, 0, 1]]
    beg, adj = _csr(rows, n)
    db, da = torch.from_numpy(beg).cuda(), torch.from_numpy(adj).cuda()
    lo, hi = n // 2 - 3, n // 2 + 3
    r = T.count_csr(db, da, direction_split=1, row_range=(lo, hi))
    assert r.direction_split == int(where == "none") and r.triangles == _slice_count(beg, adj, lo, hi)


def test_slices_of_little_work():
    """Slices that repay the conversion, that do not by their rows' squares, and that do not by their probes
    alone (planned for the bitmaps first): a clique and rows that point into it, in a graph of 2 M rows."""
    n, k = 2_000_000, 800
    rng = np.random.default_rng(8)
    rows = {v: np.arange(v + 1, k) for v in range(k)}
    for v in range(k, 6000):
        rows[v] = np.unique(np.concatenate([rng.integers(0, k, size=4), rng.integers(k, n, size=3)]))
    beg, adj = _csr(rows, n)
    db, da = torch.from_numpy(beg).cuda(), torch.from_numpy(adj).cuda()
    d = np.diff(beg)
    with T.Context() as ctx:
        cuts = [0, 100, 300, k, 3000, n]
        ranges = [(0, k), (0, 200), (0, 6000), (100, 900)] + list(zip(cuts[:-1], cuts[1:]))
        for _ in range(2):
            for lo, hi in ranges:
                r = T.count_csr(db, da, ctx=ctx, direction_split=1, row_range=(lo, hi))
                assert r.direction_split == 1
                assert r.triangles == O.count_forward_sorted_range(beg, adj, lo, hi, 2, 8)
                at = slice(beg[lo], beg[hi])
                src = np.repeat(np.arange(lo, hi), d[lo:hi])
                assert r.wedges == int(np.minimum(d[adj[at]], d[src])[d[src] >= 2].sum())


@pytest.mark.parametrize("off", [0, 1, 2, 3])
@pytest.mark.parametrize("size", [290, 300, 1000, 4099])
def test_slice_check_on_unaligned_entries(off, size):
    """The check streams 16 bytes at a time: one descent at every place of small arrays of every alignment."""
    n = 4100
    beg = np.zeros(n + 1, dtype=np.int64)
    beg[n // 2 + 1:] = 280  # row n/2, the slice; the last row holds the rest
    beg[-1] = size
    good = np.concatenate([np.arange(280), np.arange(size - 280)]).astype(np.int32)
    buf = torch.zeros(size + 8, dtype=torch.int32, device="cuda")
    da, db = buf[off:off + size], torch.from_numpy(beg).cuda()
    with T.Context() as ctx:
        places = [None] + [p for p in {281, 282, 283, 284, 285, size - 3, size - 2, size - 1} if 280 < p < size]
        for at in places:
            a = good.copy()
            if at is not None:
                a[at] = a[at - 1]
            da.copy_(torch.from_numpy(a))
            r = T.count_csr(db, da, ctx=ctx, direction_split=1, row_range=(n // 2, n // 2 + 1))
            assert r.direction_split == int(at is None)
            assert r.triangles == _slice_count(beg, a, n // 2, n // 2 + 1)


@pytest.mark.parametrize("n", [425_984, 425_985, 2_000_000])
@pytest.mark.parametrize("popular", [0, 1000])
def test_wide_graphs(n, popular):
    """More columns than two bitmaps hold: entries spread over all of them (hash passes), or most of them in
    a few popular ones; one graph and tile jobs."""
    rng = np.random.default_rng(n + popular)
    hubs, row = 30, 700
    rows = {h: np.unique(np.concatenate([np.arange(h + 1, hubs), rng.integers(hubs, n, size=row)])) for h in range(hubs)}
    for v in range(hubs, n, 40):
        own = rng.integers(hubs, n, size=rng.integers(1, 6))
        rows[v] = np.unique(np.concatenate([own, rng.integers(0, popular, size=20)]) if popular else own)
    beg, adj = _csr(rows, n)
    _check(beg, adj)
    db, da = torch.from_numpy(beg).cuda(), torch.from_numpy(adj).cuda()
    r = T.count_tiles(db, da, 2, direction_split=1)
    assert r.triangles == O.count_forward_sorted_range(beg, adj, 0, n, 2, 8) and r.direction_split >= 1
