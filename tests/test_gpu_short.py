"""The short-row kernel (tc_short.cu: graphs of 65,536 rows or more, none longer than 8) against the
oracle: rows of every length, unsorted and with duplicates, unaligned neighbour arrays, row ranges,
and the schedules and graphs that do not take it."""
import numpy as np
import pytest

import trust_gb300 as T
from oracle import oracle as O

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _graph(seed, n, longest, sorted_rows):
    rng = np.random.default_rng(seed)
    d = rng.integers(0, longest + 1, size=n)
    d[n // 3] = longest
    beg = np.concatenate([[0], np.cumsum(d)]).astype(np.int64)
    src = np.repeat(np.arange(n), d)
    adj = np.where(rng.random(src.size) < 0.8, (src + rng.integers(1, 60, src.size)) % n,
                   rng.integers(0, n, src.size)).astype(np.int32)
    if sorted_rows:  # strictly increasing rows: what the direction split needs
        key = np.unique(src.astype(np.int64) << 32 | adj)
        src, adj = key >> 32, (key & 0xFFFFFFFF).astype(np.int32)
        beg = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))]).astype(np.int64)
    return beg, adj


@pytest.mark.parametrize("n", [65_536, 65_567, 200_001])
@pytest.mark.parametrize("longest", [2, 4, 5, 8, 9])
@pytest.mark.parametrize("sorted_rows", [False, True])
def test_short_rows(n, longest, sorted_rows):
    beg, adj = _graph(n + sorted_rows, n, longest, sorted_rows)
    expect = O.count_forward(beg, adj, threads=8)
    db = torch.from_numpy(beg).cuda()
    buf = torch.zeros(adj.size + 8, dtype=torch.int32, device="cuda")
    with T.Context() as ctx:
        for off in (0, 1, 2, 3):  # 16-byte aligned and not
            view = buf[off:off + adj.size]
            view.copy_(torch.from_numpy(adj))
            r = T.count_csr(db, view, ctx=ctx)
            assert r.triangles == expect and r.wedges == O.wedges(beg, adj)
        da = torch.from_numpy(adj).cuda()
        plain = T.count_csr(db, da, ctx=ctx, schedule=T.SCHED_PLAIN)
        assert plain.triangles == expect
        cuts = [0, 7, n // 2 + 5, n]
        parts = [T.count_csr(db, da, ctx=ctx, schedule=T.SCHED_TUNED, row_range=(a, b)).triangles
                 for a, b in zip(cuts[:-1], cuts[1:])]
        assert sum(parts) == expect
        d = np.diff(beg)
        r = T.count_csr(db, da, ctx=ctx, schedule=T.SCHED_TUNED)
        assert r.class_sizes["g4"] == int(np.sum((d >= 2) & (d <= 4)))
        assert r.class_sizes["g8"] == int(np.sum((d > 4) & (d <= 8)))
        for sch in (T.SCHED_TUNED, T.SCHED_LEARNED):
            s = T.count_csr(db, da, ctx=ctx, schedule=sch, direction_split=1)
            assert s.triangles == expect and s.direction_split == int(sorted_rows)
        cyc = torch.zeros(n, dtype=torch.int64, device="cuda")
        assert T.count_csr(db, da, ctx=ctx, cycles=cyc).triangles == expect
        assert int(cyc.sum()) > 0  # recorded by the general kernel
