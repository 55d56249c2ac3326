"""The batch counting kernel (tc_batch_count.cu) where its row sets change: graphs around the sizes
whose ids fit a warp's bitmap or half of it, rows of every class up to spill tables, dense graphs,
and buffers refilled after the batch was made."""
import numpy as np
import pytest

import trust_gb300 as T
from trust_gb300 import _lib
from trust_gb300 import batch as B
from oracle import oracle as O
from tests import graphs

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _er(rng, n, deg):
    return O.build_csr(rng.integers(0, n, size=(n * deg // 2, 2)).astype(np.int32), n)


def _hub(rng, n, longest):
    """Row 0 of `longest` entries, every other row up to 40: not oriented, sorted, no duplicates."""
    rows = [np.sort(rng.choice(n, size=longest, replace=False))]
    rows += [np.unique(rng.integers(0, n, size=rng.integers(0, 41))) for _ in range(n - 1)]
    beg = np.concatenate([[0], np.cumsum([r.size for r in rows])]).astype(np.int64)
    return beg, np.concatenate(rows).astype(np.int32)


def _union(csrs):
    vb = np.concatenate([[0], np.cumsum([b.size - 1 for b, _ in csrs])]).astype(np.int64)
    eb = np.concatenate([[0], np.cumsum([a.size for _, a in csrs])]).astype(np.int64)
    beg = np.concatenate([b[:-1] + eb[g] for g, (b, _) in enumerate(csrs)] + [eb[-1:]])
    adj = np.concatenate([a + np.int32(vb[g]) for g, (_, a) in enumerate(csrs)])
    return torch.from_numpy(beg).cuda(), torch.from_numpy(adj.astype(np.int32)).cuda(), vb


def _check(csrs, settings=((256, 128, 8),)):
    beg, adj, vb = _union(csrs)
    expect = np.array([O.count_forward(b, a, threads=8) for b, a in csrs], dtype=np.uint64)
    wedges = sum(O.wedges(b, a) for b, a in csrs)
    with T.Context() as ctx:
        bt = B.Batch(beg, adj, vb, ctx=ctx)
        for threads, warp_max, chunk in settings:
            for s in range(4):
                bt.set_class(s, threads, warp_max, chunk)
            for _ in range(2):
                counts, r = bt.run()
                assert np.array_equal(counts, expect)
                assert r.triangles == int(expect.sum()) and r.wedges == wedges
        bt.close()


@pytest.mark.parametrize("n", [25_088, 25_089, 50_176, 50_177, 51_200, 51_201, 70_000])
def test_bitmap_bounds(n):
    rng = np.random.default_rng(n)
    _check([_er(rng, n, 24), _er(rng, 300, 40), _er(rng, n, 64), _er(rng, 7, 3)])


@pytest.mark.parametrize("settings", [((256, 128, 8), (1024, 64, 4)), ((64, 32, 1), (512, 1024, 16))])
def test_every_class(settings):
    rng = np.random.default_rng(11)
    cs = [O.build_csr(graphs.complete(k)[0], k) for k in (3, 5, 9, 17, 33, 34, 130, 300)]
    cs += [_hub(rng, 6000, 5000), _hub(rng, 90_000, 3000), _er(rng, 900, 100)]
    _check(cs, settings)


def test_refilled_buffers():
    """A run counts what the buffers hold: other graphs of the same sizes, and an arc that leaves its
    graph (out of its bitmap's range) is looked up as any other entry."""
    rng = np.random.default_rng(5)
    cs = [_er(rng, 400, 30), _er(rng, 400, 30)]
    beg, adj, vb = _union(cs)
    with T.Context() as ctx:
        bt = B.Batch(beg, adj, vb, ctx=ctx)
        a = adj.cpu().numpy().copy()
        b = beg.cpu().numpy()
        v = int(np.argmax(np.diff(b)[:400]))  # a long row of graph 0: its last two entries leave the graph
        a[b[v + 1] - 2:b[v + 1]] = [int(vb[1]) + 3, int(vb[1]) + 4]
        adj.copy_(torch.from_numpy(a))
        counts, r = bt.run()
        assert r.triangles == int(counts.sum()) == O.count_forward(b, a)
        bt.close()


@pytest.mark.parametrize("made,refilled", [(100, 5000), (4096, 4097), (5000, 4097), (4097, 9000)])
def test_refilled_with_longer_rows(made, refilled):
    """Buffers refilled with a row longer than any the batch was made for are counted or refused, never
    counted in part."""
    rng = np.random.default_rng(made + refilled)
    (beg, adj, vb), (b, a) = _union([_hub(rng, 12_000, made)]), _hub(rng, 12_000, refilled)
    if a.size > adj.numel():  # the same number of entries: the first rows' are kept
        b, a = np.minimum(b, adj.numel()), a[:adj.numel()]
    else:
        b = b.copy()
        b[-1] = adj.numel()  # the last row takes the rest, repeated entries
        a = np.concatenate([a, np.full(adj.numel() - a.size, 7, dtype=np.int32)])
    expect = O.count_forward(b, a, threads=8)
    with T.Context() as ctx:
        bt = B.Batch(beg, adj, vb, ctx=ctx)
        beg.copy_(torch.from_numpy(b))
        adj.copy_(torch.from_numpy(a))
        try:
            counts, r = bt.run()
            assert r.triangles == int(counts[0]) == expect
            assert made > 4096
        except T.TrustTcError as e:
            assert e.status == _lib.E_DEVICE and refilled > made
        bt.close()


@pytest.mark.parametrize("which,at,value,status", [("adj", 0, -1, _lib.E_IDS), ("adj", -1, 1 << 30, _lib.E_IDS),
                                                   ("beg", 0, 2, _lib.E_OFFSETS), ("beg", 300, -5, _lib.E_OFFSETS),
                                                   ("beg", 300, 1 << 40, _lib.E_OFFSETS), ("beg", -1, 1, _lib.E_OFFSETS)])
def test_refilled_with_invalid_input(which, at, value, status):
    """Refilled buffers are validated by every run before a row or entry of theirs is indexed."""
    rng = np.random.default_rng(7)
    cs = [_er(rng, 400, 30), _hub(rng, 6000, 5000), _er(rng, 3000, 6)]
    beg, adj, vb = _union(cs)
    expect = [O.count_forward(b, a) for b, a in cs]
    with T.Context() as ctx:
        bt = B.Batch(beg, adj, vb, ctx=ctx)
        x = beg if which == "beg" else adj
        keep = x[at].clone()
        x[at] = value
        with pytest.raises(T.TrustTcError) as e:
            bt.run()
        assert e.value.status == status
        x[at] = keep
        assert list(bt.run()[0]) == expect
        bt.close()


@pytest.mark.parametrize("n", [55_423, 55_424, 55_425, 120_000])
@pytest.mark.parametrize("share", [0, 1, 2])
def test_graphs_around_the_bitmap_bound(n, share):
    """Graphs whose ids just fit the words of a warp, just do not, or by far do not, alone and beside as many
    vertices, or more, in graphs that do (bitmaps only where those hold half of the vertices)."""
    rng = np.random.default_rng(n + share)
    cs = [_er(rng, n, d) for d in (6, 30, 64)] + [_hub(rng, n, 4500)]
    cs += [_er(rng, 40_000, 30) for _ in range(share * len(cs) * n // 40_000)] + [_er(rng, 50, 49), _hub(rng, 8000, 70)]
    _check(cs, ((256, 128, 8), (1024, 64, 4)))
