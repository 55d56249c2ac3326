"""The one-launch path for small graphs (tc_small.cu) against the oracle: any CSR (unsorted rows,
duplicates, self-loops), its size bounds, dense graphs whose rows are shared by several warps, row
ranges, and invalid input at every position."""
import numpy as np
import pytest

import trust_gb300 as T
from trust_gb300 import _lib
from oracle import oracle as O
from tests import graphs

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _dev(beg, adj):
    return (torch.from_numpy(np.ascontiguousarray(beg, dtype=np.int64)).cuda(),
            torch.from_numpy(np.ascontiguousarray(adj, dtype=np.int32)).cuda())


@pytest.fixture(scope="module")
def ctx():
    with T.Context() as c:
        yield c


def _same_as_general(ctx, beg, adj, expect):
    db, da = _dev(beg, adj)
    r = T.count_csr(db, da, ctx=ctx)
    g = T.count_csr(db, da, ctx=ctx, chunk=8)  # a launch parameter: the general path
    assert r.triangles == g.triangles == expect
    assert (r.wedges, r.max_out_degree, r.class_sizes) == (g.wedges, g.max_out_degree, g.class_sizes)
    assert r.wedges == O.wedges(beg, adj)
    h = T.count_csr(beg, adj, ctx=ctx)  # host input
    assert h.triangles == expect


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, 65, 500])
@pytest.mark.parametrize("max_deg", [1, 3, 32, 33, 200])
def test_any_csr(ctx, n, max_deg):
    rng = np.random.default_rng(n * 1000 + max_deg)
    for _ in range(3):
        beg, adj = graphs.random_csr(rng, n, max_deg)
        _same_as_general(ctx, beg, adj, O.count_forward(beg, adj))


@pytest.mark.parametrize("n", [65_535, 65_536, 65_537])
@pytest.mark.parametrize("m", [100_000, (1 << 21) - 1, 1 << 21])
def test_size_bounds(ctx, n, m):
    rng = np.random.default_rng(n + m)
    d = rng.multinomial(m, np.full(n, 1 / n))
    beg = np.concatenate([[0], np.cumsum(d)]).astype(np.int64)
    adj = rng.integers(0, n, size=m).astype(np.int32)
    adj[rng.random(m) < 0.2] = n - 1
    _same_as_general(ctx, beg, adj, O.count_forward(beg, adj, threads=8))


@pytest.mark.parametrize("n", [40, 130, 300, 600])
def test_dense(ctx, n):
    pairs, tri = graphs.complete(n)
    beg, adj = O.build_csr(pairs, n)
    _same_as_general(ctx, beg, adj, tri)
    whole = 0
    for lo, hi in ((0, 1), (1, n // 3), (n // 3, n)):
        r = T.count_csr(*_dev(beg, adj), ctx=ctx, row_range=(lo, hi))
        assert r.triangles == O.count_forward_sorted_range(beg, adj, lo, hi, 2, 1)
        whole += r.triangles
    assert whole == tri


def test_invalid_input(ctx):
    rng = np.random.default_rng(2)
    n = 300
    beg, adj = graphs.random_csr(rng, n, 60, 0, 0)
    expect = O.count_forward(beg, adj)
    for pos in (0, 1, 31, 32, adj.size // 2, adj.size - 1):
        for bad in (-1, n, 2**31 - 1):
            a = adj.copy()
            a[pos] = bad
            with pytest.raises(T.TrustTcError) as e:
                T.count_csr(*_dev(beg, a), ctx=ctx)
            assert e.value.status == _lib.E_IDS
            assert T.count_csr(*_dev(beg, adj), ctx=ctx).triangles == expect  # the context is clean again
    for pos, val in ((0, 1), (1, -5), (n // 2, 2**40), (n // 2, -(2**40)), (n, adj.size - 1), (n, adj.size + 1)):
        b = beg.copy()
        b[pos] = val
        with pytest.raises(T.TrustTcError) as e:
            T.count_csr(*_dev(b, adj), ctx=ctx)
        assert e.value.status == _lib.E_OFFSETS
        assert T.count_csr(*_dev(beg, adj), ctx=ctx).triangles == expect


@pytest.mark.parametrize("longest", [511, 512, 513, 1025, 16_384, 16_385, 60_000])
@pytest.mark.parametrize("n,short", [(65_536, 2), (20_000, 40)])
def test_long_rows(ctx, longest, n, short):
    """Rows at the bounds of what a warp takes, one or several warps to a row (n, short), that point at each
    other, with repeated entries, counted or not (slices), unsorted, and with an invalid entry."""
    rng = np.random.default_rng(longest + n)
    lens = rng.integers(0, 2 * short, size=n)
    hubs = rng.choice(n, 5, replace=False)
    lens[hubs] = (longest, longest - 1, 700, longest, 0)
    beg = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    adj = rng.integers(0, n, size=int(beg[-1])).astype(np.int32)
    for h in hubs[:4]:
        adj[beg[h]:beg[h] + 5] = hubs
    if adj.size >= 1 << 21:
        pytest.skip("not a small graph")
    _same_as_general(ctx, beg, adj, O.count_forward(beg, adj, threads=8))
    db, da = _dev(beg, adj)
    cuts = (0, int(hubs[0]), int(hubs[0]) + 1, n)
    parts = [T.count_csr(db, da, ctx=ctx, row_range=(a, b)) for a, b in zip(cuts[:-1], cuts[1:]) if a < b]
    assert sum(r.triangles for r in parts) == O.count_forward(beg, adj, threads=8)
    assert sum(r.wedges for r in parts) == O.wedges(beg, adj)
    for row_range in (None, (int(hubs[0]) + 1, n)):  # the entry's row is counted, and is only checked
        bad = da.clone()
        bad[int(beg[hubs[0]]) + longest // 2] = n
        with pytest.raises(T.TrustTcError) as e:
            T.count_csr(db, bad, ctx=ctx, row_range=row_range)
        assert e.value.status == _lib.E_IDS


@pytest.mark.parametrize("splits", [1, 2, 8])
def test_rows_shared_by_warps_and_long(ctx, splits):
    """Rows of up to `splits` times a warp's bound stay with their warps, longer ones do not."""
    n = 2000
    rng = np.random.default_rng(splits)
    fill = 16 * n * splits // n + 8 if splits < 8 else 140
    lens = np.full(n, fill)
    for k, d in enumerate((512 * splits - 1, 512 * splits, 512 * splits + 1, 512 * splits + 33)):
        lens[3 * k] = d
    beg = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    adj = rng.integers(0, n, size=int(beg[-1])).astype(np.int32)
    assert min(8, max(1, adj.size // (16 * n))) == splits
    _same_as_general(ctx, beg, adj, O.count_forward(beg, adj, threads=8))


@pytest.mark.parametrize("length", [2, 500, 5000, 60_000])
def test_overlapping_rows_end_early(ctx, length):
    """Offsets that go back and forth make every other row overlap, with more arcs in all than can be walked:
    refused at once."""
    import time
    n = 60_000
    beg = np.zeros(n + 1, dtype=np.int64)
    beg[1::2] = length
    beg[-1] = 1_900_000
    beg[-2] = 0
    adj = np.zeros(1_900_000, dtype=np.int32)
    db, da = _dev(beg, adj)
    t = time.perf_counter()
    with pytest.raises(T.TrustTcError) as e:
        T.count_csr(db, da, ctx=ctx)
    assert e.value.status == _lib.E_OFFSETS and time.perf_counter() - t < 5.0
    ok, tri = graphs.complete(40)
    assert T.count_csr(*_dev(*O.build_csr(ok, 40)), ctx=ctx).triangles == tri


_CAPTURE = """
import ctypes as C
import torch
import trust_gb300 as T
from trust_gb300 import _lib
from oracle import oracle as O
from tests import graphs
pairs, expect = graphs.complete(60)
db, da = (torch.from_numpy(x).cuda() for x in O.build_csr(pairs, 60))
# no zeroed memory by chance: freed blocks of the accumulators' size that held offsets
dirty, lib, p = [], T.load(), torch.from_numpy(pairs).cuda()
for _ in range(64):
    x = [C.c_void_p(), C.c_void_p(), C.c_int64(), C.c_int64()]
    T.check(lib.trust_tc_build_csr_device(None, C.c_void_p(p.data_ptr()), p.shape[0], 60, *[C.byref(y) for y in x]), "")
    dirty.append(x)
for x in dirty:
    lib.trust_tc_free_device(x[0])
with T.Context() as c:
    s = torch.cuda.Stream()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.stream(s):
        g.capture_begin(capture_error_mode="relaxed")
        try:
            T.count_csr(db, da, ctx=c, stream=s.cuda_stream)
            status = _lib.OK
        except T.TrustTcError as e:
            status = e.status
        try:
            g.capture_end()
        except RuntimeError:  # the capture is invalid
            pass
    assert status == _lib.E_CUDA, status
    for _ in range(2):
        assert T.count_csr(db, da, ctx=c).triangles == expect
print("counted")
"""


def test_first_call_on_a_capturing_stream():
    """A call cannot be captured (it synchronises): it fails, and the context's next call counts.  In a
    process of its own: torch's allocator keeps a failed capture's state."""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", _CAPTURE], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "counted", r.stderr[-2000:]


def test_callers_streams_and_contexts_at_once():
    """Non-blocking streams and several contexts at a time, one host thread each."""
    import threading
    rng = np.random.default_rng(3)
    beg, adj = graphs.random_csr(rng, 500, 90)
    expect = O.count_forward(beg, adj)
    pairs = T.gen_rmat(15, 24, 0.7, 0.125, 0.125, seed=3)
    big = T.build_csr(pairs, 1 << 15)
    whole = O.count_forward(*(x.cpu().numpy() for x in big), threads=8)
    torch.cuda.synchronize()
    wrong = []

    def work(k):
        s = torch.cuda.Stream()
        db, da = _dev(beg, adj)
        torch.cuda.synchronize()
        with T.Context() as c:
            for _ in range(20):
                r = T.count_csr(db, da, ctx=c, stream=s.cuda_stream)
                b = T.count_csr(*big, ctx=c, stream=s.cuda_stream, direction_split=1)
                if r.triangles != expect or b.triangles != whole or b.direction_split != 1:
                    wrong.append((k, r, b))

    ts = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not wrong
