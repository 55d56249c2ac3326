"""The preprocessing's sort, dedupe and orientation at the edges of their tiles (4096 keys), against
the oracle's pipeline byte for byte; pairs that are only 4-byte aligned; invalid ids."""
import ctypes as C

import numpy as np
import pytest

import trust_gb300 as T
from trust_gb300._lib import check
from oracle import oracle as O

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _pairs(rng, npairs, ids):
    hub = rng.integers(0, max(ids // 50, 1), size=npairs)
    return np.stack([np.where(rng.random(npairs) < 0.3, hub, rng.integers(0, ids, npairs)),
                     rng.integers(0, ids, npairs)], 1).astype(np.int32)


@pytest.mark.parametrize("npairs", [1, 2, 31, 4095, 4096, 4097, 8191, 12289, 100_003])
@pytest.mark.parametrize("ids", [1, 2, 3, 255, 256, 257, 40_000, 1 << 24])
def test_sizes_and_key_widths(npairs, ids):
    p = _pairs(np.random.default_rng(npairs * 7 + ids), npairs, ids)
    eb, ea = O.build_csr(p, ids)
    gb, ga = T.build_csr(torch.from_numpy(p).cuda(), ids)
    np.testing.assert_array_equal(gb.cpu().numpy(), eb)
    np.testing.assert_array_equal(ga.cpu().numpy(), ea)


def test_unaligned_pairs_and_invalid_ids():
    rng = np.random.default_rng(3)
    ids, k = 5000, 50_001
    p = _pairs(rng, k, ids)
    ok = p.copy()
    bad = rng.choice(k, 500, replace=False)
    p[bad[:200], 0] = -1 - rng.integers(0, 1000, 200)
    p[bad[200:350], 1] = ids + rng.integers(0, 1000, 150)
    p[bad[350:], 1] = p[bad[350:], 0]
    keep = np.ones(k, dtype=bool)
    keep[bad] = False
    eb, ea = O.build_csr(ok[keep], ids)
    raw = torch.empty(2 * k + 1, dtype=torch.int32, device="cuda")
    raw[1:] = torch.from_numpy(p).cuda().view(-1)
    for off in (0, 1):  # 8-byte and 4-byte aligned
        buf = raw[1:].clone() if off == 0 else raw
        pb, pa, n, m = C.c_void_p(), C.c_void_p(), C.c_int64(), C.c_int64()
        lib = T.load()
        check(lib.trust_tc_build_csr_device(None, C.c_void_p(buf.data_ptr() + 4 * off), k, ids, C.byref(pb), C.byref(pa),
                                            C.byref(n), C.byref(m)), "build")
        beg = torch.empty(n.value + 1, dtype=torch.int64, device="cuda")
        adj = torch.empty(m.value, dtype=torch.int32, device="cuda")
        check(lib.trust_tc_copy(C.c_void_p(beg.data_ptr()), pb, 8 * (n.value + 1)), "copy")
        check(lib.trust_tc_copy(C.c_void_p(adj.data_ptr()), pa, 4 * m.value), "copy")
        lib.trust_tc_free_device(pb)
        lib.trust_tc_free_device(pa)
        np.testing.assert_array_equal(beg.cpu().numpy(), eb)
        np.testing.assert_array_equal(adj.cpu().numpy(), ea)


def test_no_pairs():
    beg, adj = T.build_csr(torch.empty((0, 2), dtype=torch.int32, device="cuda"), 7)
    assert beg.tolist() == [0] and adj.numel() == 0


@pytest.mark.parametrize("npairs", [1, 2, 5000])
@pytest.mark.parametrize("over", [-1, 0, 1, 100_000, (1 << 26)])
def test_ids_far_apart(npairs, over):
    """Around as many ids as the pairs have ends (out-degrees by id, then by compacted id), renumbered and in
    batches, where the order is kept."""
    ids = 2 * npairs + over
    rng = np.random.default_rng(ids)
    p = rng.integers(0, ids, size=(npairs, 2)).astype(np.int32)
    p[-1] = [0, ids - 1]
    eb, ea = O.build_csr(p, ids)
    gb, ga = T.build_csr(torch.from_numpy(p).cuda(), ids)
    np.testing.assert_array_equal(gb.cpu().numpy(), eb)
    np.testing.assert_array_equal(ga.cpu().numpy(), ea)
    from trust_gb300 import batch as B
    bb, ba, gv = B.build_batch(torch.from_numpy(p).cuda(), np.array([0, ids // 3, ids], dtype=np.int64))
    present = np.unique(p[p[:, 0] != p[:, 1]])
    e = np.unique(np.sort(np.searchsorted(present, p[p[:, 0] != p[:, 1]]), axis=1), axis=0)
    deg = np.bincount(e.ravel(), minlength=present.size)
    e[deg[e[:, 0]] > deg[e[:, 1]]] = e[deg[e[:, 0]] > deg[e[:, 1]]][:, ::-1]
    e = e[np.lexsort((e[:, 1], e[:, 0]))]
    np.testing.assert_array_equal(ba.cpu().numpy(), e[:, 1])
    np.testing.assert_array_equal(np.diff(bb.cpu().numpy()), np.bincount(e[:, 0], minlength=present.size))
    assert list(gv) == [0, int(np.searchsorted(present, ids // 3)), present.size]
