"""Counting calls where most of the device's memory is taken: the split's scratch does not fit, the count
is made without it."""
import pytest

import trust_gb300 as T

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

MIB = 1 << 20


@pytest.fixture(scope="module")
def graph():
    beg, adj = T.build_csr(T.gen_rmat(20, 16, seed=2), 1 << 20)  # 15.7 M arcs, the split pays
    with T.Context() as ctx:  # every kernel and its module loaded while there is room
        on = T.count_csr(beg, adj, ctx=ctx)
        off = T.count_csr(beg, adj, ctx=ctx, schedule=T.SCHED_TUNED, direction_split=0)
        assert on.direction_split == 1 and off.triangles == on.triangles
    return beg, adj, on.triangles


def _hold(room):
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.empty(torch.cuda.mem_get_info()[0] - room * MIB, dtype=torch.uint8, device="cuda")


@pytest.mark.parametrize("split", [-1, 0, 1])
@pytest.mark.parametrize("room", [128, 256, 384, 448, 512, 1024])
def test_count_without_room_for_the_split(graph, room, split):
    """Per arc the scheduling pass takes 14 bytes (215 MB here) and the block bitmaps 9 more (145 MB);
    the unsplit count takes about 60 MB in all."""
    beg, adj, expect = graph
    with T.Context() as ctx:
        held = _hold(room)
        try:
            for _ in range(2):
                r = T.count_csr(beg, adj, ctx=ctx, direction_split=split)
                assert r.triangles == expect
        finally:
            del held
            torch.cuda.empty_cache()
        assert r.direction_split in ((0,) if split == 0 or room <= 256 else (1,) if room == 1024 else (0, 1))
        if split:  # the context is whole again
            r = T.count_csr(beg, adj, ctx=ctx, direction_split=split)
            assert r.triangles == expect and r.direction_split == 1
