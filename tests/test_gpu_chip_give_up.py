"""The on-chip multigrid levels (k_mg_chip) when a block's wait for its
constants runs out: the scene's error is set, the cluster's blocks leave
together, nothing hangs, the other scenes' results and the context's next
solves are those of a context where it never happened.  The wait is made to
run out by giving one block of each cluster no tries."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BREAK = 0x04   # BS_ERR_SOLVER_BREAK
FIELDS = ("x", "y", "vx", "vy", "p", "pid")


def _lose(api, c, rank):
    f = api.lib.bs_mg_chip_lose
    f.restype, f.argtypes = C.c_int, [C.c_void_p, C.c_int32]
    assert f(c.h, rank) == 0


def _same(a, b):
    return all(np.array_equal(a[f], b[f]) for f in FIELDS)


@pytest.mark.parametrize("dxs,precision,blocks,rank,hit", [
    ([0.05], 1, 1, 0, [True]),                     # one block does it all
    ([0.027], 1, 2, 1, [True]),
    ([0.0133], 1, 8, 0, [True]),                   # the block of the levels that are not split
    ([0.0133], 1, 8, 5, [True]),
    ([0.0133], 0, 8, 7, [True]),
    ([0.0047], 1, 16, 15, [True]),
    ([0.05, 0.011, 0.02], 1, 8, 2, [False, True, True]),   # the first scene's levels are not split: its block 2 rests
])
def test_a_block_that_gives_up_takes_its_cluster_along(api, dxs, precision, blocks, rank, hit):
    from beachslope_gb300 import scene
    scenes = [scene.beach_scene(dx=dx, precision=precision) for dx in dxs]

    def context():
        c = api.Context([q[0] for q in scenes], [q[1] for q in scenes], [q[2] for q in scenes], tuning="auto")
        for k, v in (("mg_sub", 0), ("mg_exact", 0), ("mg_fp32", precision), ("mg_wlev", 1)):
            c.set_option(k, v)
        c.prime()
        return c

    want = context()
    want.step(1)
    first = [want.download(s, full=False) for s in range(len(dxs))]
    want.step(1)
    second = [want.download(s, full=False) for s in range(len(dxs))]
    want.close()

    c = context()
    assert c.get_option("mg_tail_blocks") == blocks
    _lose(api, c, rank)
    c.step(1)
    for s in range(len(dxs)):
        assert bool(c.info(s)["err_bits"] & BREAK) == hit[s]
        if not hit[s]:
            assert c.info(s)["err_bits"] == 0 and _same(c.download(s, full=False), first[s])
    _lose(api, c, -1)
    for s, q in enumerate(scenes):
        c.upload(s, q[1], q[2])
    c.clear_errors()
    c.prime()
    c.step(2)
    for s in range(len(dxs)):
        assert c.info(s)["err_bits"] == 0
        assert _same(c.download(s, full=False), second[s])
    c.close()
