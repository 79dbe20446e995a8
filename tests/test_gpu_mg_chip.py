"""The lower multigrid levels of a visit on chip (option mg_tail, k_mg_chip)
against one launch per level operation, at the sizes where its split can go
wrong: scenes whose levels all fit one block, scenes split over clusters of
two to sixteen blocks with odd grids and uneven columns, W-cycles on chip
(the visit's two passes with the residual between them), batches whose scenes
end on different levels.  The same operations in the same order: the states
are equal bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("x", "y", "vx", "vy", "p", "pid")


def _run(api, dxs, precision, wlev, prec, tail, fp32=1):
    from beachslope_gb300 import scene
    scenes = [scene.beach_scene(dx=dx, precision=precision) for dx in dxs]
    c = api.Context([q[0] for q in scenes], [q[1] for q in scenes], [q[2] for q in scenes], tuning="auto")
    c.set_option("mg_sub", 0)
    c.set_option("mg_exact", 0)
    c.set_option("mg_fp32", fp32)
    c.set_option("mg_wlev", wlev)
    c.set_option("mg_prec", prec)
    c.set_option("mg_tail", tail)
    level = c.get_option("mg_tail_level")
    c.prime()
    c.step(2)
    out = [c.download(s, full=False) for s in range(len(dxs))]
    iters = [c.info(s)["ppe_iters"] for s in range(len(dxs))]
    c.close()
    return level, out, iters


@pytest.mark.parametrize("dxs,precision,wlev,prec,fp32", [
    ([0.05], 1, 1, 1, 1),                       # a few hundred particles: one block
    ([0.027], 1, 2, 1, 1),
    ([0.0133], 1, 1, 0, 1),                     # no pre-sweep on the cell levels
    ([0.0071], 1, 3, 1, 1),                     # W-cycles on chip
    ([0.0047], 1, 0, 1, 1),
    ([0.0031], 1, 2, 1, 1),                     # both visits of a W-cycle level in one launch
    ([0.0133], 0, 1, 1, 0),                     # FP64 cycle
    ([0.0047], 0, 2, 1, 0),
    ([0.05, 0.011, 0.02, 0.031, 0.0083], 1, 1, 1, 1),   # uneven depths, one scene a single level
    ([0.05, 0.011, 0.0207], 0, 2, 1, 0),
])
def test_chip_levels_equal_separate_launches(api, dxs, precision, wlev, prec, fp32):
    level, a, ia = _run(api, dxs, precision, wlev, prec, 1, fp32)
    off, b, ib = _run(api, dxs, precision, wlev, prec, 0, fp32)
    assert level >= 1 and off == 0
    assert ia == ib
    for x, y in zip(a, b):
        for f in FIELDS:
            assert np.array_equal(x[f], y[f]), f
