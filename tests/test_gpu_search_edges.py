"""The neighbour and grain scans where their batches and shortcuts can go wrong:
a lattice whose points lie on the middles of the cells and exactly 2h apart
(with and without a jitter far below FP32's resolution of a cell), cells holding
none to many grains, grains on particles, and fluid clear of all grains.  The
neighbour lists are the CPU restatement's in order; FP64 porosity and drag are
its values to rounding.  Mixed porosity: a compensated sum of FP32 kernel values,
each within 8 ulp (5e-7 of it), clamped at 1 - por, so within 1e-6; the drag's
terms go with (1 - phi)^2 / phi^3 and (1 - phi) / phi^3, so within 2 / (1 - por)
+ 3 / por of that (below 20) of the largest."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("dx,jitter,hfac", [(2.0 ** -10, 0.0, 1.0), (1e-3, 0.0, 1.0), (1e-3, 1e-9, 1.0),
                                            (2.0 ** -10, 0.0, 2.0), (1e-3, 0.3, 1.3)])
def test_scan_edges(api, oracle, dx, jitter, hfac, mixed):
    from beachslope_gb300 import abi, scene
    p, st, _ = scene.lattice_scene(n=21, dx=dx, jitter=jitter, hfac=hfac)
    p.kmax = 64
    p.precision = abi.PREC_MIXED if mixed else abi.PREC_FP64
    rng = np.random.default_rng(3)
    # grains over the lower left part: a few to many per cell, some on particles
    gx = np.concatenate([rng.uniform(0.0, 14 * dx, 90), st["x"][-441:-300:7], np.full(17, 9.25 * dx)])
    gy = np.concatenate([rng.uniform(0.0, 14 * dx, 90), st["y"][-441:-300:7], rng.uniform(6 * dx, 8 * dx, 17)])
    gr = {"x": gx, "y": gy, "mass": np.full(len(gx), 2650.0 * 0.3 * dx * dx), "rho": np.full(len(gx), 2650.0)}
    moving = st["tid"] == abi.TID_FLUID
    for k in ("vx", "vy"):   # every third fluid particle at rest
        st[k] = np.where(moving & (np.arange(len(moving)) % 3 > 0), rng.uniform(-1, 1, len(moving)), 0.0)
    ctx = api.Context([p], [st], [gr])
    o = oracle.Oracle(p, st, gr)
    for a, b in (("search", "neighbour"), ("porosity", "effpor")):
        ctx.stage(a)
        o.stage(b)
    cg, ig, *_ = ctx.neighbours()
    co, io, *_ = o.neighbours(p.kmax)
    np.testing.assert_array_equal(cg, co)
    m = np.arange(p.kmax)[None, :] < co[:, None]
    np.testing.assert_array_equal(ig[m], io[m])
    g, r = ctx.download(), o.get()
    clear = r["porosity"] == 1.0
    assert 0 < clear.sum() < len(clear)
    np.testing.assert_array_equal(g["porosity"][clear], 1.0)
    assert np.abs(g["porosity"] - r["porosity"]).max() <= (1e-6 if mixed else 1e-13)
    for k in ("resx", "resy"):
        np.testing.assert_array_equal(g[k][clear], 0.0)
        assert np.abs(g[k] - r[k]).max() <= (20 * 1e-6 if mixed else 1e-12) * np.abs(r[k]).max()
    # both halves in one launch (a priming pass) give what each gave alone
    both = api.Context([p], [st], [gr])
    both.prime()
    b = both.download()
    order = np.argsort(b["pid"])
    mine = np.argsort(g["pid"])
    np.testing.assert_array_equal(b["porosity"][order], g["porosity"][mine])
