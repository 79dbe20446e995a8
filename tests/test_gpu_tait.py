"""Tait's power and root (WCSPH equation of state and its inverse): exponent 7 by
products and Newton steps, any other by pow.  Against the same expressions in
extended precision.  The argument (three products, a division, a sum) is exact to
the bits of numpy's; the root and the product with rho then round once each: 2
ulp = 4.5e-16 of the density.  The power's error (1 ulp at most) counts absolutely
in x^gam - 1: 2.3e-16 x^gam B / gam, and three further roundings of the pressure."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gamma", [7.0, 6.5, 1.0])
def test_tait_against_extended_precision(api, gamma):
    from beachslope_gb300 import scene
    p, st, _ = scene.lattice_scene(n=64, dx=1e-3, seed=4)
    p.wc_gamma = gamma
    rng = np.random.default_rng(8)
    n = len(st["x"])
    B = p.rho * (p.wc_c0 * p.wc_c0)
    press = np.concatenate([rng.uniform(0.0, 1.0, n // 4) * B, 10.0 ** rng.uniform(-8, 8, n // 4) * B,
                            rng.uniform(-0.14, 0.14, n - 2 * (n // 4)) * B / gamma])
    rng.shuffle(press)
    press[:3] = 0.0, B * 1e20, B * 1e40   # the last beyond FP32's range
    ctx = api.Context([p], [dict(st, p=press)], [None])
    before = ctx.download()
    ctx.stage("wcsph_pressure_to_density")
    got = ctx.download()["rho"]
    L = np.longdouble
    arg = before["p"] * gamma / B + 1
    # pow takes the exponent 1 / gamma rounded to FP64, the seventh root is exact
    root = np.where((gamma == 7.0) & (arg < 2.0 ** 100), L(1) / L(7), L(1.0 / gamma))
    ref = L(p.rho) * L(arg) ** root
    assert np.all(np.abs(L(got) - ref) <= L(4.5e-16) * ref)
    rho = p.rho * rng.uniform(0.98, 1.3, n)
    ctx.set_fields({"rho": rho})
    ctx.stage("wcsph_eos")
    out = ctx.download()
    fluid = out["tid"] > 2
    pw = L(rho / p.rho) ** L(gamma)
    ref = L(B) * (pw - 1) / L(gamma)
    ref = np.where(ref < 0, L(0), ref)
    tol = L(2.3e-16) * pw * L(B) / L(gamma) + L(4.5e-16) * np.abs(ref)
    assert np.all(np.abs(L(out["p"]) - ref)[fluid] <= tol[fluid])
