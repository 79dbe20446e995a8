"""FGMRES on CSR systems at the sizes where its reductions change form: one
row, one block and one row more, 64 row blocks (the last size whose sums one
block takes) and one row more, and cycles long enough that every lane of the
rotations' scan holds several of them, across restarts too.  Against the CPU
restatement: the same columns, solutions equal to the solve's tolerance times
the systems' condition (below 2e3: rows sum to 1/500 of their diagonal or
more), and the residual from numpy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _system(n, seed):
    rng = np.random.default_rng(seed)
    i = np.arange(n)
    rows, cols, vals = [i], [i], [np.full(n, 1.0)]
    for d in (-61, -7, -1, 1, 7, 61):
        ok = (i + d >= 0) & (i + d < n)
        rows.append(i[ok])
        cols.append(i[ok] + d)
        vals.append(-rng.uniform(0.6, 1.4, int(ok.sum())))
    rows, cols, vals = np.concatenate(rows), np.concatenate(cols), np.concatenate(vals)
    off = -np.bincount(rows[n:], weights=vals[n:], minlength=n)
    vals[:n] = np.maximum(off * 1.002, 1.0)
    vals = vals / vals[:n][rows]
    order = np.lexsort((cols, rows))
    ptr = np.zeros(n + 1, np.int32)
    ptr[1:] = np.cumsum(np.bincount(rows, minlength=n))
    return ptr, cols[order].astype(np.int32), vals[order], rows[order], rng.standard_normal(n)


@pytest.mark.parametrize("n,restart", [(1, 150), (5, 3), (256, 150), (257, 40), (16384, 150), (16385, 150), (16385, 60)])
def test_fgmres_reductions(api, oracle, n, restart):
    ptr, col, val, row, b = _system(n, n + restart)
    tol = 1e-10
    rc, x, it, rr = api.fgmres_csr(ptr, col, val, b, np.zeros(n), tol=tol, maxit=2000, restart=restart, rule=0)
    ref = oracle.fgmres_csr(ptr, col, val, b, np.zeros(n), tol=tol, maxit=2000, restart=restart, rule=0)
    assert (rc, it) == (ref[0], ref[2])
    if rc:   # five rows restarted every three columns stagnate, here as there
        assert n == 5 and it == 2000
        return
    res = np.linalg.norm(b - np.bincount(row, weights=val * x[col], minlength=n)) / np.linalg.norm(b)
    assert res <= 1.01 * tol + 1e-13
    assert np.linalg.norm(x - ref[1]) <= 2e3 * tol * np.linalg.norm(ref[1])
