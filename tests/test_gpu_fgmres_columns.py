"""The solves of test_gpu_fgmres_fin.py are as long as they are meant to be: in
both forms more columns than one restart cycle holds, so a whole cycle of more
than 128 columns (more sums than a block of k_fg_fin has threads) and a restart
lie behind each."""
import pytest

from test_gpu_fgmres_fin import _solve

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dx,restart", [(0.02, 150), (0.0075, 150), (0.0075, 140)])
def test_the_long_cycles_are_long(api, dx, restart):
    for df in (1, 0):
        info = _solve(api, dx, df, restart)[1]
        assert restart > 128 and info["ppe_iters"] > restart and info["err_bits"] == 0
