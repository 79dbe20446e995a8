"""How many columns or iterations of a host CSR solve are launched between two
looks at the converged count: no more than a restart cycle holds, so that a
short cycle does not run empty columns, and one iteration of BiCGStab on small
systems (host logic, no GPU)."""
import numpy as np
import pytest

from _fake_gpu import FakeGpu


def _identity(n):
    return np.arange(n + 1, dtype=np.int32), np.arange(n, dtype=np.int32), np.ones(n), np.ones(n), np.zeros(n)


@pytest.mark.parametrize("n", [5, 9801])
@pytest.mark.parametrize("restart,want", [(1, 1), (2, 2), (3, 3), (4, 4), (30, 4), (150, 4)])
def test_fgmres_columns(monkeypatch, tmp_path, n, restart, want):
    gpu = FakeGpu(monkeypatch, tmp_path)
    gpu.api.fgmres_csr(*_identity(n), maxit=1, restart=restart)
    assert len(gpu.calls("k_fg_arn1")) == want   # (a captured chunk is recorded once)


@pytest.mark.parametrize("n,want", [(5, 1), (1023, 1), (1024, 4), (20000, 4)])
def test_bicgstab_iterations(monkeypatch, tmp_path, n, want):
    gpu = FakeGpu(monkeypatch, tmp_path)
    gpu.api.bicgstab_csr(*_identity(n), maxit=1)
    assert len(gpu.calls("k_it1_64")) == want
