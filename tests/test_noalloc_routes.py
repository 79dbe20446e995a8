"""bs_bicgstab_csr_noalloc where its cooperative launch is refused (a partition
of the device, a green context): the call runs its launches per phase instead
of failing, also when only a later chunk is refused (host logic, no GPU); and
on the GPU these launches give the cooperative kernel's iterates, bit for bit
(the same operations in the same order)."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_static_edges import _system


def _call(lib, name, n, ptrs, tol, maxit):
    f = getattr(lib, name)
    f.restype = C.c_int
    f.argtypes = [C.c_int32] + [C.c_void_p] * 5 + [C.c_double, C.c_int32, C.c_void_p, C.c_void_p, C.c_void_p]
    it, rr = C.c_int32(), C.c_double()
    return f(n, *ptrs, tol, maxit, None, C.byref(it), C.byref(rr)), it.value, rr.value


@pytest.mark.parametrize("n", [1, 300, 65536])
@pytest.mark.parametrize("refused", [False, True])
def test_refused_cooperative_launch(monkeypatch, tmp_path, n, refused):
    from _fake_gpu import FakeGpu
    gpu = FakeGpu(monkeypatch, tmp_path)
    arrays = [np.zeros(n + 1, np.int32), np.zeros(1, np.int32), np.zeros(1), np.zeros(n), np.zeros(n)]
    gpu.lib.fake_refuse_cooperative(720 if refused else 0)   # cudaErrorCooperativeLaunchTooLarge
    gpu.clear()
    rc, _, _ = _call(gpu.lib, "bs_bicgstab_csr_noalloc", n, [a.ctypes.data for a in arrays], 0.0, 300)
    assert rc == 0   # (an empty right-hand side is solved)
    assert gpu.lib.fake_pending_error() == 0
    blocks = (n + 255) // 256
    if refused:
        assert not gpu.calls("ks_solve")
        assert len(gpu.calls("ks_init")) == 1 and len(gpu.calls("ks_true")) == 1
        assert len(gpu.calls("ks_v")) == 300 and all(g == blocks for _, g, _ in gpu.calls("ks_v"))
    else:   # two chunks of 256
        assert [g for _, g, _ in gpu.calls("ks_solve")] == [blocks] * 2 and not gpu.calls("ks_init")


@pytest.mark.gpu
@pytest.mark.parametrize("n,half,maxit", [(1, 1, 50), (256, 3, 3), (257, 5, 2000), (152 * 256 + 1, 4, 2000),
                                          (1000, 40, 2000)])
def test_phases_give_the_same_iterates(api, n, half, maxit):
    torch = pytest.importorskip("torch")
    ptr, col, val, b, _ = _system(n, half, 3 * n + half)
    dev = [torch.from_numpy(a).cuda() for a in (ptr, col, val, b)]
    got = []
    for name in ("bs_bicgstab_csr_noalloc", "bs_bicgstab_csr_noalloc_phases"):
        x = torch.zeros(n, dtype=torch.float64, device="cuda")
        rc, it, rr = _call(api.lib, name, n, [t.data_ptr() for t in dev] + [x.data_ptr()], 1e-11, maxit)
        torch.cuda.synchronize()
        got.append((rc, it, rr, x.cpu().numpy()))
    (rc0, it0, rr0, x0), (rc1, it1, rr1, x1) = got
    assert rc0 == rc1 and it0 == it1 and rr0 == rr1
    assert np.array_equal(x0, x1)
