"""Which buffers bs_download lets a kernel write: those that lie whole in a live
bs_host_alloc allocation.  Every other one takes the copies, page-locked at its
start or not: its end may not be (host logic only, no GPU)."""
import numpy as np
import pytest

from _fake_gpu import FakeGpu


@pytest.fixture
def gpu(monkeypatch, tmp_path):
    return FakeGpu(monkeypatch, tmp_path)


def _kernel(gpu, c, out, full=False):
    gpu.clear()
    c.download(0, full=full, out=out)
    return bool(gpu.calls("k_read_back"))


def _context(gpu):
    from beachslope_gb300 import scene
    p, st, gr = scene.beach_scene(dx=0.05)
    return gpu.api.Context([p], [st], [gr]), len(st["x"])


@pytest.mark.parametrize("full", [False, True])
def test_whole_allocations_take_the_kernel(gpu, full):
    c, n = _context(gpu)
    for rows in (n, n + 300, c.capacity_rows() + 7):
        assert _kernel(gpu, c, gpu.api.pinned_state(rows, full=full), full)
    # a part of an allocation, to its last byte
    out = gpu.api.pinned_state(n)
    out["vx"] = gpu.api.pinned_empty(n + 5)[5:]
    assert _kernel(gpu, c, out)


@pytest.mark.parametrize("field,dtype", [("x", np.float64), ("con", np.float64), ("pid", np.int32),
                                         ("flags", np.uint8), ("coff", np.float64), ("cell", np.int32)])
def test_registered_start_does_not_stand_for_the_end(gpu, field, dtype):
    """Page-locked by the caller's own registration: over the first rows only,
    or the first and the last with a gap between them."""
    c, n = _context(gpu)
    for both in (False, True):
        out = gpu.api.pinned_state(n, full=True)
        a = np.zeros((n, 4) if field == "coff" else n, dtype)
        out[field] = a
        part = a.nbytes // 3
        gpu.lib.fake_pin(a.ctypes.data, part)
        if both:
            gpu.lib.fake_pin(a.ctypes.data + a.nbytes - part, part)
        assert not _kernel(gpu, c, out, full=True)
        gpu.lib.fake_unpin(a.ctypes.data)
        gpu.lib.fake_unpin(a.ctypes.data + a.nbytes - part)


def test_beyond_and_after_an_allocation(gpu):
    import ctypes as C
    c, n = _context(gpu)
    p = C.c_void_p()
    assert gpu.lib.bs_host_alloc(8 * n - 1, C.byref(p)) == 0
    short = np.frombuffer((C.c_char * (8 * n)).from_address(p.value), np.float64)
    out = gpu.api.pinned_state(n)
    out["y"] = short   # its last byte lies beyond the allocation
    assert not _kernel(gpu, c, out)
    assert gpu.lib.bs_host_free(p) == 0
    gone = gpu.api.pinned_empty(n)
    out["y"] = gone
    assert _kernel(gpu, c, out)
    gpu.lib.fake_unpin(gone.ctypes.data)   # freed by the runtime's own call
    assert not _kernel(gpu, c, out)
