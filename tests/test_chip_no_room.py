"""No device memory left for the on-chip multigrid levels' constants: the
context is made all the same and takes the separate launches, and no CUDA error
is left behind for the next call to report (host logic, no GPU)."""
import ctypes as C

from _fake_gpu import FakeGpu


def test_no_room_for_the_chip_image(monkeypatch, tmp_path):
    from beachslope_gb300 import scene
    gpu = FakeGpu(monkeypatch, tmp_path)
    p, st, gr = scene.beach_scene(dx=0.0133)
    c = gpu.api.Context([p], [st], [gr])
    assert c.get_option("mg_tail_level") == 1
    total = C.c_size_t()
    assert gpu.lib.bs_context_bytes(c.h, C.byref(total)) == 0
    c.close()
    gpu.lib.fake_room(total.value * 59 // 60)   # all but a part of the constants
    c = gpu.api.Context([p], [st], [gr])
    assert c.get_option("mg_tail_level") == 0
    assert gpu.lib.fake_pending_error() == 0
    c.search()   # (its launch check would report one)
    gpu.lib.fake_room(1 << 30)
    c.set_option("mg_tail", 1)   # room again
    assert c.get_option("mg_tail_level") == 1
    c.close()


def test_the_image_takes_no_room_that_the_context_needs(monkeypatch, tmp_path):
    """With just the memory that a context needs without the constants, and with
    anything up to what it takes with them, it is made."""
    from beachslope_gb300 import scene
    gpu = FakeGpu(monkeypatch, tmp_path)
    p, st, gr = scene.beach_scene(dx=0.0133)

    def made(room):
        gpu.lib.fake_room(room)
        c = gpu.api.Context([p], [st], [gr])
        n = C.c_size_t()
        assert gpu.lib.bs_context_bytes(c.h, C.byref(n)) == 0
        level = c.get_option("mg_tail_level")
        c.close()
        return n.value, level

    total, level = made(1 << 30)
    assert level == 1
    bare, level = made(total * 59 // 60)
    assert level == 0 and bare < total
    for room in (bare, bare + 1, (bare + total) // 2, total - 1):
        assert made(room) == (bare, 0)
    assert made(total) == (total, 1)


def test_no_constants_without_the_preconditioner(monkeypatch, tmp_path):
    """Solves that run no multigrid cycle (the reference's settings, the CSR
    calls) do not allocate its constants; switching it on does."""
    from beachslope_gb300 import scene
    gpu = FakeGpu(monkeypatch, tmp_path)
    p, st, gr = scene.beach_scene(dx=0.0133)
    p.ppe_precond = 0
    c = gpu.api.Context([p], [st], [gr])
    n = [C.c_size_t(), C.c_size_t()]
    assert gpu.lib.bs_context_bytes(c.h, C.byref(n[0])) == 0
    assert c.get_option("mg_tail_level") == 0
    c.set_option("ppe_precond", 1)
    assert gpu.lib.bs_context_bytes(c.h, C.byref(n[1])) == 0
    assert c.get_option("mg_tail_level") == 1 and n[1].value > n[0].value
    c.close()
