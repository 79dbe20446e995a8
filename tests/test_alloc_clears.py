"""Device memory that a living context allocates is cleared on the null stream,
for which the context's own (non-blocking) stream does not wait: nothing may be
launched before the clearing has ended (host logic, no GPU)."""
import pytest

from _fake_gpu import FakeGpu


@pytest.mark.parametrize("options", [
    [],
    [("ppe_solver", 1)],                            # the FGMRES basis and its counters
    [("ppe_solver", 1), ("ppe_restart", 40)],
    [("mg_fp32", 1)],                               # the FP32 matrix
    [("mg_exact", 1)],                              # the exact level's inverse
    [("mg_exact", 1), ("mg_exact", 0)],
    [("mg_sub", 1), ("mg_sub", 0)],
])
def test_no_launch_before_the_clearing_ends(monkeypatch, tmp_path, options):
    from beachslope_gb300 import scene
    gpu = FakeGpu(monkeypatch, tmp_path)
    p, st, gr = scene.beach_scene(dx=0.03)
    c = gpu.api.Context([p], [st], [gr])
    for k, v in options:
        c.set_option(k, v)
        c.eddy()
    c.download_async(0, out=gpu.api.pinned_state(c.capacity_rows()))   # (allocates the snapshot)
    c.eddy()
    c.close()
    assert gpu.lib.fake_early_launches() == 0


def test_new_image_of_the_chip_levels(monkeypatch, tmp_path):
    """A scene that needs more constants than the one before it in its slot."""
    from beachslope_gb300 import scene
    gpu = FakeGpu(monkeypatch, tmp_path)
    big, small = scene.beach_scene(dx=0.0133), scene.beach_scene(dx=0.05)
    c = gpu.api.Context([big[0]], [big[1]], [big[2]])
    c.set_option("mg_tail", 0)
    c.set_scene(0, *small)
    c.set_option("mg_tail", 1)
    c.set_scene(0, *big)
    c.eddy()
    c.close()
    assert gpu.lib.fake_early_launches() == 0
