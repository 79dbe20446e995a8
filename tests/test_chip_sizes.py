"""The cluster sizes of the on-chip multigrid levels (k_mg_chip) on the scenes
of the GPU tests: one block, two, eight and sixteen, from the first level down
and from a deeper one (host logic, no GPU)."""
import pytest

from _fake_gpu import FakeGpu


@pytest.mark.parametrize("dxs,precision,wlev,level,blocks", [
    ([0.05], 1, 1, 1, 1), ([0.027], 1, 2, 1, 2), ([0.0133], 1, 1, 1, 8), ([0.0071], 1, 3, 1, 16),
    ([0.0047], 1, 0, 1, 16), ([0.0031], 1, 2, 2, 16), ([0.0133], 0, 1, 1, 8), ([0.0047], 0, 2, 2, 16),
    ([0.05, 0.011, 0.02, 0.031, 0.0083], 1, 1, 1, 16), ([0.05, 0.011, 0.0207], 0, 2, 1, 8),
    ([0.00125], 1, 2, 3, 16),
])
def test_cluster_sizes(monkeypatch, tmp_path, dxs, precision, wlev, level, blocks):
    from beachslope_gb300 import scene
    gpu = FakeGpu(monkeypatch, tmp_path)
    q = [scene.beach_scene(dx=dx, precision=precision) for dx in dxs]
    c = gpu.api.Context([v[0] for v in q], [v[1] for v in q], [v[2] for v in q], tuning="auto")
    for k, v in (("mg_sub", 0), ("mg_exact", 0), ("mg_fp32", precision), ("mg_wlev", wlev)):
        c.set_option(k, v)
    assert (c.get_option("mg_tail_level"), c.get_option("mg_tail_blocks")) == (level, blocks)
    c.set_option("mg_tail", 0)
    assert (c.get_option("mg_tail_level"), c.get_option("mg_tail_blocks")) == (0, 0)
    c.close()
