"""The block size of the neighbour sweeps (option sweep_tpb): the size asked for
is the size that runs, on small scenes too; a context that was not told takes
blocks of 256, smaller ones where a scene has too few rows for two on each SM
(host logic, no GPU)."""
import pytest

from _fake_gpu import FakeGpu


def _context(gpu, rows):
    from beachslope_gb300 import scene
    p, st, gr = scene.beach_scene(dx=0.05)
    return gpu.api.Context([p], [st], [gr], capacity=[rows])


def _blocks(gpu, c):
    gpu.clear()
    c.eddy()
    c.porosity()
    got = {b for name in ("k_eddy", "k_search") for _, _, b in gpu.calls(name)}
    assert len(got) == 1
    return got.pop()


@pytest.mark.parametrize("rows", [1000, 20000, 200000])
@pytest.mark.parametrize("tpb", [64, 128, 256])
def test_the_size_asked_for_runs(monkeypatch, tmp_path, rows, tpb):
    gpu = FakeGpu(monkeypatch, tmp_path)
    c = _context(gpu, rows)
    c.set_option("sweep_tpb", tpb)
    assert c.get_option("sweep_tpb") == tpb and c.get_option("sweep_tpb_used") == tpb
    assert _blocks(gpu, c) == tpb


@pytest.mark.parametrize("rows,want", [(1000, 32), (13681, 32), (20000, 64), (39000, 128), (78000, 256),
                                       (200000, 256)])   # two blocks on each of 152 SMs
def test_the_default_fills_the_device(monkeypatch, tmp_path, rows, want):
    gpu = FakeGpu(monkeypatch, tmp_path)
    c = _context(gpu, rows)
    assert c.get_option("sweep_tpb") == 256 and c.get_option("sweep_tpb_used") == want
    assert _blocks(gpu, c) == want
