"""bs_download into page-locked buffers (one kernel over the host link) against
the copies into pageable ones: every field of full and plain read-backs, for
buffers of exactly the scene's rows, larger ones, an unaligned one (which takes
the copies), an empty scene; buffers too small are refused and left alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ctx(api, n_scenes=2):
    from beachslope_gb300 import scene
    q = [scene.beach_scene(dx=dx) for dx in (0.05, 0.031)[:n_scenes]]
    c = api.Context([v[0] for v in q], [v[1] for v in q], [v[2] for v in q])
    c.prime()
    return c


@pytest.mark.parametrize("full", [False, True])
@pytest.mark.parametrize("extra", [0, 1, 300])
def test_pinned_read_back_equals_copies(api, full, extra):
    c = _ctx(api)
    for s in range(2):
        ref = c.download(s, full=full)
        n = len(ref["x"])
        out = api.pinned_state(n + extra, full=full)
        got = c.download(s, full=full, out=out)
        assert sorted(got) == sorted(ref)
        for k in ref:
            assert got[k].shape == ref[k].shape and np.array_equal(got[k], ref[k]), k
    c.close()


def test_unaligned_and_small_buffers(api):
    from beachslope_gb300 import abi
    c = _ctx(api, 1)
    ref = c.download(0, full=False)
    n = len(ref["x"])
    out = api.pinned_state(n)
    raw = api.pinned_empty(8 * n + 8, np.uint8)
    out["vx"] = raw[4:4 + 8 * n].view(np.float64)   # not on an 8-byte boundary: the copies
    got = c.download(0, full=False, out=out)
    for k in ref:
        assert np.array_equal(got[k], ref[k]), k
    small = api.pinned_state(n - 1)
    for v in small.values():
        v[...] = 7
    with pytest.raises(ValueError):
        c.download(0, full=False, out=small)
    assert all(np.all(v == 7) for v in small.values())
    c.close()
    p, st, gr = __import__("beachslope_gb300.scene", fromlist=["x"]).beach_scene(dx=0.05)
    c = api.Context([p], [abi.empty_state()], [None], capacity=[1000])
    assert len(c.download(0, full=False, out=api.pinned_state(256))["x"]) == 0
    c.close()
