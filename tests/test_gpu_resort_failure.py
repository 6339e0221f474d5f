"""Failures of HK_BUILD_SAH_RESORT that stay on the host's side of a GPU fault.

Its single-pass scans wait (bounded) for earlier tiles. A test aid
(hk_set_debug_flags) makes a scan's first tile withhold its flag: the waits run
out, every later kernel of the build returns on the error word before it
indexes with a scan's result, and hk_build returns HK_E_DEVICE_TIMEOUT. The
failed output is no tree, and the next build on the context equals a build of
another context array for array."""
import numpy as np
import pytest

from hulktracer_b200 import scenes

pytestmark = pytest.mark.gpu

HK_E_DEVICE_TIMEOUT, HK_E_STATE = 17, 20


def built(c, hk):
    c.build(hk.BUILD_SAH_RESORT)
    return c.export_compact()


@pytest.mark.parametrize("tris, ci, leaf", [
    (20000, 1.5, 4),   # level 1's first radix pass: its digit counts' scan
    (3000, 20.0, 1),   # level 1 sorts without it: the first level of more than 1,024 nodes
])
def test_scan_wait_runs_out_and_context_recovers(hk, tris, ci, leaf):
    sc = scenes.random_soup(tris, seed=6)
    cfg = dict(traverse_cost=1.0, intersect_cost=ci, max_depth=24, leaf_size=leaf, sah_sample=1)
    fresh = hk.Context(**cfg)
    fresh.upload(sc.verts, sc.tris)
    good_n, good_r = built(fresh, hk)
    fresh.close()
    c = hk.Context(spin_limit=2000, **cfg)
    c.upload(sc.verts, sc.tris)
    c.precompute()
    c.set_debug_flags(1)
    rays = np.zeros((4, 8), np.float32)
    rays[:, 4] = 1.0
    for _ in range(2):
        with pytest.raises(hk.HkError) as e:
            c.build(hk.BUILD_SAH_RESORT)
        assert e.value.status == HK_E_DEVICE_TIMEOUT
        with pytest.raises(hk.HkError) as e:
            c.trace(rays, hk.SHORTSTACK)
        assert e.value.status == HK_E_STATE
    c.set_debug_flags(0)
    for _ in range(2):
        n, r = built(c, hk)
        assert np.array_equal(n, good_n) and np.array_equal(r, good_r)
    c.close()
