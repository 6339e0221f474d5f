"""A ray's hit does not depend on how many rays are traced with it: the counts
around a warp, and around one ray, a few rays and a full load per lane of the
persistent grid, at several block sizes and grids."""
import numpy as np
import pytest

from hulktracer_b200 import scenes

pytestmark = pytest.mark.gpu

VARIANTS = ["ropes", "shortstack", "smemstack", "fullstack", "restart", "restart_early"]


@pytest.fixture(scope="module")
def case():
    sc = scenes.cluster_soup(20_000, seed=5)
    rays = scenes.incoherent_rays(sc, 260_000, seed=6)
    rays[::97, 4:7] *= np.float32(-1.0)     # away from the scene as well
    return sc, rays


@pytest.mark.parametrize("block,per_sm", [(128, 0), (32, 0), (256, 0), (64, 1)])
@pytest.mark.parametrize("variant", VARIANTS)
def test_hits_independent_of_the_ray_count(hk, case, variant, block, per_sm):
    sc, rays = case
    ctx = hk.Context(block_size=block, blocks_per_sm=per_sm)
    ctx.upload(sc.verts, sc.tris)
    ctx.precompute()
    ctx.build()
    v = hk.VARIANTS[variant]
    ref = ctx.trace(rays, v)
    brute = ctx.trace(rays[:2000], hk.BRUTE)
    m = brute["tri"] >= 0
    assert np.array_equal(ref["tri"][:2000] >= 0, m) and np.array_equal(ref["t"][:2000][m], brute["t"][m])
    for n in (1, 2, 31, 32, 33, 63, 997, 5919, 5920, 5921, 14_601, 47_360, 189_440, 189_441):
        hits = ctx.trace(rays[:n], v)
        assert np.array_equal(hits["tri"], ref["tri"][:n]) and np.array_equal(hits["t"], ref["t"][:n]), n
    ctx.close()
