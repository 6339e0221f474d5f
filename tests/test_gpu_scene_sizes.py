"""Triangle, vertex, pixel and light counts around the sizes where a launch
changes its grid, its block or its list layout, against the oracle."""
import numpy as np
import pytest

from hulktracer_b200 import scenes
from oracle.oracle import NORM_IEEE, SHORTSTACK as O_SHORT

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("exact_max", [0, 64])
@pytest.mark.parametrize("n", [1, 255, 4735, 4736, 4737, 9473, 37_889, 131_072, 131_073])
def test_trees_identical_to_oracle(hk, oracle, n, exact_max):
    sc = scenes.cluster_soup(n, seed=n)
    box = scenes.scene_box(sc.verts)
    ctx = hk.Context(exact_max=exact_max)
    ctx.upload(sc.verts, sc.tris)
    ctx.set_box(box)
    ctx.precompute()
    on, orf = oracle.build_binned(sc.verts, sc.tris, box, exact_max=exact_max)
    for _ in range(2):      # a build leaves its counters ready for the next
        ctx.build()
        cn, cr = ctx.export_compact()
        assert np.array_equal(cn, on) and np.array_equal(cr, orf)
    ctx.close()


@pytest.mark.parametrize("n", [1, 85, 86, 50_517, 50_518, 60_000])
def test_transform_box(hk, oracle, n):
    """Vertices around one CTA and around the transform's largest grid."""
    rng = np.random.default_rng(n)
    V = np.ones((3 * n, 4), np.float32)
    V[:, :3] = rng.normal(size=(3 * n, 3))
    T = np.zeros((n, 4), np.uint32)
    T[:, :3] = np.arange(3 * n).reshape(n, 3)
    part = rng.integers(0, 5, 3 * n).astype(np.uint32)
    ctx = hk.Context()
    ctx.upload(V, T)
    ctx.set_parts(part, 5)
    for _ in range(3):      # a smaller box follows a larger one
        mats = (rng.normal(size=(5, 12)) * rng.choice([0.01, 1.0, 100.0])).astype(np.float32)
        ctx.transform(mats)
        o = oracle.transform(V, part, mats)
        ob = oracle.scene_box(o)
        box = ctx.get_box()
        assert np.array_equal(ctx.get_vertices().view(np.uint32), o.view(np.uint32))
        assert np.array_equal(box[:3], ob[:3]) and np.array_equal(box[4:7], ob[4:7])
    ctx.close()


@pytest.mark.parametrize("w,h", [(1, 1), (7, 5), (32, 8), (257, 3), (104, 76)])
@pytest.mark.parametrize("kinds", ["p", "d", "pdp", "dppd", "ppppppp", ""])
def test_shadow_lists(hk, oracle, w, h, kinds):
    """Mixes of point (p) and directional (d) lights at pixel counts around a CTA."""
    sc = scenes.cluster_soup(3000, seed=11)
    rng = np.random.default_rng(len(kinds) + w)
    lights = np.zeros((len(kinds), 8), np.float32)
    for i, k in enumerate(kinds):
        lights[i, :3] = rng.uniform(0.1, 0.4, 3)
        lights[i, 3] = 1.0 if k == "p" else 0.0
        p = rng.normal(size=3)
        lights[i, 4:7] = 80.0 * p if k == "p" else p / np.linalg.norm(p)
    box = scenes.scene_box(sc.verts)
    ctx = hk.Context(short_stack=6)
    ctx.upload(sc.verts, sc.tris)
    ctx.set_box(box)
    ctx.precompute()
    ctx.build()
    cn, cr = oracle.build_binned(sc.verts, sc.tris, box)
    tree = oracle.make_tree(sc.verts, sc.tris, oracle.cache(sc.verts, sc.tris, NORM_IEEE), oracle.compact_to_ref(cn),
                            cr, box)
    rays = oracle.camera_rays(sc.camera, w, h, NORM_IEEE)
    oimg = oracle.render_cpu(tree, rays, w, h, lights, O_SHORT, 6, NORM_IEEE)
    for _ in range(2):      # a frame leaves nothing for the next
        assert np.array_equal(ctx.render(sc.camera, lights, w, h, hk.SHORTSTACK), oimg)
    hits = ctx.trace(rays, hk.SHORTSTACK)
    assert ctx.ray_counts() == (w * h, int((hits["tri"] >= 0).sum()) * kinds.count("p"))
    ctx.close()


@pytest.mark.parametrize("scale", [1.0, 2.0 ** -40, 2.0 ** 40])
@pytest.mark.parametrize("ct,ci", [(1.0, 1.5), (0.0, 1.0), (500.0, 1.5), (1.0, 1e-3), (0.0, 1e-30), (1.0, 1e30)])
@pytest.mark.parametrize("lattice", [False, True])
def test_costs_identical_to_oracle(hk, oracle, lattice, ct, ci, scale):
    """Costs dominated by either term, and scenes of unusual size, with many
    equal costs (lattice) or few."""
    sc = scenes.cluster_soup(4000, seed=21)
    V = sc.verts.copy()
    if lattice:
        V[:, :3] = np.round(V[:, :3] * 0.25)
    V[:, :3] *= np.float32(scale)
    box = scenes.scene_box(V)
    ctx = hk.Context(traverse_cost=ct, intersect_cost=ci, leaf_size=1, subtree_depth=0)
    ctx.upload(V, sc.tris)
    ctx.set_box(box)
    ctx.precompute()
    ctx.build()
    cn, cr = ctx.export_compact()
    on, orf = oracle.build_binned(V, sc.tris, box, ct=ct, ci=ci, leaf_size=1, defer_margin=0)
    assert np.array_equal(cn, on) and np.array_equal(cr, orf)
    ctx.close()
