"""Split search of small nodes on the GPU against the oracle at the sizes
where its groups, passes and lanes change, with references that lie flat on
candidate planes, repeated bounds, and triangles that span the whole scene."""
import numpy as np
import pytest

from hulktracer_b200 import scenes

pytestmark = pytest.mark.gpu


def mixed_scene(n, seed):
    """n triangles on a coarse lattice (equal bounds, axis-aligned flat ones,
    planes that coincide with bin planes), a few of them very large."""
    rng = np.random.default_rng(seed)
    p = rng.integers(-8, 9, size=(n, 1, 3)).astype(np.float64)
    e = rng.integers(-2, 3, size=(n, 2, 3)).astype(np.float64)
    v = np.concatenate([p, p + e], axis=1)
    flat = rng.random(n) < 0.3
    ax = rng.integers(0, 3, n)
    for i in np.nonzero(flat)[0]:
        v[i, :, ax[i]] = v[i, 0, ax[i]]
    loose = rng.random(n) < 0.3
    v[loose] += rng.normal(size=(int(loose.sum()), 3, 3))
    big = rng.random(n) < 0.05
    v[big] *= 3.0
    V = np.ones((3 * n, 4), np.float32)
    V[:, :3] = v.reshape(-1, 3)
    V[:, :3][V[:, :3] == 0.0] *= -1.0     # -0 as well
    T = np.zeros((n, 4), np.uint32)
    T[:, :3] = np.arange(3 * n).reshape(n, 3)
    return V, T


@pytest.mark.parametrize("subtree_max,subtree_depth,leaf_size", [(32, 0, 4), (32, 0, 1), (0, 0, 0), (16, 8, 2)])
@pytest.mark.parametrize("exact_max", [0, 32, 1024])
def test_small_nodes_identical_to_oracle(hk, oracle, exact_max, subtree_max, subtree_depth, leaf_size):
    ctx = hk.Context(exact_max=exact_max, subtree_max=subtree_max, subtree_depth=subtree_depth, leaf_size=leaf_size)
    for n in (1, 2, 3, 4, 5, 8, 9, 15, 16, 17, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 1023, 1024, 1025,
              2500):
        V, T = mixed_scene(n, n)
        box = scenes.scene_box(V)
        ctx.upload(V, T)
        ctx.set_box(box)
        ctx.precompute()
        ctx.build()
        cn, cr = ctx.export_compact()
        on, orf = oracle.build_binned(V, T, box, leaf_size=leaf_size, exact_max=exact_max, defer=subtree_max,
                                      defer_margin=subtree_depth)
        assert np.array_equal(cn, on) and np.array_equal(cr, orf), n
    ctx.close()


@pytest.mark.parametrize("topk", [1, 2, 3, 5, 6, 8])
def test_learned_nodes_identical_to_oracle(hk, oracle, topk):
    """Learned builds (untrained network) around the sizes where a proposer row
    changes kernel, replayed by the oracle from the logged proposals."""
    ctx = hk.Context(topk=topk, subtree_depth=0)
    ctx.mlp_init(topk)
    ctx.set_proposal_log(True)
    for n in (33, 64, 127, 128, 129, 255, 256, 257, 700, 1023, 1024, 1025, 2500):
        V, T = mixed_scene(n, 1000 * topk + n)
        box = scenes.scene_box(V)
        ctx.upload(V, T)
        ctx.set_box(box)
        ctx.precompute()
        ctx.build(hk.BUILD_LEARNED)
        cn, cr = ctx.export_compact()
        on, orf = oracle.build_binned(V, T, box, proposals=ctx.proposal_log(), topk=topk, fallback_ratio=1.0, defer=32,
                                      defer_margin=0)
        assert np.array_equal(cn, on) and np.array_equal(cr, orf), n
    ctx.close()
