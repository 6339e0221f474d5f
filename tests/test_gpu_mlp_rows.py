"""The training step's kernels at the row counts where their tiles, splits and
kept buffers change, against the FP32 oracle."""
import numpy as np
import pytest

from oracle import mlp

pytestmark = pytest.mark.gpu

# sums of at most 2,400 FP32 products in another order than the oracle's: a
# relative error near sqrt(2400) * 2^-24 = 3e-6 on each side
TOL = 1e-5


def test_gradients_at_tile_and_split_edges(hk):
    ctx = hk.Context()
    ctx.mlp_init(3)
    p = ctx.mlp_params()
    rng = np.random.default_rng(4)
    # (a large call first, so that the later ones run in its buffers)
    for n in (2049, 1, 15, 16, 17, 63, 64, 65, 127, 128, 255, 256, 257, 400, 1025, 2400):
        X = rng.random((n, mlp.IN), dtype=np.float32)
        y = rng.integers(0, mlp.OUT, n).astype(np.int32)
        g, loss = ctx.mlp_grad(X, y)
        og, oloss = mlp.grad_fp32(p, X, y)
        assert abs(loss - oloss) <= TOL * max(1.0, abs(oloss)), n
        o = 0
        for name, shp in mlp.SHAPES:
            k = int(np.prod(shp))
            assert np.linalg.norm(g[o:o + k] - og[o:o + k]) <= TOL * np.linalg.norm(og[o:o + k]) + 1e-12, (n, name)
            o += k
    ctx.close()
