"""Batches in the variants and the counting mode whose leaf tests are shared
by the warp or kept in order: every scene's hits equal the single-scene trace,
and the batch's counters are the sum of the single traces'."""
import numpy as np
import pytest

from hulktracer_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant", ["restart", "restart_early", "smemstack", "fullstack", "shortstack", "ropes", "brute"])
@pytest.mark.parametrize("counting", [False, True], ids=["plain", "counting"])
def test_batch_equals_per_scene(hk, variant, counting):
    import torch
    v = hk.VARIANTS[variant]
    tris, rays_per = ((40, 300), (1, 500)) if variant == "brute" else ((40, 9_000), (1, 7_000))
    sets = scenes.batch_scenes(n_scenes=3, seed=21, tris=tris, rays=rays_per)
    ctx, single = hk.Context(), hk.Context()
    ctx.set_counting(counting)
    single.set_counting(counting)
    batch = hk.engine.Batch(ctx)
    rays, offsets, expected, counts = [], [0], [], np.zeros(3, np.uint64)
    for i, (sc, nr) in enumerate(sets):
        batch.add_scene(sc.verts, sc.tris)
        rays.append(scenes.incoherent_rays(sc, nr, seed=50 + i))
        offsets.append(offsets[-1] + nr)
        single.upload(sc.verts, sc.tris)
        single.precompute()
        single.build()
        expected.append(single.trace(rays[-1], v))
        if counting:
            counts += single.counters()
    d_rays = torch.from_numpy(np.concatenate(rays)).cuda()
    d_hits = torch.zeros(2 * offsets[-1], dtype=torch.int32, device="cuda")
    batch.trace_device(d_rays.data_ptr(), offsets, d_hits.data_ptr(), v)
    torch.cuda.synchronize()
    hits = d_hits.cpu().numpy().view(hk._lib.HIT_DTYPE)
    for i, e in enumerate(expected):
        h = hits[offsets[i]:offsets[i + 1]]
        assert np.array_equal(h["tri"], e["tri"])
        assert np.array_equal(h["t"], e["t"])
    if counting:
        assert np.array_equal(ctx.counters(), counts)
    batch.close()
    ctx.close()
    single.close()
