"""HK_BUILD_SAH_RESORT at the sizes where its launches change: a root of 128 /
129 polygons (a segment's sort by a warp or a CTA), 1,023 to 1,025 (one or two
scan tiles) and 2,048 / 2,049 (CTA or radix sort), the latter also as sampled
polygons; builds of large, small and large scenes on one context, each twice, so
that the scans' flags and workspaces of earlier builds lie there. Every tree
equals the oracle's."""
import numpy as np
import pytest

from hulktracer_b200 import scenes
from test_gpu_resort import compare_compact

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sample, sizes", [
    (1, [2049, 128, 1025, 1, 2048, 129, 1024, 1023, 8192]),
    (5, [10245, 640, 641, 10240, 4, 10241]),
], ids=["every", "fifth"])
def test_sizes_on_one_context(hk, oracle, sample, sizes):
    c = hk.Context(traverse_cost=1.0, intersect_cost=1.5, max_depth=24, leaf_size=4, sah_sample=sample)
    for k, tris in enumerate(sizes):
        sc = scenes.random_soup(tris, seed=30 + k)
        v = sc.verts.astype(np.float32)
        c.upload(v, sc.tris)
        rn, rr = oracle.build_sah_resort(v, sc.tris, c.get_box(), ct=1.0, ci=1.5, max_depth=24, leaf_below=5,
                                         reduction=sample)
        want = oracle.ref_to_compact(rn)
        for _ in range(2):
            c.build(hk.BUILD_SAH_RESORT)
            cn, cr = c.export_compact()
            compare_compact(cn, cr, want, rr)
    c.close()
