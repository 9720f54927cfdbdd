"""Patches and triangles mixed, over leaf sizes and coarse grids where a leaf's
object boxes, a patch's blocks and a block's cells end unevenly: the wavefront,
the small-batch kernel and single queries against the oracle, bit for bit.

No tolerance: every path computes the oracle's doubles."""
import numpy as np
import pytest

import oracle
from billardballraytracing3d_b200 import _capi as C
from billardballraytracing3d_b200 import api, scenes

pytestmark = pytest.mark.gpu


def _rays(n, seed):
    """Cone rays at the spheres, a few of them axis-parallel, zero or inside."""
    o, d = scenes.cone_rays(n, seed, 4.0, 3.0, 25.0)
    d[0::97] = (0.0, 0.0, -1.0)
    d[5] = 0.0
    o[7] = (1.5, 0.1, 0.2)
    o[11] = (np.nan, 0.0, 4.0)
    return o, d


@pytest.mark.parametrize("leaf,coarse_n", [(1, 17), (4, 9), (4, 18), (5, 6), (33, 17), (70, 23), (4, 100)])
def test_mixed_leaves_match_oracle(built, leaf, coarse_n):
    patches = scenes.scene_two_spheres()
    tris = [(-0.4, -0.5 + 0.2 * k, 1.0 + 0.1 * k, 0.4, -0.5 + 0.2 * k, 1.2, 0.0, -0.2 + 0.2 * k, 0.9 + 0.1 * k)
            for k in range(7)]
    cfg = C.default_config(coarse_grid_n=coarse_n, newton_tol=1e-12, leaf_threshold=leaf)
    sc = api.Scene(patches, triangles=tris, config=cfg)
    orc = oracle.Oracle(patches, triangles=tris, config=cfg)
    o, d = _rays(9001, 5)
    r = orc.trace(o, d, 12, K=5)
    for n in (9001, 700, 33, 1):
        for stats in (True, False):
            g = sc.trace(o[:n], d[:n], 12, record=5, want_stats=stats)
            for k in ("status", "bounce_count", "hit_object", "err_object", "hit_point", "hit_uv", "end_point",
                      "exit_dir"):
                assert np.array_equal(g[k], r[k][:n], equal_nan=True), (k, n, stats)
    d[5] = (0.1, 0.2, -1.0)
    for mode, sizes in ((C.QUERY_BVH, (2001, 650, 1)), (C.QUERY_BRUTE, (40,))):
        for n in sizes:
            a, b = sc.intersect(o[:n], d[:n], mode=mode), orc.intersect(o[:n], d[:n], mode=mode)
            for k in ("object", "status", "err_object", "t", "point", "normal", "uv"):
                assert np.array_equal(a[k], b[k], equal_nan=True), (k, n, mode)
