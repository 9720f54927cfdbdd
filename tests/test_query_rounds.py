"""Batches of single queries that run as wavefront rounds: every schedule gives
the oracle's records, bit for bit, and the same as a warp per query."""
import numpy as np
import pytest

import oracle
from billardballraytracing3d_b200 import _capi as C
from billardballraytracing3d_b200 import api, scenes

pytestmark = pytest.mark.gpu

KEYS = ("object", "status", "err_object", "t", "point", "normal", "uv", "err_value")


@pytest.fixture(scope="module")
def nested(built):
    """Concentric spheres (queries with many stage-1 hits) and 9,001 rays at
    them; every fifth direction is longer than a unit, so its query is not
    culled and leaves the rounds through the overflow list."""
    patches = []
    for k, r in enumerate((1.0, 1.4, 1.9, 2.5, 3.2)):
        patches += scenes.obstacle_patches(k, (0.0, 0.0, 0.0), (r, r, r), None, m=2, n_nodes=5)
    rng = np.random.Generator(np.random.PCG64(3))
    o = rng.normal(size=(9001, 3))
    o = 6.0 * o / np.linalg.norm(o, axis=1, keepdims=True)
    d = -o + rng.normal(size=(9001, 3)) * 0.8
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    d[::5] *= 2.0
    cfg = C.default_config(coarse_grid_n=9, newton_tol=1e-12)
    return patches, cfg, o, d, oracle.Oracle(patches, config=cfg).intersect(o, d)


@pytest.mark.parametrize("graph_rounds", [1, 0])
@pytest.mark.parametrize("warp_tail", [1, 0])
@pytest.mark.parametrize("wave_tail", [0, 4096, 1000000])
def test_schedules_do_not_change_query_results(nested, graph_rounds, warp_tail, wave_tail):
    patches, cfg, o, d, ref = nested
    sc = api.Scene(patches, config=cfg)
    sc.tuning(graph_rounds=graph_rounds, warp_tail=warp_tail, wave_tail=wave_tail, wave_min_rays=1)
    got = sc.intersect(o, d)
    for k in KEYS:
        assert np.array_equal(got[k], ref[k], equal_nan=True), k


def test_workspace_does_not_grow_with_the_batch(built):
    """9M queries at two spheres: device memory taken by the call beyond its rays
    and records (152 bytes a query), and records equal to a warp per query's."""
    import ctypes
    import torch
    n = 9000001
    sc = api.Scene(scenes.scene_two_spheres(), config=C.default_config(coarse_grid_n=9, newton_tol=1e-12))
    rng = np.random.Generator(np.random.PCG64(5))
    o = rng.uniform(-3.0, 3.0, (n, 3))
    o[:, 2] = 4.0
    d = np.zeros((n, 3))
    d[:, :2] = rng.uniform(-0.3, 0.3, (n, 2))
    d[:, 2] = -0.9
    torch.cuda.init()
    sc.intersect(o[:64], d[:64])
    free = torch.cuda.mem_get_info()[0]
    got = sc.intersect(o, d)
    taken = free - torch.cuda.mem_get_info()[0]
    assert taken - 152 * n < 3.5e9, taken
    to, td = torch.from_numpy(o).cuda(), torch.from_numpy(d).cuda()
    hits = torch.zeros(n * C.HIT_DTYPE.itemsize, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    C.check(sc.lib, sc.lib.bbrt_intersect(sc.h, ctypes.c_void_p(to.data_ptr()), ctypes.c_void_p(td.data_ptr()), n,
                                          C.QUERY_BVH, 0, C.DEVICE_PTRS, ctypes.c_void_p(hits.data_ptr()), None),
            "bbrt_intersect")
    torch.cuda.synchronize()
    ref = hits.cpu().numpy().view(C.HIT_DTYPE)
    assert (ref["object"] >= 0).sum() > n // 10
    for k in KEYS:
        assert np.array_equal(got[k], ref[k], equal_nan=True), k


@pytest.mark.parametrize("graph_rounds", [1, 0])
def test_a_watchdog_set_for_traces_does_not_stop_queries(nested, graph_rounds):
    patches, cfg, o, d, ref = nested
    sc = api.Scene(patches, config=cfg)
    sc.tuning(graph_rounds=graph_rounds, wave_min_rays=1, watchdog_cycles=1)
    got = sc.intersect(o, d)
    for k in KEYS:
        assert np.array_equal(got[k], ref[k], equal_nan=True), k
    assert sc.tuning()["watchdog_cycles"] == 1
    with pytest.raises(RuntimeError, match="watchdog"):
        sc.trace(o, d, 30)
