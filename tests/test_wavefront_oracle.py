"""The wavefront's rounds against the oracle, bit for bit, in scenes that reach
their less common parts: triangles among patches, leaves of many slots (k_advance
instead of split rounds), grids beyond a quadtree's 16 x 16 cells, rays that
meet more leaves or have more stage-1 hits than their lists hold.

Every call states its schedule, so that it runs rounds whatever the default
threshold is, and the statistics are asked whether it did.  No tolerance: every
path computes the oracle's doubles."""
import os
import subprocess
import sys

import numpy as np
import pytest

import oracle
from billardballraytracing3d_b200 import _capi as C
from billardballraytracing3d_b200 import api, scenes
from conftest import ROOT

pytestmark = pytest.mark.gpu

KEYS = ("status", "bounce_count", "hit_object", "err_object", "hit_point", "hit_uv", "end_point", "exit_dir")
SCHEDULES = [dict(graph_rounds=1, wave_tail=0), dict(graph_rounds=1, wave_tail=4096), dict(graph_rounds=0, wave_tail=0),
             dict(graph_rounds=0, wave_tail=512, warp_tail=0)]


def _check(patches, tris, cfg, o, d, maxb, overflow):
    ref = oracle.Oracle(patches, triangles=tris, config=cfg).trace(o, d, maxb, K=5)
    sc = api.Scene(patches, triangles=tris, config=cfg)
    for tune in SCHEDULES:
        sc.tuning(wave_min_rays=1, **tune)
        for stats in (True, False):   # with and without counters
            got = sc.trace(o, d, maxb, record=5, want_stats=stats)
            for k in KEYS:
                assert np.array_equal(got[k], ref[k], equal_nan=True), (tune, stats, k)
            if stats:
                assert got["stats"]["rounds"] >= 1
                if tune["wave_tail"] == 0:   # then only overflowed rays are finished by the tail
                    assert overflow[0] <= got["stats"]["tail_rays"] <= overflow[1], got["stats"]["tail_rays"]


def _cone(n, seed):
    """Cone rays at the two spheres, a few of them axis-parallel, zero or inside."""
    o, d = (np.ascontiguousarray(a[:n]) for a in scenes.cone_rays(n, seed, 4.0, 3.0, 25.0))
    d[0::97] = (0.0, 0.0, -1.0)
    d[5] = 0.0
    o[7] = (1.5, 0.1, 0.2)
    return o, d


# leaves of 1, 4, 5 and 33 slots; 5, 8, 16, 17 and 99 cells a side
@pytest.mark.parametrize("leaf,coarse_n", [(1, 17), (4, 9), (4, 18), (5, 6), (33, 17), (4, 100)])
def test_mixed_scene(built, leaf, coarse_n):
    tris = [(-0.4, -0.5 + 0.2 * k, 1.0 + 0.1 * k, 0.4, -0.5 + 0.2 * k, 1.2, 0.0, -0.2 + 0.2 * k, 0.9 + 0.1 * k)
            for k in range(7)]
    cfg = C.default_config(coarse_grid_n=coarse_n, newton_tol=1e-12, leaf_threshold=leaf)
    # (k_advance, for leaves of more than four slots, overflows on no ray here)
    _check(scenes.scene_two_spheres(), tris, cfg, *_cone(5001, 5), 12, overflow=(0, 0))


@pytest.mark.parametrize("coarse_n", [9, 18])
def test_many_hits_a_query(built, coarse_n):
    """Concentric spheres: up to ten surfaces on a ray."""
    patches = []
    for k, r in enumerate((1.0, 1.4, 1.9, 2.5, 3.2)):
        patches += scenes.obstacle_patches(k, (0.0, 0.0, 0.0), (r, r, r), None, m=2, n_nodes=5)
    rng = np.random.Generator(np.random.PCG64(11))
    o = rng.normal(size=(20000, 3))
    o = 6.0 * o / np.linalg.norm(o, axis=1, keepdims=True)
    d = -o + rng.normal(size=(20000, 3)) * 0.8
    _check(patches, [], C.default_config(coarse_grid_n=coarse_n, newton_tol=1e-12), o, d, 30, overflow=(1, 20000))


@pytest.mark.parametrize("layers", [8, 9, 32, 33, 40])
def test_many_leaves_a_query(built, layers):
    """Triangles one behind the other beside the spheres, one to a leaf: 1,501 of
    3,001 rays meet `layers` leaves and hit every one of them (up to eight fit a
    ray's list), the others are cone rays."""
    tris = [(-0.3, -0.3, 1.5 - 0.05 * k, 0.3, -0.3, 1.5 - 0.05 * k, 0.0, 0.4, 1.5 - 0.05 * k) for k in range(layers)]
    cfg = C.default_config(coarse_grid_n=9, newton_tol=1e-12, leaf_threshold=1)
    o, d = _cone(3001, 9)
    o[::2] = np.column_stack([np.linspace(-0.05, 0.05, o[::2].shape[0])] * 2 + [np.full(o[::2].shape[0], 4.0)])
    d[::2] = (0.0, 0.0, -1.0)
    _check(scenes.scene_two_spheres(), tris, cfg, o, d, 12, overflow=(0, 1500) if layers <= 8 else (1501, 3001))


ADVANCE_SCRIPT = r'''
import sys, numpy as np
sys.path.insert(0, sys.argv[1])
from billardballraytracing3d_b200 import scenes, api, _capi as C
patches, o, d, maxb, cn, tol = scenes.workload("tetra_spheres", 10000)
sc = api.Scene(patches, config=C.default_config(coarse_grid_n=cn, newton_tol=tol, leaf_threshold=int(sys.argv[3])))
out = {}
for shape in range(7):
    sc.tuning(wave_min_rays=1, wave_tail=64, advance_shape=shape)
    t = sc.trace(o, d, maxb, record=4)
    assert t["stats"]["rounds"] >= 2
    out.update({f"{shape}_{k}": t[k] for k in ("status", "bounce_count", "hit_object", "hit_point", "end_point", "exit_dir")})
np.savez(sys.argv[2], **out)
'''


# leaves of eight slots, or no FP32 node tests: k_advance runs the rounds
@pytest.mark.parametrize("leaf,env", [(8, {}), (8, {"BBRT_RESUME": "0"}), (8, {"BBRT_ADAPT_LANES": "0"}),
                                      (8, {"BBRT_GRAPH": "0"}), (4, {"BBRT_NODE_F32": "0"}),
                                      (4, {"BBRT_NODE_F32": "0", "BBRT_RESUME": "0", "BBRT_GRAPH": "0"})])
def test_every_k_advance_shape(built, workloads, tmp_path, leaf, env):
    out = tmp_path / "r.npz"
    subprocess.run([sys.executable, "-c", ADVANCE_SCRIPT, ROOT, str(out), str(leaf)], check=True, env={**os.environ, **env})
    g = np.load(out)
    patches, o, d, maxb, cn, tol = workloads("tetra_spheres", 10000)
    r = oracle.Oracle(patches, config=C.default_config(coarse_grid_n=cn, newton_tol=tol, leaf_threshold=leaf)).trace(
        o, d, maxb, K=4)
    for k in g.files:
        assert np.array_equal(g[k], r[k.split("_", 1)[1]]), (env, k)
