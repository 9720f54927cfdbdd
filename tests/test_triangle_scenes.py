"""Scenes of triangles, and scenes whose culling is asked for but not in force,
at the sizes where the route of a call changes: the oracle's results bit for
bit, and rounds that do not hand every ray to the tail."""
import ctypes

import numpy as np
import pytest

import oracle
from billardballraytracing3d_b200 import _capi as C
from billardballraytracing3d_b200 import api, scenes

pytestmark = pytest.mark.gpu

CFG = dict(coarse_grid_n=9, newton_tol=1e-12)
HIT = ("object", "status", "err_object", "t", "point", "normal", "uv", "err_value")
TRACE = ("status", "bounce_count", "hit_object", "err_object", "hit_point", "hit_uv", "end_point", "exit_dir")


def _mesh(nu, nv, center, r=1.0):
    u, v = np.linspace(0, np.pi, nu + 1), np.linspace(0, 2 * np.pi, nv + 1)
    U, V = np.meshgrid(u, v, indexing="ij")
    P = np.stack([np.sin(U) * np.cos(V), np.sin(U) * np.sin(V), np.cos(U)], -1) * r + np.array(center)
    a, b, c, d = P[:-1, :-1], P[1:, :-1], P[1:, 1:], P[:-1, 1:]
    lower, upper = np.stack([a, b, c], 2).reshape(-1, 9)[nv:], np.stack([a, c, d], 2).reshape(-1, 9)[:-nv]
    return [tuple(t) for t in np.concatenate([lower, upper])]


def _rays(n, seed, plane_z=4.0, unit=True):
    o, d = (np.ascontiguousarray(a[:n]) for a in scenes.cone_rays(n, seed, plane_z, 2.0, 25.0))
    if not unit:   # queries take directions as they are
        d[::5] *= 0.25
        d[::7] *= 3.0
    d[::11] = (0.0, 0.0, -1.0)
    if n > 13:
        o[13] = (np.nan, 0.0, 4.0)
    return o, d


def _scene(kind):
    two = scenes.scene_two_spheres()
    small = _mesh(12, 16, (0.0, 0.0, 1.4)) + _mesh(12, 16, (0.0, 0.3, -1.4))
    if kind == "triangles":
        return [], small
    if kind == "triangle":
        return [], [(-1.0, -1.0, 0.1, 1.0, -1.0, 0.0, 0.0, 1.0, 0.0)]
    return two[40:42], _mesh(40, 28, (0.0, 0.0, 1.4))   # a patch among a thousand triangles


@pytest.mark.parametrize("kind,n", [("triangle", 33), ("triangles", 1), ("triangles", 2049), ("triangles", 24575),
                                    ("triangles", 24576), ("triangles", 40001), ("few_patches", 2049),
                                    ("few_patches", 65535), ("few_patches", 65536)])
def test_queries(built, kind, n):
    import torch
    patches, tris = _scene(kind)
    sc = api.Scene(patches, triangles=tris, config=C.default_config(**CFG))
    o, d = _rays(n, 5, unit=False)
    ref = oracle.Oracle(patches, triangles=tris, config=C.default_config(**CFG)).intersect(o, d)
    assert n < 33 or (ref["object"] >= 0).sum() > 0
    to, td = torch.from_numpy(o).cuda(), torch.from_numpy(d).cuda()
    hits = torch.zeros(n * C.HIT_DTYPE.itemsize, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    C.check(sc.lib, sc.lib.bbrt_intersect(sc.h, ctypes.c_void_p(to.data_ptr()), ctypes.c_void_p(td.data_ptr()), n,
                                          C.QUERY_BVH, 0, C.DEVICE_PTRS, ctypes.c_void_p(hits.data_ptr()), None),
            "bbrt_intersect")
    torch.cuda.synchronize()
    for got in (hits.cpu().numpy().view(C.HIT_DTYPE), sc.intersect(o, d)):
        for k in HIT:
            assert np.array_equal(got[k], ref[k], equal_nan=True), k


@pytest.mark.parametrize("kind", ["triangles", "few_patches"])
@pytest.mark.parametrize("n", [700, 33001])
def test_traces(built, kind, n):
    patches, tris = _scene(kind)
    sc = api.Scene(patches, triangles=tris, config=C.default_config(**CFG))
    o, d = _rays(n, 6)
    got = sc.trace(o, d, 12, record=5)
    ref = oracle.Oracle(patches, triangles=tris, config=C.default_config(**CFG)).trace(o, d, 12, K=5)
    for k in TRACE:
        assert np.array_equal(got[k], ref[k], equal_nan=True), k
    if n > 32768:
        assert got["stats"]["rounds"] >= 1 and got["stats"]["tail_rays"] <= 4096


def test_set_with_a_member_of_triangles(built):
    import torch
    members = [([], _scene("triangles")[1]), (scenes.scene_two_spheres(), [])]
    scs = [api.Scene(p, triangles=t, config=C.default_config(**CFG)) for p, t in members]
    rays = [_rays(20001, 7), _rays(20002, 8)]
    keys = {"status": (torch.int32, ()), "bounce_count": (torch.int32, ()), "end_point": (torch.float64, (3,))}
    outs = [{k: torch.zeros((o.shape[0],) + sh, dtype=dt, device="cuda") for k, (dt, sh) in keys.items()} for o, _ in rays]
    dev = [[torch.from_numpy(a).cuda() for a in r] for r in rays]
    st, _ = api.SceneSet(scs).trace_device([r[0].data_ptr() for r in dev], [r[1].data_ptr() for r in dev],
                                           [r[0].shape[0] for r in rays], 12,
                                           [dict(record=0, **{k: t.data_ptr() for k, t in out.items()}) for out in outs])
    torch.cuda.synchronize()
    assert st["tail_rays"] <= 8192
    for (p, t), (o, d), out in zip(members, rays, outs):
        ref = oracle.Oracle(p, triangles=t, config=C.default_config(**CFG)).trace(o, d, 12, K=0)
        for k in keys:
            assert np.array_equal(out[k].cpu().numpy(), ref[k], equal_nan=True), k
