"""The work this framework is measured by: the calls its users make, over the sizes they make them at.

Scenes are the named workloads of billardballraytracing3d_b200.scenes (two spheres, the sphere
tetrahedron, sixteen ellipsoids) and seeded scenes of the multi-scene kind; rays are seeded anew for
every state.  A state holds what a program keeps between calls: the compiled and uploaded scene (its
geometry does not depend on the seed), the rays, and for device calls the output arrays.

  query    Scene.intersect: one BVH query per ray, host arrays
  paths    Scene.trace: whole ray paths with their recorded hits, host arrays
  device   Scene.trace_device: rays and results in device memory (a solver that stays on the GPU)
  plane    Scene.plane_source: a grid of parallel rays, hit counts per object
  bounce   Scene.bounce_map: launch points on patches times a cone of directions
  set      SceneSet.trace_device: several scenes in one trace
  train    Scene.guess_train: the learned Newton start's samples, forward and backward passes and
           optimiser steps

The learned start's own traces are left out: which bounces take it depends on the launch schedule, so
its whole-number outputs are not a function of its inputs.  Training runs one batch per epoch, which
holds every sample, so that the order in which samples are recorded does not matter.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from billardballraytracing3d_b200 import _capi as C
from billardballraytracing3d_b200 import api, scenes

# coarse_n / tol: the workloads' own constants; "reference" ones are the library's defaults (100, 1e-3)
_SCENES = {
    # name: (z of the source plane, its half extent, cone half angle, default max bounces, coarse n)
    "two_spheres": (4.0, 3.0, 17.0, 20, 9),
    "tetra": (5.0, 3.0, 10.0, 200, 17),
    "ellipsoids": (8.0, 6.0, 20.0, 100, 17),
}


def listed():
    return [
        # a handful of line-of-sight checks: launch and copy latency
        {"name": "query_small", "kind": "query", "scene": "two_spheres", "n": 96, "reference": False},
        # a visibility map
        {"name": "query_large", "kind": "query", "scene": "tetra", "n": 200003, "reference": False},
        # a few chosen rays with their whole paths, as a plot needs them
        {"name": "paths_small", "kind": "paths", "scene": "tetra", "n": 61, "record": 16, "reference": False},
        # a ray fan at the library's default constants (100 x 100 coarse grid, tolerance 1e-3)
        {"name": "paths_reference", "kind": "paths", "scene": "two_spheres", "n": 4099, "record": 8,
         "reference": True},
        # a path data set copied back to the host
        {"name": "paths_large", "kind": "paths", "scene": "tetra", "n": 262147, "record": 8, "reference": False},
        # the tetrahedron workload at full size, reference arithmetic
        {"name": "device_tetra_1m", "kind": "device", "scene": "tetra", "n": 1048576, "reference": False,
         "split": False},
        # a middle-sized batch with the FP32 / FP64 split Newton
        {"name": "device_tetra_split", "kind": "device", "scene": "tetra", "n": 130001, "reference": False,
         "split": True},
        # the largest workload: 16 ellipsoids, 4M rays
        {"name": "device_ellipsoids_4m", "kind": "device", "scene": "ellipsoids", "n": 4194304, "reference": False,
         "split": False},
        # a plane source over the tetrahedron
        {"name": "plane_tetra", "kind": "plane", "scene": "tetra", "nx": 1001, "ny": 640, "reference": False},
        # a bounce map of a few patches
        {"name": "bounce_tetra", "kind": "bounce", "scene": "tetra", "patches": 3, "grid": 7, "theta": 24,
         "phi": 40, "reference": False},
        # uneven scenes traced together
        {"name": "set_of_6", "kind": "set", "scenes": 6, "first": 16384, "last": 262144},
        # fitting the learned start to a scene
        {"name": "train_tetra", "kind": "train", "scene": "tetra", "n": 16384, "epochs": 8, "reference": False},
    ]


def _log_size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["query", "query", "paths", "paths", "device", "device", "device", "plane", "bounce", "set"])
    scene = rng.choice(sorted(_SCENES))
    ref = scene == "two_spheres" and rng.random() < 0.5   # the default grid is kept for the small scene
    if kind == "query":
        return {"kind": kind, "scene": scene, "n": _log_size(rng, 32, 300000), "reference": ref}
    if kind == "paths":
        return {"kind": kind, "scene": scene, "n": _log_size(rng, 32, 300000), "record": rng.randint(1, 16),
                "reference": ref}
    if kind == "device":
        return {"kind": kind, "scene": scene, "n": _log_size(rng, 5000, 2000000), "reference": ref,
                "split": rng.random() < 0.3}
    if kind == "plane":
        return {"kind": kind, "scene": scene, "nx": _log_size(rng, 40, 1200), "ny": _log_size(rng, 40, 1200),
                "reference": ref}
    if kind == "bounce":
        return {"kind": kind, "scene": scene, "patches": rng.randint(1, 5), "grid": rng.randint(2, 9),
                "theta": rng.randint(4, 40), "phi": rng.randint(4, 40), "reference": ref}
    return {"kind": kind, "scenes": rng.randint(2, 8), "first": _log_size(rng, 4000, 30000),
            "last": _log_size(rng, 40000, 300000)}


# ---- scenes -----------------------------------------------------------------

@functools.lru_cache(maxsize=None)
def _obstacles(scene):
    """(centre, semi-axes, rotation, m, nodes per axis) of every obstacle."""
    if scene == "two_spheres":
        return [((cx, 0.0, 0.0), (1.0, 1.0, 1.0), None, 4, 5) for cx in (-1.5, 1.5)]
    if scene == "tetra":
        return [(c, (1.0, 1.0, 1.0), None, 8, 7) for c in scenes.tetrahedron_centers(2.5)]
    if scene == "ellipsoids":
        g = np.random.Generator(np.random.PCG64(2024))
        return [(c, a, q, 8, 7) for c, a, q in scenes.random_ellipsoids(g, 16)]
    # member k of the multi-scene kind: 1 to 5 spheres and ellipsoids, 96 or 384 patches each
    k = int(scene.split("_")[1])
    g = np.random.Generator(np.random.PCG64(770 + k))
    out = []
    for c, a, q in scenes.random_ellipsoids(g, 1 + (3 * k + 2) % 5):
        if g.random() < 0.5:
            a, q = (a[0], a[0], a[0]), None
        out.append((c, a, q, 4 if g.random() < 0.5 else 8, 5 if g.random() < 0.5 else 7))
    return out


@functools.lru_cache(maxsize=None)
def _patches(scene):
    out = []
    for k, (c, a, q, m, nn) in enumerate(_obstacles(scene)):
        out += scenes.obstacle_patches(k, c, a, q, m=m, n_nodes=nn)
    return out


@functools.lru_cache(maxsize=None)
def _table(scene):
    return C.ObjectTable(_patches(scene))


def _shape(scene):
    return _SCENES.get(scene, _SCENES["ellipsoids"])


def _scene(scene, reference, split=False):
    cfg = C.default_config() if reference else C.default_config(coarse_grid_n=_shape(scene)[4], newton_tol=1e-12)
    s = api.Scene(config=cfg, table=_table(scene))
    if split:
        s.set_modes(precision=C.PREC_SPLIT)
    s.upload()
    return s


def _rays(scene, n, seed):
    """Origins uniform on the source plane, directions uniform in a cone about -z (CUDA tensors)."""
    z, h, deg, _, _ = _shape(scene)
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = torch.rand((n, 4), generator=g, device="cuda", dtype=torch.float64)
    o = torch.stack([h * (2.0 * r[:, 0] - 1.0), h * (2.0 * r[:, 1] - 1.0), torch.full_like(r[:, 0], z)], dim=1)
    mu = 1.0 - r[:, 2] * (1.0 - math.cos(math.radians(deg)))
    st, ph = torch.sqrt(torch.clamp(1.0 - mu * mu, min=0.0)), 2.0 * math.pi * r[:, 3]
    d = torch.stack([st * torch.cos(ph), st * torch.sin(ph), -mu], dim=1)
    return o.contiguous(), d.contiguous()


def _device_outputs(n):
    return {"status": torch.empty(n, dtype=torch.int32, device="cuda"),
            "bounce_count": torch.empty(n, dtype=torch.int32, device="cuda"),
            "exit_dir": torch.empty((n, 3), dtype=torch.float64, device="cuda"),
            "end_point": torch.empty((n, 3), dtype=torch.float64, device="cuda")}


def _members(case):
    """(scene, ray count) of a set's members, the counts spread evenly in their logarithm."""
    k = case["scenes"]
    f = (case["last"] / case["first"]) ** (1.0 / max(1, k - 1))
    return [("member_%d" % j, int(round(case["first"] * f ** j)) + j) for j in range(k)]


# ---- states -----------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    if kind == "set":
        mem = [_scene(name, False) for name, _ in _members(case)]
        rays = [_rays(name, n, 64 * seed + j) for j, (name, n) in enumerate(_members(case))]
        torch.cuda.synchronize()
        return {"case": case, "set": api.SceneSet(mem), "members": mem, "rays": rays,
                "outs": [_device_outputs(n) for _, n in _members(case)]}
    scene = case["scene"]
    st = {"case": case, "scene": _scene(scene, case["reference"], case.get("split", False))}
    z, h, deg, _, _ = _shape(scene)
    if kind in ("query", "paths", "train"):
        o, d = _rays(scene, case["n"], seed)
        st["o"], st["d"] = o.cpu().numpy(), d.cpu().numpy()
    elif kind == "device":
        st["o"], st["d"] = _rays(scene, case["n"], seed)
        st["out"] = _device_outputs(case["n"])
        torch.cuda.synchronize()
    elif kind == "plane":
        rng = np.random.Generator(np.random.PCG64(seed))
        w, t, p = h * (0.9 + 0.1 * rng.random()), math.radians(deg) * rng.random(), 2.0 * math.pi * rng.random()
        st["corner0"], st["corner1"] = (-w, -w, z), (w, w, z)
        st["dir"] = (math.sin(t) * math.cos(p), math.sin(t) * math.sin(p), -math.cos(t))
    elif kind == "bounce":
        rng = np.random.Generator(np.random.PCG64(seed))
        st["patches"] = [_patches(scene)[int(k)] for k in rng.choice(len(_patches(scene)), case["patches"], False)]
        st["cone"] = 120.0 + 50.0 * rng.random()
    return st


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "set":
        ptrs = [{k: v.data_ptr() for k, v in o.items()} for o in state["outs"]]
        state["set"].trace_device([o.data_ptr() for o, _ in state["rays"]], [d.data_ptr() for _, d in state["rays"]],
                                  [o.shape[0] for o, _ in state["rays"]], 100, ptrs, want_stats=False)
        return state["outs"]
    s, bounces = state["scene"], _shape(case["scene"])[3]
    if kind == "query":
        hit = s.intersect(state["o"], state["d"])
        return {k: hit[k] for k in ("t", "point", "normal", "uv", "object", "status")}
    if kind == "paths":
        return dict(s.trace(state["o"], state["d"], bounces, record=case["record"], want_stats=False))
    if kind == "device":
        o = state["o"]
        s.trace_device(o.data_ptr(), state["d"].data_ptr(), o.shape[0], bounces,
                       {k: v.data_ptr() for k, v in state["out"].items()})
        return state["out"]
    if kind == "plane":
        return s.plane_source(state["corner0"], state["corner1"], state["dir"], case["nx"], case["ny"], bounces)
    if kind == "bounce":
        return s.bounce_map(state["patches"], case["grid"], case["theta"], case["phi"], state["cone"], 50)
    s.guess_train(state["o"], state["d"], bounces, epochs=case["epochs"], batch=1 << 22,
                  max_positive=8 * case["n"], max_negative=64 * case["n"])
    return s.guess_params()


# ---- what a pass cannot do without ------------------------------------------

def _rays_of(case):
    kind = case["kind"]
    if kind == "set":
        return sum(n for _, n in _members(case))
    if kind == "plane":
        return case["nx"] * case["ny"]
    if kind == "bounce":
        return case["patches"] * case["grid"] ** 2 * case["theta"] * case["phi"]
    return case["n"]


def _scene_bytes(scene):
    """Node values of a scene's patches: 12 doubles per node, and its boxes."""
    return sum(6 * m * m * (nn * nn * 96 + 48) for _, _, _, m, nn in _obstacles(scene))


def work(case):
    """Rays in, results out and the scene once; operations: per bounce one Newton solve of about five
    iterations (18 N^2 + 24 N + 70) and per query one path down the tree (25 node tests of 16)."""
    kind, n = case["kind"], _rays_of(case)
    per_ray = {"query": 48 + 112, "paths": 48 + 80 + 44 * case.get("record", 0), "device": 48 + 56, "plane": 0,
               "bounce": 0, "set": 48 + 56, "train": 48}[kind]
    names = [m for m, _ in _members(case)] if kind == "set" else [case["scene"]]
    nn = max(o[4] for name in names for o in _obstacles(name))
    per_bounce = 5 * (18 * nn * nn + 24 * nn + 70)
    flops = n * (0.5 * per_bounce + 1.5 * 25 * 16)
    if kind == "train":
        flops += case["epochs"] * n * 3 * 86e3
    return {"bytes": float(n * per_ray + sum(_scene_bytes(x) for x in names)), "flops": float(flops)}


# ---- 64-bit values ----------------------------------------------------------
#
# Closed convex obstacles: the surface point a ray meets is found on the exact ellipsoid, which names the
# patch and a start, and Newton in plain torch then solves on that patch's interpolant.  A ray that the
# framework ends with an error status has no such value; the few there are stay in as they are.

def _t(a):
    return torch.as_tensor(np.asarray(a), dtype=torch.float64, device="cuda")


@functools.lru_cache(maxsize=2)
def _surface(scene):
    obs = _obstacles(scene)
    eye = ((1.0, 0.0, 0.0), (0.0, 1.0, 0.0), (0.0, 0.0, 1.0))
    nn = max(o[4] for o in obs)
    return {"c": _t([o[0] for o in obs]), "a": _t([o[1] for o in obs]), "q": _t([o[2] or eye for o in obs]),
            "m": obs[0][3], "x": _t(scenes.cheb_lobatto(nn)),
            "f": _t(np.stack([np.stack([p.x, p.y, p.z, p.dxdu, p.dydu, p.dzdu, p.dxdv, p.dydv, p.dzdv, p.nu_x, p.nu_y,
                                        p.nu_z], 1).reshape(nn, nn, 12) for p in _patches(scene)]))}


_FRAMES = [((1, 0, 0), (0, 1, 0), (0, 0, 1)), ((-1, 0, 0), (0, 0, 1), (0, 1, 0)), ((0, 1, 0), (0, 0, 1), (1, 0, 0)),
           ((0, -1, 0), (1, 0, 0), (0, 0, 1)), ((0, 0, 1), (1, 0, 0), (0, 1, 0)), ((0, 0, -1), (0, 1, 0), (1, 0, 0))]


def _basis(x, u):
    """Lagrange polynomials on the nodes x at u, in product form."""
    k = x.numel()
    off = ~torch.eye(k, dtype=torch.bool, device=x.device)
    num = torch.where(off, u[:, None, None] - x[None, None, :], 1.0).prod(-1)
    return num / torch.where(off, x[:, None] - x[None, :], 1.0).prod(-1)


def _first_hit(S, o, d, last):
    """(hit, t, point, normal, uv, obstacle) of the first surface each ray meets; `last`: the obstacle it leaves."""
    lo = torch.einsum("kji,nkj->nki", S["q"], o[:, None] - S["c"]) / S["a"]
    ld = torch.einsum("kji,nj->nki", S["q"], d) / S["a"]
    A, B, G = (ld * ld).sum(-1), (lo * ld).sum(-1), (lo * lo).sum(-1) - 1.0
    disc = B * B - A * G
    t = torch.where(disc > 0, (-B - torch.sqrt(disc.clamp(min=0.0))) / A, torch.inf)
    t = torch.where(t > 0, t, torch.inf)
    t[torch.arange(S["c"].shape[0], device=t.device)[None] == last[:, None]] = torch.inf
    t, k = t.min(1)
    hit = torch.isfinite(t)
    t0, k = torch.where(hit, t, 0.0), torch.where(hit, k, 0)
    ar = torch.arange(o.shape[0], device=o.device)
    s = lo[ar, k] + t0[:, None] * ld[ar, k]
    face = 2 * s.abs().argmax(1)
    face = face + (s.gather(1, (face // 2)[:, None])[:, 0] < 0)
    fr = _t(_FRAMES)[face]
    w = (s * fr[:, 0]).sum(1)
    ab = torch.stack([(s * fr[:, 1]).sum(1) / w, (s * fr[:, 2]).sum(1) / w], 1)
    m = S["m"]
    cell = torch.floor((ab + 1.0) * 0.5 * m).clamp(0, m - 1)
    uv = ((ab + 1.0) * m - 2.0 * cell - 1.0).clamp(-1.0, 1.0)
    f = S["f"][((k * 6 + face) * m + cell[:, 0].long()) * m + cell[:, 1].long()]
    x = torch.cat([uv, t0[:, None]], 1)
    for _ in range(4):
        e = torch.einsum("ni,nj,nijf->nf", _basis(S["x"], x[:, 0]), _basis(S["x"], x[:, 1]), f)
        J = torch.stack([e[:, 3:6], e[:, 6:9], -d], 2)
        J = torch.where(hit[:, None, None], J, torch.eye(3, dtype=J.dtype, device=J.device))
        x = x - torch.linalg.solve(J, e[:, 0:3] - o - x[:, 2:] * d)
    e = torch.einsum("ni,nj,nijf->nf", _basis(S["x"], x[:, 0]), _basis(S["x"], x[:, 1]), f)
    return hit, x[:, 2], e[:, 0:3], torch.nn.functional.normalize(e[:, 9:12], dim=1), x[:, 0:2], k


def _exact_trace(scene, o, d, bounces, record):
    S, n = _surface(scene), o.shape[0]
    exit_dir = torch.nn.functional.normalize(d, dim=1)
    point = torch.zeros((n, record, 3), dtype=torch.float64, device="cuda")
    at, p, last = torch.arange(n, device="cuda"), o.clone(), torch.full((n,), -1, device="cuda")
    for b in range(bounces):
        hit, _, q, nrm, _, k = _first_hit(S, p, exit_dir[at], last)
        at, p, nrm, last = at[hit], q[hit], nrm[hit], k[hit]
        if not at.numel():
            break
        if b < record:
            point[at, b] = p
        v = exit_dir[at]
        exit_dir[at] = v - 2.0 * (v * nrm).sum(1, keepdim=True) * nrm
    return exit_dir, point


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("query", "paths", "device"):
        return None
    scene = case["scene"]
    o, d = _rays(scene, case["n"], seed)
    step = 1 << 17
    if kind == "query":
        S, got = _surface(scene), []
        for k in range(0, case["n"], step):
            a, b = o[k:k + step], d[k:k + step]
            hit, t, p, nrm, uv, _ = _first_hit(S, a, b, torch.full((a.shape[0],), -1, device="cuda"))
            got.append([torch.where(hit.reshape((-1,) + (1,) * (x.dim() - 1)), x, 0.0) for x in (t, p, nrm, uv)])
        t, p, nrm, uv = (torch.cat(x) for x in zip(*got))
        return {"t": t, "point": p, "normal": nrm, "uv": uv, "object": None, "status": None}
    record = case.get("record", 0)
    got = [_exact_trace(scene, o[k:k + step], d[k:k + step], _shape(scene)[3], record)
           for k in range(0, case["n"], step)]
    out = {"exit_dir": torch.cat([x for x, _ in got])}
    if record:
        out["hit_point"] = torch.cat([x for _, x in got])
    return out
