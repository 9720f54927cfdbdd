"""Host arrays of every size class (pinned block without copies, one copy each
way, threaded chunks; pageable and already pinned) give the results of the same
rays in device memory, bit for bit."""
import ctypes

import numpy as np
import pytest

from billardballraytracing3d_b200 import _capi as C
from billardballraytracing3d_b200 import api, scenes

pytestmark = pytest.mark.gpu
OUTS = {"status": (np.int32, 1), "exit_dir": (np.float64, 3), "end_point": (np.float64, 3)}   # 100 bytes a ray with the inputs


@pytest.fixture(scope="module")
def traced(built):
    import torch
    sc = api.Scene(scenes.scene_two_spheres(), config=C.default_config(coarse_grid_n=9, newton_tol=1e-12))
    o, d = scenes.cone_rays(60011, 3, 4.0, 3.0, 20.0)
    n = o.shape[0]
    to, td = torch.from_numpy(o).cuda(), torch.from_numpy(d).cuda()
    t = {k: torch.zeros((n, w), dtype=torch.int32 if dt == np.int32 else torch.float64, device="cuda")
         for k, (dt, w) in OUTS.items()}
    sc.trace_device(to.data_ptr(), td.data_ptr(), n, 20, {k: v.data_ptr() for k, v in t.items()})
    torch.cuda.synchronize()
    return sc, o, d, {k: v.cpu().numpy() for k, v in t.items()}


# around 64 KB (640 rays of 100 bytes and padding), 1 MB and several chunks
@pytest.mark.parametrize("n", [1, 630, 640, 660, 10400, 10486, 10500, 21800, 60011])
@pytest.mark.parametrize("pinned", ["none", "outputs", "all"])
def test_host_arrays_match_device_arrays(traced, n, pinned):
    import torch
    sc, o, d, ref = traced
    keep = []

    def host(a, pin):
        if pin:
            t = torch.from_numpy(np.ascontiguousarray(a)).pin_memory()
            keep.append(t)
            return t.numpy()
        return np.ascontiguousarray(a).copy()

    ho, hd = host(o[:n], pinned == "all"), host(d[:n], pinned == "all")
    out, res = C.TraceOut(), {}
    for k, (dt, w) in OUTS.items():
        res[k] = host(np.full((n, w), -7, dt), pinned != "none")
        setattr(out, k, C.ptr(res[k], ctypes.c_int if dt == np.int32 else ctypes.c_double))
    C.check(sc.lib, sc.lib.bbrt_trace(sc.h, api.P(ho), api.P(hd), n, 20, 0, ctypes.byref(out), None, None), "bbrt_trace")
    for k in OUTS:
        assert np.array_equal(res[k], ref[k][:n]), k
