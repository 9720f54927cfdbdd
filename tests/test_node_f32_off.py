"""BBRT_NODE_F32=0: no BVH node is tested in FP32, in any size of call (so none is
left over for the FP64 test), and the results are the same."""
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

SCRIPT = r'''
import sys, numpy as np
sys.path.insert(0, sys.argv[1])
from billardballraytracing3d_b200 import scenes, api, _capi as C
patches, o, d, maxb, cn, tol = scenes.workload("tetra_spheres", 40000)
sc = api.Scene(patches, config=C.default_config(coarse_grid_n=cn, newton_tol=tol))
out = {}
for n in (7000, 40000):   # a warp per ray; rounds
    t = sc.trace(o[:n], d[:n], maxb, record=4)
    out.update({f"{n}_{k}": t[k] for k in ("status", "bounce_count", "hit_object", "hit_point", "end_point", "exit_dir")})
    out[f"tests_{n}"] = np.array([t["stats"]["node_tests"], t["stats"]["node_tests_fp64"]])
np.savez(sys.argv[2], **out)
'''


def _run(tmp_path, value):
    path = str(tmp_path / f"r{value}.npz")
    subprocess.run([sys.executable, "-c", SCRIPT, ROOT, path], check=True, env={**os.environ, "BBRT_NODE_F32": value})
    return np.load(path)


def test_no_fp32_node_tests(built, tmp_path):
    on, off = _run(tmp_path, "1"), _run(tmp_path, "0")
    for n in (7000, 40000):
        assert on[f"tests_{n}"][1] > 0 and off[f"tests_{n}"][0] > 0
        assert off[f"tests_{n}"][1] == 0, n
    for k in on.files:
        if not k.startswith("tests"):
            assert np.array_equal(on[k], off[k]), k
