"""The autotuner varies what acts on the scene: the launch shape only where
k_advance runs the rounds."""
import numpy as np
import pytest

from billardballraytracing3d_b200 import _capi as C
from billardballraytracing3d_b200 import api, scenes

pytestmark = pytest.mark.gpu


def test_launch_shape_is_left_alone_in_split_rounds(built):
    patches, o, d, maxb, cn, tol = scenes.workload("tetra_spheres", 16384)
    o, d = np.ascontiguousarray(o[:12000]), np.ascontiguousarray(d[:12000])
    shapes = set()
    for _ in range(6):   # four shapes that do the same: noise would pick one of them
        sc = api.Scene(patches, config=C.default_config(coarse_grid_n=cn, newton_tol=tol))
        shapes.add(sc.autotune(o, d, maxb, trials=1)["advance_shape"])
    assert shapes == {3}
