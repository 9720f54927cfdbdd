"""Plane source, bounce map and large query batches over odd sizes against the
oracle: whole numbers and doubles bit for bit."""
import numpy as np
import pytest

import oracle
from billardballraytracing3d_b200 import _capi as C
from billardballraytracing3d_b200 import api, scenes

pytestmark = pytest.mark.gpu
CFG = dict(coarse_grid_n=9, newton_tol=1e-12)


@pytest.fixture(scope="module")
def pair(built):
    patches = scenes.scene_two_spheres()
    return patches, api.Scene(patches, config=C.default_config(**CFG)), oracle.Oracle(patches, config=C.default_config(**CFG))


@pytest.mark.parametrize("nx,ny", [(1, 7), (33, 1), (97, 31), (300, 257)])
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_plane_source_grids(pair, nx, ny, axis):
    _, sc, orc = pair
    c0, c1 = [-2.0, -2.5, -3.0], [2.5, 2.0, 3.0]
    c0[axis] = c1[axis] = 4.0
    d = [0.2, 0.1, -0.3]
    d[axis] = -1.0
    o = scenes.plane_grid(c0, c1, nx, ny)
    ref = orc.plane_counts(o, np.array(d), 20, False)
    assert np.array_equal(sc.plane_source(c0, c1, d, nx, ny, 20), ref)


@pytest.mark.parametrize("theta_n,phi_n", [(1, 1), (1, 31), (4, 8), (3, 11), (13, 5)])
def test_bounce_map_direction_counts(pair, theta_n, phi_n):
    patches, sc, orc = pair
    samples = [patches[3], patches[100]]
    a = sc.bounce_map(samples, 3, theta_n, phi_n, 170.0, 20)
    b = orc.bounce_map(samples, 3, theta_n, phi_n, 170.0, 20)
    for x, y in zip(a, b):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("n", [32767, 32768, 40001])
@pytest.mark.parametrize("precision", [C.PREC_FP64, C.PREC_SPLIT])
def test_large_query_batches(pair, n, precision):
    _, sc, orc = pair
    o, d = scenes.cone_rays(n, 8, 4.0, 3.0, 25.0)
    d[::5] *= 0.25                   # shorter and longer than unit: queries take directions as they are
    d[::7] *= 3.0
    d[::11] = (0.0, 0.0, -1.0)
    o[13] = (np.nan, 0.0, 4.0)
    sc.set_modes(precision)
    a = sc.intersect(o, d)
    sc.set_modes(C.PREC_FP64)
    b = orc.intersect(o, d)
    for k in ("object", "status", "err_object", "t", "point", "normal", "uv", "err_value"):
        assert np.array_equal(a[k], b[k], equal_nan=True), k
