"""The surface search's FP32 pre-test on bodies from unit size to sizes whose FP32
products overflow, against the oracle, bit for bit: soups of triangles, and cells just
below the top of a body (where the ray is short against the body) beside a wall that
leans by less than the FP32 error of the ray's direction."""
import numpy as np
import pytest

from vfs_poisson import configs as CF
from test_gpu_ibm import _assert_same, _run_both
from test_gpu_ibm_rays import _box, _surface

pytestmark = pytest.mark.gpu

RAND1 = 1804289383 / 2.0 ** 31 - 0.5  # the first ray's offset in its hash cell, in cells


@pytest.mark.parametrize("scale", [1e2, 1e4, 1e8, 3e13, 1e14])
@pytest.mark.parametrize("name", ["soup", "slivers"])
def test_scaled_bodies(cuda_lib, name, scale):
    c = CF.cylinder(26, 18, 22)
    c.coor = c.coor * scale
    xyz, tri = _surface(name)
    _assert_same(*_run_both(c, [(xyz * scale, tri)]))


@pytest.mark.parametrize("scale", [1e2, 1e3, 1e4, 1e6])
def test_short_rays_beside_leaning_walls(cuda_lib, scale):
    # a large low body gives the box its size; a tower whose wall leans towards the
    # first ray's aim rises over it; the cells are the last 0.3 below its top
    xyz, tri = _box((0.0, 0.0, 0.0), (scale, scale, 0.4 * scale))
    at = (20.5 + RAND1) * (scale + 0.1) / 39.0 - 0.05
    top = 0.9 * scale
    for lean, x0 in ((1e-3, at - 0.004), (1e-5, at + 0.011), (-1e-4, at + 0.037)):
        v, t = _box((x0, at - 0.21 * scale, 0.5 * scale), (x0 + 0.2 * scale, at + 0.23 * scale, top))
        v[:, 0] += lean * (v[:, 2] - top)
        tri = np.concatenate([tri, t + len(xyz)])
        xyz = np.concatenate([xyz, v])
    c = CF.channel(24, 16, 24)
    unit = c.coor / c.coor.reshape(-1, 3).max(0)
    c.coor = np.array([at - 0.06, at - 0.05, top - 0.3]) + unit * np.array([0.12, 0.1, 0.32])
    _assert_same(*_run_both(c, [(xyz, tri.astype(np.int32))]))
