"""The surface search's FP32 pre-test and its passes over the index box of a
body against the oracle, bit for bit: slivers, triangles far smaller than a
cell, faces edge-on to the rays and in planes of cell centres, a soup of
random triangles (rays that give up included), a body outside the grid; and
the first body over masks with values off 0..3, walls, and boundary points
that count as marks (the whole-grid passes)."""
import numpy as np
import pytest

from vfs_poisson import configs as CF
from test_gpu_ibm import _assert_same, _run_both

pytestmark = pytest.mark.gpu


def _box(lo, hi):
    v = np.array([[(lo, hi)[i][0], (lo, hi)[j][1], (lo, hi)[k][2]] for k in (0, 1) for j in (0, 1) for i in (0, 1)])
    q = [(0, 1, 3, 2), (4, 6, 7, 5), (0, 4, 5, 1), (2, 3, 7, 6), (0, 2, 6, 4), (1, 5, 7, 3)]
    return v, np.array([t for a, b, c, d in q for t in ((a, b, c), (a, c, d))], np.int32)


def _surface(name):
    rng = np.random.default_rng(4)
    if name == "slivers":
        return CF.rod_surface((0.4, 0.1, 0.45), (0.1, 1.0, 0.05), 0.7, 0.15, 90, 1)
    if name == "tiny":
        return CF.rod_surface((0.5, 0.45, 0.5), (0.3, 0.2, 1.0), 0.06, 0.03, 64, 40)
    if name == "edge_on":
        return _box((0.25, 0.25, 0.25), (0.75, 0.625, 0.75))
    if name == "outside":
        return _box((3.0, 3.0, 3.0), (3.5, 3.5, 3.5))
    xyz = rng.uniform(0.1, 0.9, (40, 3))
    return xyz, rng.permuted(np.tile(np.arange(40, dtype=np.int32), (60, 1)), axis=1)[:, :3].copy()


@pytest.mark.parametrize("name", ["slivers", "tiny", "edge_on", "soup", "outside"])
def test_ray_pretest(cuda_lib, name):
    c = CF.channel(32, 24, 32) if name == "edge_on" else CF.cylinder(34, 23, 29)
    if name == "edge_on":  # uniform in y, too: faces through cell centres
        c.coor[..., 1] = np.arange(c.coor.shape[1])[None, :, None] / 24.0
    surf = _surface(name)
    _assert_same(*_run_both(c, [surf, _surface("slivers")]))


@pytest.mark.parametrize("boundary4", [False, True])
def test_first_body_on_odd_masks(cuda_lib, boundary4):
    c = CF.cylinder(26, 18, 22)
    rng = np.random.default_rng(6)
    nv = rng.choice([0.0, 1.0, 3.0, 5.0, 6.0, -0.5, 2.5, 4.0], size=(c.nz + 2, c.ny + 2, c.nx + 2))
    b = np.ones_like(nv, dtype=bool)
    b[1:-1, 1:-1, 1:-1] = False
    nv[b] = rng.choice([0.0, 1.0, 3.0, -1.0, 6.0] + ([4.0] if boundary4 else []), size=int(b.sum()))
    for bc in (None, (-1, 0, 0, -2, 0, 0)):
        _assert_same(*_run_both(c, [_surface("slivers"), _surface("tiny")], nvert0=nv, bctype=bc))
