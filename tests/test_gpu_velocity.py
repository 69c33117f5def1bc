"""Contra2Cart and IB_BC against the oracle, bit for bit, on host and on device
arrays: boxes from one cell on, every periodic axis, blanking values off 0, 1
and 3 (on ghost points too), and fluxes whose quotients leave the range of the
reciprocal path (zeros of both signs, subnormals, huge values)."""
import numpy as np
import pytest

import oracle as O
from test_gpu_stages import BOXES, build

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("values", ["plain", "scales"])
@pytest.mark.parametrize("kind", ["none", "odd"])
@pytest.mark.parametrize("dims,periodic", BOXES, ids=["x".join(map(str, b[0])) for b in BOXES])
def test_velocity_stages(cuda_lib, dims, periodic, kind, values):
    import torch
    import vfs_poisson as V
    case, rng = build(dims, periodic, kind)
    d = O.dims_of(case)
    met = O.form_metrics(d, case.coor)
    u0, v0 = case.ucont, rng.normal(size=case.ucont.shape)
    if values == "scales":
        u0 = u0 * 2.0 ** rng.integers(-1040, 1000, size=u0.shape[:3] + (1,))
        u0[rng.random(u0.shape[:3]) < 0.3] = 0.0
        u0[rng.random(u0.shape[:3]) < 0.3] = -0.0
    s = V.PoissonSolver(*case.dims, periodic=periodic)
    try:
        s.set_grid(case.coor)
        s.set_nvert(case.nvert)
        for device in (False, True):
            def arr(a):
                return torch.from_numpy(a.copy()).cuda() if device else a.copy()

            def bits(a):
                return (a.cpu().numpy() if device else a).view(np.int64)

            for zero in (True, False):
                want = O.contra2cart(d, case.nvert, met, u0, v0, zero_solid=zero)
                got = arr(v0)
                s.contra2cart(arr(u0), got, zero_solid=zero)
                np.testing.assert_array_equal(bits(got), want.view(np.int64))
            for bc, immersed in (((0,) * 6, 1), ((10, 10, 10, 10, 10, 10), 3), ((-1, -2, -1, -2, 0, 10), 0)):
                want = O.ib_bc(d, case.nvert, met, v0, case.ucont, bctype=bc, immersed=immersed)
                got = arr(v0), arr(case.ucont)
                s.ib_bc(*got, immersed=immersed, bctype=bc)
                for a, b in zip(got, want):
                    np.testing.assert_array_equal(a.cpu().numpy() if device else a, b)
    finally:
        s.close()
