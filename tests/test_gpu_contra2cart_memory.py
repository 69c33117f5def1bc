"""Contra2Cart where its twelve planes of grid quantities do not fit (VFS_CONTRA2CART_PLANES=0
stands for an allocation that fails): the same bits from the cell metrics."""
import numpy as np
import pytest

import oracle as O
from test_gpu_stages import BOXES, build

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,periodic", BOXES, ids=["x".join(map(str, b[0])) for b in BOXES])
def test_without_planes(cuda_lib, monkeypatch, dims, periodic):
    import torch
    import vfs_poisson as V
    case, rng = build(dims, periodic, "odd")
    d = O.dims_of(case)
    met = O.form_metrics(d, case.coor)
    v0 = rng.normal(size=case.ucont.shape)
    u0 = case.ucont * 2.0 ** rng.integers(-1040, 1000, size=case.ucont.shape[:3] + (1,))
    monkeypatch.setenv("VFS_CONTRA2CART_PLANES", "0")
    s = V.PoissonSolver(*case.dims, periodic=periodic)
    try:
        s.set_grid(case.coor)
        s.set_nvert(case.nvert)
        got = torch.from_numpy(v0.copy()).cuda()
        s.contra2cart(torch.from_numpy(u0).cuda(), got)
        want = O.contra2cart(d, case.nvert, met, u0, v0, zero_solid=True)
        np.testing.assert_array_equal(got.cpu().numpy().view(np.int64), want.view(np.int64))
    finally:
        s.close()
