"""The dof numbering, four cells a thread, against the oracle's: row lengths
that are no multiple of four, part blocks, rows shorter than a
thread's cells, blanked and scattered masks; and the product of the operator
with an array on the device, read and written where it lies."""
import numpy as np
import pytest

import oracle as O
from test_gpu_stages import build

pytestmark = pytest.mark.gpu

BOXES = [((1, 6, 5), (0, 0, 0, 0, 0, 0)), ((3, 5, 7), (0, 0, 0, 1, 0, 0)), ((37, 5, 5), (0, 0, 0, 0, 0, 1)),
         ((33, 5, 6), (1, 0, 0, 0, 0, 0)), ((12, 9, 10), (0, 0, 0, 1, 1, 1))]


@pytest.mark.parametrize("kind", ["none", "plain", "odd"])
@pytest.mark.parametrize("dims,periodic", BOXES, ids=["x".join(map(str, b[0])) for b in BOXES])
def test_numbering_and_apply(cuda_lib, dims, periodic, kind):
    import torch
    import vfs_poisson as V
    case, rng = build(dims, periodic, kind, seed=9)
    d = O.dims_of(case)
    met = O.form_metrics(d, case.coor)
    lhs = O.poisson_lhs(d, case.nvert, met)
    s = V.PoissonSolver(*case.dims, periodic=periodic)
    try:
        s.set_grid(case.coor)
        s.set_nvert(case.nvert)
        ndof, gid = s.numbering()
        assert ndof == lhs["ndof"]
        np.testing.assert_array_equal(gid, lhs["gid"])
        x = rng.standard_normal(case.nvert.shape)
        want = s.apply(x)
        got = torch.full(x.shape, np.nan, dtype=torch.float64, device="cuda")
        xd = torch.from_numpy(x).cuda()
        assert V.load().vfs_poisson_apply(s.h, V._ptr(xd), V._ptr(got, True)) == 0
        np.testing.assert_array_equal(got.cpu().numpy(), want)
    finally:
        s.close()
