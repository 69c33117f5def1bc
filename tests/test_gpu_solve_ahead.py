"""Solves from zero, whose first step is launched before its norm is known,
against the same solves started from a given zero array (norm read first),
bit for bit: one step, a restart after every one or two steps, no step at
all, both orthogonalisations; and right-hand sides that are zero or not
finite, which take no step."""
import numpy as np
import pytest

from vfs_poisson import configs as CF

pytestmark = pytest.mark.gpu

OPTS = [{}, {"max_it": 1}, {"max_it": 2}, {"restart": 1, "max_it": 5}, {"restart": 2, "max_it": 7}, {"rtol": 0.9},
        {"rtol": 1.0}, {"nu2_near": 1, "rtol": 0.05}, {"precision": 1, "restart": 3}]


@pytest.mark.parametrize("orth", [0, 1])
@pytest.mark.parametrize("dims", [(24, 16, 24), (9, 8, 6)], ids=["24x16x24", "9x8x6"])
def test_from_zero_bitexact(cuda_lib, dims, orth):
    import vfs_poisson as V
    case = CF.cylinder(*dims, seed=3)
    s = V.PoissonSolver.from_case(case)
    try:
        s.rhs(case.ucont)
        for kw in OPTS:
            a, b = np.zeros(case.nvert.shape), np.zeros(case.nvert.shape)
            (a, sa), (b, sb) = s.solve(a, orth=orth, **kw), s.solve(b, orth=orth, warm_start=1, **kw)
            assert sa.iterations == sb.iterations and sa.status == sb.status, kw
            assert sa.rel_residual == sb.rel_residual and sa.initial_rel_residual == sb.initial_rel_residual, kw
            np.testing.assert_array_equal(a, b, err_msg=str(kw))
        for value in (0., np.nan, np.inf):
            s.rhs(np.full_like(case.ucont, value))
            a, b = np.zeros(case.nvert.shape), np.zeros(case.nvert.shape)
            (a, sa), (b, sb) = s.solve(a, orth=orth), s.solve(b, orth=orth, warm_start=1)
            assert sa.iterations == sb.iterations == 0 and sa.status == sb.status, value
            np.testing.assert_array_equal(a, b, err_msg=str(value))
    finally:
        s.close()
