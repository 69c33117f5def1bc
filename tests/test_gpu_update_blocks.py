"""The Gram-Schmidt update of boxes past 304 blocks of 2048 cells, whose last
block is half full (328.5 blocks) or full: the solution's true residual, and the
other orthogonalisation's solution, whose kernels are not the update's.  Both
solves end at 1e-9 of ||b||; their solutions agree to that times the condition of
the preconditioned system, taken as 1e3 (about ten iterations to 1e-9)."""
import numpy as np
import pytest

from vfs_poisson import configs as CF

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(96, 73, 96), (96, 72, 96)], ids=["half", "full"])
def test_update_past_small_boxes(cuda_lib, dims):
    import vfs_poisson as V
    case = CF.cylinder(*dims, seed=6)
    s = V.PoissonSolver.from_case(case)
    try:
        s.rhs(case.ucont)
        b = s.rhs_array()
        a, sa = s.solve(rtol=1e-9, orth=0)
        c, sc = s.solve(rtol=1e-9, orth=1)
        assert sa.status == 0 and sc.status == 0 and abs(sa.iterations - sc.iterations) <= 1
        for phi in (a, c):
            assert np.linalg.norm(b - s.apply(phi)) <= 1.2e-9 * np.linalg.norm(b)
        assert np.linalg.norm(a - c) <= 1e-6 * np.linalg.norm(c)
    finally:
        s.close()
