"""The mean removal of the right-hand side at the ends of the FP64 range.  Its quotients
are the division's bits, so a flux scaled by a power of two gives the right-hand side
scaled by it as long as every result is normal, whatever the remainders are; and an
infinite product of sum and aj gives an infinite quotient."""
import numpy as np
import pytest

import oracle as O
from test_gpu_stages import build

pytestmark = pytest.mark.gpu


def _solver(scale):
    import vfs_poisson as V
    case, _ = build((12, 9, 10), (0, 0, 0, 1, 0, 0), "none", seed=7)
    case.coor = case.coor * scale
    u = np.round(case.ucont * 2.0 ** 20) / 2.0 ** 20  # few bits: scaled exactly, summed exactly
    d = O.dims_of(case)
    met = O.form_metrics(d, case.coor)
    gid = O.poisson_lhs(d, case.nvert, met)["gid"]
    total = O.rhs(d, case.nvert, gid, u, met["aj"], bctype3=-10).sum()
    s = V.PoissonSolver.from_case(case)
    return s, u, total, met["aj"][1:-1, 1:-1, 1:-1]


@pytest.mark.parametrize("log2_grid", [12, 20])
def test_power_of_two_scaling(cuda_lib, log2_grid):
    s, u, total, aj = _solver(2.0 ** log2_grid)
    try:
        s.rhs(u)
        base = s.rhs_array()
        # the smallest numerator |total aj| lands just above the smallest normal value
        for lowest in (-1021, -1016, -990, -500, 100):
            k = lowest + 1 - int(np.floor(np.log2(abs(total) * aj.min())))
            s.rhs(np.ldexp(u, k))
            np.testing.assert_array_equal(s.rhs_array().view(np.int64), np.ldexp(base, k).view(np.int64), err_msg=str(k))
    finally:
        s.close()


def test_infinite_numerators_and_zero_sums(cuda_lib):
    s, u, total, aj = _solver(2.0 ** -30)
    try:
        s.rhs(np.ldexp(u, 1000))
        b = s.rhs_array()[1:-1, 1:-1, 1:-1]
        np.testing.assert_array_equal(b, np.where(total > 0, -np.inf, np.inf) + np.zeros_like(b))
        s.rhs(np.zeros_like(u))
        assert not s.rhs_array().any()
    finally:
        s.close()
