"""Projection's division by coeff, bit for bit against the oracle's: divisors
whose reciprocal is close enough for the short correction (1 - d y at most
2^-54), divisors that need the reciprocal's rest, a power of two, divisors past
the range of both, and zero, tiny and huge numerators."""
import numpy as np
import pytest

import oracle as O
from test_gpu_stages import BOXES, build

pytestmark = pytest.mark.gpu

COEFF = [1.5, 3.0, 0.25, 1.1, 0.7, -1.7, 7.0 / 3.0, 2.0 ** 99 * 1.3, 2.0 ** 101, 2.0 ** -120 * 1.9]


@pytest.mark.parametrize("kind", ["none", "odd"])
@pytest.mark.parametrize("dims,periodic", BOXES[3:6:2], ids=["x".join(map(str, b[0])) for b in BOXES[3:6:2]])
def test_projection_quotients(cuda_lib, dims, periodic, kind):
    import vfs_poisson as V
    case, rng = build(dims, periodic, kind, seed=11)
    d = O.dims_of(case)
    met = O.form_metrics(d, case.coor)
    phi = rng.standard_normal(case.nvert.shape)
    phi *= 2.0 ** rng.integers(-900, 400, size=phi.shape[:2] + (1,))
    phi[rng.random(phi.shape) < 0.3] = 0.
    s = V.PoissonSolver(*case.dims, periodic=periodic)
    try:
        s.set_grid(case.coor)
        s.set_nvert(case.nvert)
        p, f = O.update_pressure(d, case.nvert, np.zeros_like(phi), phi)
        s.update_pressure(np.zeros_like(phi), phi.copy())
        for coeff in COEFF:
            for u0 in (case.ucont, np.zeros_like(case.ucont)):
                want = O.projection(d, case.nvert, f, met, u0, 0.3, 1.0, coeff)
                got = s.projection(u0.copy(), 0.3, 1.0, coeff)
                np.testing.assert_array_equal(got, want, err_msg=str(coeff))
    finally:
        s.close()
