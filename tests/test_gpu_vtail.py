"""The V-cycle's small levels in one cluster (smoother 4) against the same
levels launch by launch (smoother 3), bit for bit: slabs of one and of several
k-planes, fewer planes than CTAs, odd rows, lines of one chunk and of 32, part
chunks, every wrap, bodies across the seams, one, two and no pre-sweeps."""
import numpy as np
import pytest

from vfs_poisson import configs as CF

pytestmark = pytest.mark.gpu

BOXES = [((24, 16, 24), (0, 0, 0, 1, 0, 0)), ((12, 10, 40), (0, 0, 0, 1, 0, 1)), ((15, 12, 18), (1, 0, 0, 0, 0, 1)),
         ((16, 250, 12), (0, 0, 0, 0, 0, 1)), ((9, 8, 6), (0, 0, 0, 0, 1, 1)), ((40, 24, 5), (0, 0, 0, 0, 0, 0)),
         ((6, 20, 66), (0, 0, 0, 1, 1, 1)), ((20, 36, 28), (0, 0, 0, 0, 0, 0))]


@pytest.mark.parametrize("precision", [0, 1], ids=["fp32", "fp64"])
@pytest.mark.parametrize("dims,periodic", BOXES, ids=["x".join(map(str, b[0])) for b in BOXES])
def test_tail_bitexact(cuda_lib, dims, periodic, precision):
    import vfs_poisson as V
    case = CF.cylinder(*dims, seed=5)
    case.set_periodic(periodic)
    s = V.PoissonSolver.from_case(case)
    try:
        s.rhs(case.ucont)
        for kw in ({}, {"nu1": 2, "nu2": 1, "omega": 0.9}, {"nu1": 0, "nu2": 3}):
            out = [s.solve(precision=precision, rtol=1e-7, max_it=80, smoother=sm, **kw) for sm in (3, 4)]
            assert out[0][1].iterations == out[1][1].iterations and out[0][1].status == 0, kw
            np.testing.assert_array_equal(out[0][0], out[1][0], err_msg=str(kw))
    finally:
        s.close()
