"""The V-cycle's tail with lines of 5 to 16 chunks (joined through shared memory; up to
4 lie in a warp), whole and part last chunks, one and two planes a CTA: bit for bit the
launch-by-launch levels (smoother 3), with and without scattered blank cells, and shown
to have run: from level 0 a V-cycle is one launch beside the four that bring it its
input and take its result, from level 1 it is that of nine or fourteen more."""
import numpy as np
import pytest

from vfs_poisson import configs as CF

pytestmark = pytest.mark.gpu

BOXES = [((24, 40, 12), 0), ((8, 41, 16), 0), ((8, 44, 30), 0), ((16, 60, 16), 0), ((8, 100, 16), 0),
         ((8, 104, 12), 0), ((8, 122, 16), 0), ((4, 128, 8), 0), ((24, 41, 24), 1)]


@pytest.mark.parametrize("blanked", [0.0, 0.05])
@pytest.mark.parametrize("precision", [0, 1], ids=["fp32", "fp64"])
@pytest.mark.parametrize("dims,level", BOXES, ids=["x".join(map(str, b[0])) for b in BOXES])
def test_long_lines(cuda_lib, dims, level, precision, blanked):
    import vfs_poisson as V
    rng = np.random.default_rng(7)
    case = CF.cylinder(*dims, seed=5)
    if blanked:
        case.nvert = np.where(rng.random(case.nvert.shape) < blanked, 3.0, 0.0)
    s = V.PoissonSolver.from_case(case)
    try:
        r = rng.normal(size=case.nvert.shape)
        before = s.kernel_launches()
        s.mg_vcycle(r, precision)
        assert s.kernel_launches() - before == 5 + level * (14 if precision else 9)
        s.rhs(case.ucont)
        for kw in ({}, {"nu1": 2, "nu2": 1, "omega": 0.9}, {"nu1": 0, "nu2": 3}):
            out = []
            for sm in (3, 4):
                before = s.kernel_launches()
                phi, st = s.solve(precision=precision, rtol=1e-30, max_it=4, smoother=sm, use_graphs=0, **kw)
                out.append((phi, s.kernel_launches() - before))
            assert np.isfinite(out[0][0]).all()
            np.testing.assert_array_equal(out[0][0], out[1][0], err_msg=str(kw))
            assert out[1][1] < out[0][1], kw  # (the tail ran for these sweeps, too)
    finally:
        s.close()
