"""FP32 interpolation in quads of rows and planes (smoother 3, launch by launch)
against the V-cycle tail's own, cell by cell (smoother 4), bit for bit over a few
iterations: scattered blank cells (flags of every neighbour), axes that are and
are not coarsened, rows shorter than a warp; and the FP64 interpolation, which
takes rows, against the oracle."""
import numpy as np
import pytest

import oracle as O
from vfs_poisson import configs as CF

pytestmark = pytest.mark.gpu

BOXES = [(24, 16, 24), (16, 10, 12), (6, 20, 66), (40, 24, 5), (15, 12, 18)]


@pytest.mark.parametrize("blanked", [0.0, 0.02, 0.1])
@pytest.mark.parametrize("dims", BOXES, ids=["x".join(map(str, b)) for b in BOXES])
def test_interpolation_bitexact(cuda_lib, dims, blanked):
    import vfs_poisson as V
    rng = np.random.default_rng(7)
    case = CF.cylinder(*dims, seed=2)
    case.nvert = np.where(rng.random(case.nvert.shape) < blanked, 3.0, 0.0)
    s = V.PoissonSolver(*case.dims, periodic=case.periodic)
    try:
        s.set_grid(case.coor)
        s.set_nvert(case.nvert)
        s.rhs(case.ucont)
        out = [s.solve(rtol=1e-12, max_it=3, smoother=sm) for sm in (3, 4)]
        assert np.isfinite(out[0][0]).all()
        np.testing.assert_array_equal(out[0][0], out[1][0])
        levels = s.mg_levels()
        for li in range(len(levels) - 1):
            cx, cy, cz = levels[li][3:]
            cnx, cny, cnz = levels[li + 1][:3]
            df, dc = (O.dims(a + 2, b + 2, c + 2, case.periodic) for a, b, c in (levels[li][:3], levels[li + 1][:3]))
            nv_f = case.nvert if li == 0 else s.mg_nvert(li)
            xc = np.zeros((cnz + 2, cny + 2, cnx + 2))
            xc[1:-1, 1:-1, 1:-1] = rng.standard_normal((cnz, cny, cnx))
            want = O.interpolation(df, dc, 1 - cx, 1 - cy, 1 - cz, nv_f, s.mg_nvert(li + 1), xc)
            np.testing.assert_array_equal(s.mg_interpolate(li, xc), want, err_msg=str(levels[li]))
    finally:
        s.close()
