"""The rows an incremental refill finds (changed points as bits in words of 32
along i) against a fresh handle, bit for bit: rows of less than one word, of
exactly one and across word borders, changes at single points, on every side
and next to each periodic seam, on host and on device masks."""
import numpy as np
import pytest

from vfs_poisson import configs as CF

pytestmark = pytest.mark.gpu

BOXES = [((14, 12, 10), (1, 0, 0, 0, 0, 1)), ((30, 8, 12), (0, 0, 0, 0, 1, 0)), ((31, 10, 8), (0, 0, 0, 1, 0, 0)),
         ((64, 9, 10), (0, 0, 0, 1, 1, 1)), ((95, 8, 8), (0, 0, 0, 0, 0, 0))]


@pytest.mark.parametrize("dims,periodic", BOXES, ids=["x".join(map(str, b[0])) for b in BOXES])
def test_changed_rows(cuda_lib, dims, periodic):
    import torch
    import vfs_poisson as V
    rng = np.random.default_rng(8)
    case = CF.cylinder(*dims, seed=3)
    case.set_periodic(periodic)
    moved = V.PoissonSolver(*case.dims, periodic=periodic)
    try:
        moved.set_grid(case.coor)
        nv = np.zeros_like(case.nvert)
        moved.set_nvert(nv)
        for step in range(8):
            nx, ny, nz = dims
            pts = [(rng.integers(1, nx + 1), rng.integers(1, ny + 1), rng.integers(1, nz + 1)) for _ in range(3)]
            pts += [((1, nx, 31, 32, 33)[step % 5], (1, ny)[step % 2], (1, nz)[step // 2 % 2])]
            for i, j, k in pts:
                if i <= nx:
                    nv[k, j, i] = rng.choice([0.0, 1.0, 3.0])
            mask = CF.sync_periodic_ghosts(nv, periodic)
            moved.set_nvert(torch.from_numpy(mask).cuda() if step % 2 else mask)
            fresh = V.PoissonSolver(*case.dims, periodic=periodic)
            try:
                fresh.set_grid(case.coor)
                fresh.set_nvert(mask)
                for a, b in zip(moved.operator(), fresh.operator()):
                    np.testing.assert_array_equal(a, b)
                np.testing.assert_array_equal(moved.operator32(), fresh.operator32())
                (na, ga), (nb, gb) = moved.numbering(), fresh.numbering()
                assert na == nb
                np.testing.assert_array_equal(ga, gb)
                out = []
                for s in (moved, fresh):
                    s.rhs(case.ucont)
                    out.append((s.rhs_array(), s.mg_vcycle(case.ucont[..., 0].copy())))
                for a, b in zip(*out):
                    np.testing.assert_array_equal(a, b)
            finally:
                fresh.close()
    finally:
        moved.close()
