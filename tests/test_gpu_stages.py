"""The per-step stages around the solve against the oracle, bit for bit, over
box extents from one cell on, every periodic axis, and blanking values that
are not 0, 1 or 3 (fractions below and above the thresholds, -0, values only
on ghost points), on host and on device arrays."""
import numpy as np
import pytest

import oracle as O
from vfs_poisson import configs as CF

pytestmark = pytest.mark.gpu

BOXES = [((1, 6, 5), (0, 0, 0, 0, 0, 0)), ((7, 1, 9), (0, 0, 0, 1, 0, 1)), ((33, 5, 1), (0, 0, 0, 1, 0, 0)),
         ((127, 3, 4), (1, 0, 0, 0, 0, 1)), ((130, 4, 3), (0, 0, 0, 0, 1, 1)), ((12, 9, 10), (0, 0, 0, 1, 1, 1)),
         ((16, 12, 14), (0, 0, 0, 0, 0, 0))]


def blanking(rng, shape, kind):
    nv = np.zeros(shape)
    if kind == "none":
        return nv
    at = rng.random(shape)
    nv[at < 0.08] = 3.0
    nv[(at >= 0.08) & (at < 0.14)] = 1.0
    if kind == "odd":
        for lo, v in ((0.2, 0.05), (0.24, 0.07), (0.28, 0.5), (0.32, -0.0), (0.36, 1.05), (0.4, -0.2)):
            nv[(at >= lo) & (at < lo + 0.04)] = v
    return nv


def build(dims, periodic, kind, seed=3):
    rng = np.random.default_rng(seed)
    nx, ny, nz = dims
    coor = CF._nodes(nx, ny, nz, lambda e: CF._tanh_stretch(e, 1.5), 0.04)
    case = CF.channel(nx, ny, nz)
    case.coor, case.periodic = coor, periodic
    case.nvert = blanking(rng, case.nvert.shape, kind)  # (ghost points left as drawn)
    case.ucont = rng.uniform(-1, 1, case.ucont.shape)
    return case, rng


@pytest.mark.parametrize("kind", ["none", "plain", "odd"])
@pytest.mark.parametrize("dims,periodic", BOXES, ids=["x".join(map(str, b[0])) for b in BOXES])
def test_pressure_projection_divergence(cuda_lib, dims, periodic, kind):
    import torch
    import vfs_poisson as V
    case, rng = build(dims, periodic, kind)
    d = O.dims_of(case)
    met = O.form_metrics(d, case.coor)
    s = V.PoissonSolver(*case.dims, periodic=periodic)
    try:
        s.set_grid(case.coor)
        s.set_nvert(case.nvert)
        p0, f0 = rng.normal(size=case.nvert.shape), rng.normal(size=case.nvert.shape)
        p_o, f_o = O.update_pressure(d, case.nvert, p0, f0)
        for device in (False, True):
            def arr(a):
                return torch.from_numpy(a.copy()).cuda() if device else a.copy()

            def host(a):
                return a.cpu().numpy() if device else a
            p, f = s.update_pressure(arr(p0), arr(f0))
            np.testing.assert_array_equal(host(p), p_o)
            np.testing.assert_array_equal(host(f), f_o)
            for dt, st, coeff in ((1.0, 1.0, 1.0), (0.01, 1.0, 1.5), (0.37, 2.5, 1e-300), (2.0, 0.5, 3.0)):
                u_o = O.projection(d, case.nvert, f_o, met, case.ucont, dt, st, coeff)
                u = s.projection(arr(case.ucont), dt, st, coeff)
                np.testing.assert_array_equal(host(u), u_o)
            assert s.divergence(u) == O.divergence(d, case.nvert, u_o, met["aj"])
    finally:
        s.close()


@pytest.mark.parametrize("kind", ["none", "plain", "odd"])
@pytest.mark.parametrize("dims,periodic", BOXES, ids=["x".join(map(str, b[0])) for b in BOXES])
def test_volume_flux_and_rhs(cuda_lib, dims, periodic, kind):
    """The sums are reduced in another order than the oracle's: corrected
    fluxes and right-hand side to 1e-12 of the largest value, flux and area
    to 1e-10 (the tolerances of the other VolumeFlux and right-hand-side
    tests)."""
    import torch
    import vfs_poisson as V
    case, rng = build(dims, periodic, kind, seed=5)
    d = O.dims_of(case)
    met = O.form_metrics(d, case.coor)
    lhs = O.poisson_lhs(d, case.nvert, met)
    u0 = case.ucont.copy()
    u0[rng.random(u0.shape) < 0.2] *= 1e-9  # faces VolumeFlux zeroes
    s = V.PoissonSolver(*case.dims, periodic=periodic)
    try:
        s.set_grid(case.coor)
        s.set_nvert(case.nvert)

        def close(u, f, a, u_o, f_o, a_o):
            assert np.abs(u.cpu().numpy() - u_o).max() <= 1e-12
            assert abs(a - a_o) <= 1e-10 * max(abs(a_o), 1e-300)
            assert abs(f - f_o) <= 1e-10 * max(np.abs(u0).sum(), 1.0)
        for flg in range(4):
            u = torch.from_numpy(u0.copy()).cuda()
            f, a = s.volume_flux(u, flg=flg, flux_intp_sum=0.01)
            close(u, f, a, *O.volume_flux(d, case.nvert, met, u0, flg=flg, flux_intp_sum=0.01))
        for immersed in (0, 2, 3, 4):
            u = torch.from_numpy(u0.copy()).cuda()
            f, a = s.volume_flux0(u, immersed)
            close(u, f, a, *O.volume_flux0(d, case.nvert, met, u0, immersed))
        b_o = O.to_da(d, lhs["gid"], O.rhs(d, case.nvert, lhs["gid"], case.ucont, met["aj"], 0.5, 1.0, 1.5))
        for u in (case.ucont, torch.from_numpy(case.ucont).cuda()):
            s.rhs(u, 0.5, 1.0, 1.5)
            assert np.abs(s.rhs_array() - b_o).max() <= 1e-12 * np.abs(b_o).max()
    finally:
        s.close()
