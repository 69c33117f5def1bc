"""Arguments that kernels cannot take where they lie give what the same values give in
arrays of their own."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_stages import build

pytestmark = pytest.mark.gpu

DIMS, PERIODIC = (13, 9, 10), (0, 0, 0, 1, 0, 1)


class _At:
    """FP64 values on the GPU at a byte offset from an aligned address."""

    def __init__(self, a, off):
        import torch
        self.shape, self.off = a.shape, off
        self.buf = torch.zeros(a.nbytes + 16, dtype=torch.uint8, device="cuda")
        self.buf[off:off + a.nbytes] = torch.from_numpy(np.ascontiguousarray(a).view(np.uint8).ravel()).cuda()
        self.ptr = self.buf.data_ptr() + off

    def host(self):
        n = int(np.prod(self.shape)) * 8
        return self.buf[self.off:self.off + n].cpu().numpy().view(np.float64).reshape(self.shape)


def test_arrays_off_the_element_grid(cuda_lib):
    import vfs_poisson as V
    L = V.load()
    case, rng = build(DIMS, PERIODIC, "plain")
    shape = case.nvert.shape
    v0, p0, f0 = rng.normal(size=case.ucont.shape), rng.normal(size=shape), rng.normal(size=shape)
    got = []
    for off in (0, 4):
        s = V.PoissonSolver(*case.dims, periodic=PERIODIC)
        s.set_grid(case.coor)
        a = {k: _At(x, off) for k, x in dict(nv=case.nvert, u=case.ucont, v=v0, p=p0, f=f0, b=p0, x=f0, y=p0, phi=p0 * 0).items()}
        h, o, st, d = s.h, V.default_opts(rtol=1e-6), V.SolveStats(), C.c_double()
        V._check(L.vfs_poisson_set_nvert(h, a["nv"].ptr))
        V._check(L.vfs_poisson_set_nvert(h, a["nv"].ptr))
        V._check(L.vfs_poisson_volume_flux(h, a["u"].ptr, 1, 0., None, None))
        V._check(L.vfs_poisson_volume_flux0(h, a["u"].ptr, 3, None, None))
        V._check(L.vfs_poisson_rhs(h, a["u"].ptr, 1., 1., 1.))
        V._check(L.vfs_poisson_get_rhs(h, a["b"].ptr))
        V._check(L.vfs_poisson_apply(h, a["x"].ptr, a["y"].ptr))
        V._check(L.vfs_poisson_solve(h, a["phi"].ptr, C.byref(o), C.byref(st)))
        V._check(L.vfs_poisson_update_pressure(h, a["p"].ptr, a["f"].ptr))
        V._check(L.vfs_poisson_projection(h, a["u"].ptr, 0.5, 1., 1.5))
        V._check(L.vfs_poisson_divergence(h, a["u"].ptr, C.byref(d)))
        V._check(L.vfs_poisson_contra2cart(h, a["u"].ptr, a["v"].ptr, 1))
        V._check(L.vfs_poisson_ib_bc(h, 1, None, a["v"].ptr, a["u"].ptr))
        got.append({k: x.host() for k, x in a.items()} | {"div": d.value})
        s.close()
    for k in got[0]:
        np.testing.assert_array_equal(got[0][k], got[1][k], err_msg=k)


@pytest.mark.parametrize("shift", [0, 1, 300])
def test_overlapping_arrays(cuda_lib, shift):
    """Arrays that share memory, wholly or from an element on: every value from the
    arrays as they were passed, results written in the order of the arguments."""
    import torch
    import vfs_poisson as V
    from vfs_poisson import configs as CF
    L = V.load()
    case, rng = build(DIMS, PERIODIC, "plain")
    n3, n1 = case.ucont.size, case.nvert.size
    surf = CF.rod_surface((0.5, 0.2, 0.5), (0.0, 1.0, 0.0), 0.5, 0.2, 16, 6)
    base = rng.normal(size=2 * n3 + n1)
    calls = {  # offsets of the arrays in one buffer, in the order of the call's downloads
        "contra2cart": (lambda h, c, u: L.vfs_poisson_contra2cart(h, u, c, 1), (shift, 0), (n3, 0)),
        "ib_bc": (lambda h, c, u: L.vfs_poisson_ib_bc(h, 1, None, c, u), (shift, 0), (n3, n3)),
        "ibm_interpolate": (lambda h, c, p, u: L.vfs_poisson_ibm_interpolate(h, 0, None, 1, None, c, p, u),
                            (shift, 2 * n3, 0), (n3, n1, n3)),
        "update_pressure": (lambda h, p, f: L.vfs_poisson_update_pressure(h, p, f), (shift, 0), (n1, n1)),
    }
    s = V.PoissonSolver(*case.dims, periodic=PERIODIC)
    try:
        s.set_grid(case.coor)
        nv, _, nodes = s.ibm_search_nodes(surf)
        assert nodes > 0
        s.set_nvert(nv)
        for name, (call, off, size) in calls.items():
            length = {"update_pressure": n1}.get(name, n3)
            # each array alone, then the writes in order
            own = [torch.from_numpy(base[o:o + (n1 if o == 2 * n3 else length)].copy()).cuda() for o in off]
            V._check(call(s.h, *[a.data_ptr() for a in own]))
            want = base.copy()
            for o, a, k in zip(off, own, size):
                want[o:o + k] = a.cpu().numpy()[:k]
            buf = torch.from_numpy(base.copy()).cuda()
            V._check(call(s.h, *[buf.data_ptr() + 8 * o for o in off]))
            np.testing.assert_array_equal(buf.cpu().numpy(), want, err_msg=name)
    finally:
        s.close()
