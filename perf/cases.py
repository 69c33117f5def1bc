"""Performance cases: the work a user of the library has it do.

A fractional-step loop calls, per step, VolumeFlux and the right-hand side, the pressure solve, UpdatePressure,
Projection and Divergence, Contra2Cart with the immersed-boundary interpolation, and, when bodies move, the surface
search and the refill of the operator; beside it the learned-guess network trains on crops.  Each kind below is one
of these stages (or a whole step) through the public Python binding on device arrays.  The grids are those of
vfs_poisson.configs (channel, cylinder, towers, rotor, farm) at their own sizes, smaller ones and ragged ones.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "vfs-wind_gb300"))
import vfs_poisson as V  # noqa: E402
from vfs_poisson import configs as CF  # noqa: E402

DEV = "cuda" if torch.cuda.is_available() else "cpu"
F64 = torch.float64
TP = 2.0 * math.pi

PERIODIC = {"channel": (0, 0, 0, 1, 0, 1), "cylinder": (0, 0, 0, 1, 0, 0), "rotor": (0, 0, 0, 1, 0, 0),
            "towers": (0, 0, 0, 1, 0, 1), "farm": (0, 0, 0, 1, 0, 1)}


def _case(name, kind, grid, nx, ny, nz, **kw):
    return dict(name=name, kind=kind, grid=grid, nx=nx, ny=ny, nz=nz, **kw)


def listed():
    return [
        # the smallest solve in use (a coarse test grid with a body): launches and host round trips count
        _case("solve_smallest", "solve", "cylinder", 24, 16, 24, precision=0, rtol=1e-8, warm=False),
        # the channel at its own size: a stretched rectilinear grid without a body, first step from a zero guess
        _case("solve_channel", "solve", "channel", 64, 64, 64, precision=0, rtol=1e-8, warm=False),
        # the curvilinear cylinder at its own size, a step restarted from the previous step's phi
        _case("solve_cylinder", "solve", "cylinder", 128, 96, 128, precision=0, rtol=1e-8, warm=True),
        # all-FP64 V-cycle to a tight tolerance on a ragged size (odd factors 9, 5, 7 are not coarsened)
        _case("solve_fp64_ragged", "solve", "towers", 72, 40, 56, precision=1, rtol=1e-10, warm=False),
        # the towers sequence at its own size: right-hand side, guess from 8 stored solutions, solve, store
        _case("history_towers", "history", "towers", 256, 192, 256, keep=8),
        # a whole step of the turning rotor at its own size, from the surface search to Contra2Cart
        _case("step_rotor", "moving", "rotor", 192, 128, 192, rtol=1e-8),
        # the mask update of a wind farm (4 towers with rotors, 16 bodies): surface search and operator refill
        _case("mask_farm", "mask", "farm", 384, 192, 384, ax=2, az=2),
        # VolumeFlux and right-hand side at the towers' size, second-order time coefficient
        _case("rhs_towers", "rhs", "towers", 256, 192, 256, dt=0.01, coeff=1.5),
        # UpdatePressure, Projection and Divergence at the towers' size
        _case("project_towers", "project", "towers", 256, 192, 256, dt=0.01, coeff=1.5),
        # the same on a small ragged box: call latency
        _case("project_small", "project", "cylinder", 40, 33, 48, dt=1.0, coeff=1.0),
        # Contra2Cart, the IB interpolation of three rods and IB_BC at the rotor's size
        _case("velocity_rotor", "velocity", "rotor", 192, 128, 192),
        # one training step (gradient and Adam) of the learned-guess network on the crop size it trains on
        _case("unet_train", "unet", "", 64, 64, 64, lr=1e-3),
    ]


def _odd(rng, lo, hi):
    """An odd box extent between lo and hi, spread over its logarithm."""
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi)))) | 1


def _pow2(rng, lo, hi, parts=(1, 3, 5)):
    """An extent m 2^p (the hierarchy coarsens it to a few cells) between lo and hi."""
    all_ = [m << p for m in parts for p in range(2, 10) if lo <= m << p <= hi]
    t = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(all_, key=lambda v: abs(math.log(v / t)))


def draw(rng):
    kind = rng.choice(["solve", "solve", "history", "moving", "mask", "rhs", "project", "velocity", "unet"])
    if kind == "unet":
        n = [4 * rng.randrange(4, 17) for _ in range(3)]
        return dict(kind=kind, grid="", nx=n[0], ny=n[1], nz=n[2], lr=rng.choice([1e-3, 2e-4]))
    hi = {"solve": 128, "history": 192, "moving": 160, "mask": 256, "rhs": 256, "project": 256, "velocity": 192}[kind]
    odd = kind in ("solve", "rhs", "project", "velocity") and rng.random() < 0.4
    # (an odd extent stays whole on the coarsest level, which the library limits to 1024 cells)
    n = [_pow2(rng, 24 if kind in ("solve", "rhs", "project") else 64, hi if q != 1 else 3 * hi // 4,
               (1, 3) if odd else (1, 3, 5)) for q in range(3)]
    if odd:
        n[rng.randrange(3)] = _odd(rng, 24 if kind != "velocity" else 48, 63)
    c = dict(kind=kind, grid="", nx=n[0], ny=n[1], nz=n[2])
    if kind == "solve":
        c.update(grid=rng.choice(["channel", "cylinder", "towers"]), precision=rng.choice([0, 0, 1]),
                 rtol=rng.choice([1e-8, 1e-10]), warm=rng.choice([False, True]))
    elif kind == "history":
        c.update(grid="towers", keep=rng.randrange(2, 9))
    elif kind == "moving":
        c.update(grid="rotor", rtol=1e-8)
    elif kind == "mask":
        c.update(grid="farm", ax=rng.randrange(1, 3), az=rng.randrange(1, 3))
    elif kind == "velocity":
        c.update(grid="rotor")
    else:
        c.update(grid=rng.choice(["channel", "cylinder", "towers"]), dt=rng.choice([1.0, 0.01, 2.5e-3]),
                 coeff=rng.choice([1.0, 1.5]))
    return c


# ---- inputs -------------------------------------------------------------------------------------------------

def _coor(c):
    """Node coordinates [mz][my][mx][3] of the case's grid (vfs_poisson.configs' formulas, on the device)."""
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    et = np.arange(ny + 1) / ny
    amp, phys = {"channel": (0.0, 0), "cylinder": (0.05, 0), "rotor": (0.05, 0), "towers": (0.02, 1),
                 "farm": (0.02, 1)}[c["grid"]]
    if c["grid"] in ("towers", "farm"):  # the wall stretching's total ratio does not depend on the size
        ratio = (1.03 ** 192 if c["grid"] == "towers" else 1.02 ** 256) ** (1.0 / ny)
        ys = (ratio ** np.arange(ny + 1.0) - 1.0) / (ratio ** ny - 1.0)
    else:
        beta = 1.5 if c["grid"] == "channel" else 2.0
        ys = 0.5 * (1.0 + np.tanh(beta * (2.0 * et - 1.0)) / np.tanh(beta))
    X = torch.arange(nx + 1, dtype=F64, device=DEV)[None, None, :] / nx
    Z = torch.arange(nz + 1, dtype=F64, device=DEV)[:, None, None] / nz
    Y = torch.from_numpy(ys).to(DEV)[None, :, None]
    E = torch.from_numpy(ys if phys else et).to(DEV)[None, :, None]
    co = torch.zeros((nz + 2, ny + 2, nx + 2, 3), dtype=F64, device=DEV)
    n = co[: nz + 1, : ny + 1, : nx + 1]
    n[..., 0] = X + amp * torch.sin(TP * E) * torch.sin(TP * Z)
    n[..., 1] = Y + amp * torch.sin(TP * Z) * torch.sin(TP * X)
    n[..., 2] = Z + amp * torch.sin(TP * X) * torch.sin(TP * E)
    return co


def _centres(co):
    c = co[:-1, :-1, :-1]
    s = c[1:] + c[:-1]
    s = s[:, 1:] + s[:, :-1]
    return 0.125 * (s[:, :, 1:] + s[:, :, :-1])


def _ghosts(c, a):
    """Periodic ghost layers from their partners (in place, DA layout)."""
    per = [PERIODIC[c["grid"]][q] or PERIODIC[c["grid"]][q + 3] for q in range(3)]
    if per[0]:
        a[:, :, 0] = a[:, :, -2]
        a[:, :, -1] = a[:, :, 1]
    if per[1]:
        a[:, 0] = a[:, -2]
        a[:, -1] = a[:, 1]
    if per[2]:
        a[0] = a[-2]
        a[-1] = a[1]
    return a


def _static_mask(c, co):
    """nvert of the static bodies (cylinder, towers): 3 inside, 1 in the cells around, 0 fluid."""
    cc = _centres(co)
    ins = torch.zeros(cc.shape[:3], dtype=torch.bool, device=DEV)
    if c["grid"] == "cylinder":
        ins = (cc[..., 0] - 0.5) ** 2 + (cc[..., 2] - 0.5) ** 2 < 0.01
    elif c["grid"] == "towers":
        r = max(0.02, 1.2 / min(c["nx"], c["nz"]))  # at least a few cells across on small boxes
        for x0 in (0.25, 0.5, 0.75):
            for z0 in (0.35, 0.65):
                ins |= (cc[..., 0] - x0) ** 2 + (cc[..., 2] - z0) ** 2 < r * r
    big = torch.zeros((1, 1) + tuple(v + 2 for v in ins.shape), device=DEV)
    big[0, 0, 1:-1, 1:-1, 1:-1] = ins
    near = torch.nn.functional.max_pool3d(big, 3, 1, 1)[0, 0] > 0
    nv = near.to(F64)
    nv[1:-1, 1:-1, 1:-1][ins] = 3.0
    nv[0] = nv[-1] = 0.0
    nv[:, 0] = nv[:, -1] = 0.0
    nv[:, :, 0] = nv[:, :, -1] = 0.0
    return _ghosts(c, nv)


def _modes(rng, n=8, kmax=8):
    out = []
    while len(out) < n:
        kv = rng.integers(-kmax, kmax + 1, size=3)
        kn = math.sqrt(float((kv ** 2).sum()))
        if 1 <= kn <= kmax:
            out.append((kv, rng.normal() / kn, rng.uniform(0, TP, size=3)))
    return out


def _field(c, modes, step=0.0, off=(0.0, 0.0, 0.0)):
    """Fourier modes at (cell or face) positions in computational space, moved `step` half cells in x."""
    n = (c["nx"], c["ny"], c["nz"])
    f = [(torch.arange(n[q] + 2, dtype=F64, device=DEV) - off[q]) / n[q] for q in range(3)]
    acc = torch.zeros((n[2] + 2, n[1] + 2, n[0] + 2), dtype=F64, device=DEV)
    for kv, a, ph in modes:
        x = torch.cos(TP * int(kv[0]) * (f[0] - 0.5 * step / n[0]) + ph[0])
        y = torch.cos(TP * int(kv[1]) * f[1] + ph[1]) * (2.0 * a)
        z = torch.cos(TP * int(kv[2]) * f[2] + ph[2])
        acc += (z[:, None] * y[None, :])[:, :, None] * x
    return acc


class _Flux:
    """Contravariant face fluxes: Fourier modes and noise (the channel: noise alone)."""

    def __init__(self, c, seed):
        rng = np.random.default_rng(seed)
        self.c = c
        self.modes = [_modes(rng) for _ in range(3)]
        g = torch.Generator(DEV)
        g.manual_seed(seed)
        shape = (c["nz"] + 2, c["ny"] + 2, c["nx"] + 2, 3)
        self.noise = torch.rand(shape, dtype=F64, device=DEV, generator=g).mul_(2.0).sub_(1.0)

    def at(self, step=0):
        if self.c["grid"] == "channel":
            return self.noise.clone()
        u = 0.1 * self.noise
        for q in range(3):
            u[..., q] += _field(self.c, self.modes[q], step, [0.0 if q == e else 0.5 for e in range(3)])
        return u


def _mask_faces(u, nv):
    """Zero every face flux next to a blanked cell."""
    b = nv > 0.1
    u[:, :, :-1, 0].masked_fill_(b[:, :, :-1] | b[:, :, 1:], 0.0)
    u[:, :-1, :, 1].masked_fill_(b[:, :-1] | b[:, 1:], 0.0)
    u[:-1, :, :, 2].masked_fill_(b[:-1] | b[1:], 0.0)
    return u


def _rotor(c, step):
    h = 1.0 / c["nz"]
    return CF.rotor_surfaces(angle_deg=2.0 * step, rods=3, radius=3 * h, length=30 * h, hub=0.0, n_theta=32, n_len=30)


def _farm(c, step):
    out = []
    for x0 in (0.25, 0.75)[: c["ax"]]:
        for z0 in (0.3, 0.7)[: c["az"]]:
            out.append(CF.rod_surface((x0, -0.05, z0), (0.0, 1.0, 0.0), 0.55, 0.02, 32, 4))
            out += CF.rotor_surfaces(centre=(x0, 0.5, z0), angle_deg=2.0 * step, rods=3, radius=3.0 / c["nx"],
                                     length=0.08, hub=0.0, n_theta=16, n_len=12)
    return out


class _State:
    pass


def _search(s, bodies, nodes=False):
    for ibi, surf in enumerate(bodies):
        if nodes:
            s.h.ibm_search_nodes(surf, nvert=s.nv, ibi=ibi)
        else:
            s.h.ibm_search(surf, nvert=s.nv, ibi=ibi)
    _ghosts(s.c, s.nv)
    s.h.set_nvert(s.nv)


def prepare(case, seed):
    c = dict(case)
    s = _State()
    s.c, s.kind, s.t = c, c["kind"], 0
    if s.kind == "unet":
        return _prepare_unet(s, seed)
    s.h = V.PoissonSolver(c["nx"] + 2, c["ny"] + 2, c["nz"] + 2, periodic=PERIODIC[c["grid"]])
    co = _coor(c)
    s.h.set_grid(co)
    flux = _Flux(c, seed)
    rng = np.random.default_rng(seed + 1)
    if s.kind in ("solve", "history", "rhs", "project"):
        s.nv = _static_mask(c, co)
        s.h.set_nvert(s.nv)
    else:
        s.nv = torch.zeros(co.shape[:3], dtype=F64, device=DEV)
        s.bodies = [(_rotor if c["grid"] == "rotor" else _farm)(c, step + seed % 90) for step in range(8)]
        _search(s, s.bodies[7], nodes=s.kind == "velocity")
    s.phi = torch.zeros_like(s.nv)
    if s.kind == "solve":
        s.opts = V.default_opts(rtol=c["rtol"], precision=c["precision"], warm_start=1 if c["warm"] else 0)
        s.u = _mask_faces(flux.at(1), s.nv)
        s.prev = None
        if c["warm"]:
            s.prev = torch.zeros_like(s.nv)
            s.h.solver_hypre(_mask_faces(flux.at(0), s.nv), phi=s.prev, rtol=c["rtol"], precision=c["precision"])
    elif s.kind == "history":
        s.h.set_history(c["keep"])
        s.us = [_mask_faces(flux.at(t), s.nv) for t in range(16)]
        s.cold, s.warm = V.default_opts(), V.default_opts(warm_start=2)
        for t in range(c["keep"]):
            _history_step(s, t)
        s.t = c["keep"]
    elif s.kind == "moving":
        s.us = [flux.at(t) for t in range(8)]
        s.opts = V.default_opts(rtol=c["rtol"], warm_start=1)
        s.p, s.ucat = torch.zeros_like(s.nv), torch.zeros_like(s.us[0])
        s.u, s.prev = torch.empty_like(s.us[0]), torch.zeros_like(s.nv)
        s.h.solver_hypre(_mask_faces(flux.at(7), s.nv), phi=s.prev, rtol=c["rtol"])
    elif s.kind == "mask":
        s.x = _field(c, _modes(rng))
        s.y = torch.empty_like(s.x)
    elif s.kind == "rhs":
        s.u = flux.at()
        s.b = torch.empty_like(s.nv)
    elif s.kind == "project":
        s.u = flux.at()
        phi = _field(c, _modes(rng), 0.0, (0.5, 0.5, 0.5)) * 0.01
        s.phi = _ghosts(c, phi.masked_fill_(s.nv > 0.1, 0.0))
        s.p = _ghosts(c, _field(c, _modes(rng), 0.0, (0.5, 0.5, 0.5)))
    elif s.kind == "velocity":
        s.u = flux.at()
        s.p = _field(c, _modes(rng), 0.0, (0.5, 0.5, 0.5))
        s.ucat = torch.zeros_like(s.u)
        s.us = [torch.from_numpy(np.cross([0.0, 0.0, 0.5], b[0] - 0.5)).to(DEV) for b in s.bodies[7]]
    return s


def _history_step(s, t):
    s.h.rhs(s.us[t % len(s.us)])
    if t:
        s.h.history_guess()
    s.h.solve(s.phi, opts=s.warm if t else s.cold)


def _prepare_unet(s, seed):
    c = s.c
    s.net = V.UNet(seed=seed % 100000)
    g = torch.Generator(DEV)
    g.manual_seed(seed)
    shape = (c["nz"], c["ny"], c["nx"])
    f = dict(nx=c["nx"] - 2, ny=c["ny"] - 2, nz=c["nz"] - 2)
    rng = np.random.default_rng(seed)
    s.feat = torch.stack([_field(f, _modes(rng)).float() for _ in range(3)]
                         + [(torch.rand(shape, device=DEV, generator=g) > 0.03).float()]).contiguous()
    s.feat[:3] /= s.feat[:3].square().mean(dim=(1, 2, 3), keepdim=True).sqrt()
    s.wt = s.feat[3].clone()
    s.tgt = (_field(f, _modes(rng)).float() * s.wt).contiguous()
    s.batch = s.net.batch(s.feat, s.tgt, s.wt)
    s.grad = torch.empty(s.net.num_params, device=DEV)
    return s


def run(s):
    c, h = s.c, getattr(s, "h", None)
    if s.kind == "solve":
        if s.prev is not None:
            s.phi.copy_(s.prev)
        h.solver_hypre(s.u, phi=s.phi, opts=s.opts)
        return {"phi": s.phi}
    if s.kind == "history":
        _history_step(s, s.t)
        s.t += 1
        return {"phi": s.phi}
    if s.kind == "moving":
        t = s.t % 8
        s.t += 1
        _search(s, s.bodies[t])
        s.u.copy_(s.us[t])
        h.volume_flux(s.u)
        h.rhs(s.u)
        s.phi.copy_(s.prev)
        h.solve(s.phi, opts=s.opts)
        h.update_pressure(s.p, s.phi)
        h.projection(s.u)
        div = h.divergence(s.u)
        h.contra2cart(s.u, s.ucat)
        return {"nvert": s.nv, "phi": s.phi, "p": s.p, "ucont": s.u, "ucat": s.ucat, "finite": math.isfinite(div)}
    if s.kind == "mask":
        t = s.t % 8
        s.t += 1
        _search(s, s.bodies[t])
        # the operator the refill left, as its product with a vector (C entry point: device arrays)
        V._check(V.load().vfs_poisson_apply(h.h, s.x.data_ptr(), s.y.data_ptr()))
        return {"nvert": s.nv, "y": s.y}
    if s.kind == "rhs":
        # (the corrected flux itself is rounding noise about 0)
        _, area = h.volume_flux(s.u)
        h.rhs(s.u, dt=c["dt"], coeff=c["coeff"])
        V._check(V.load().vfs_poisson_get_rhs(h.h, s.b.data_ptr()))
        return {"ucont": s.u, "area": area, "b": s.b}
    if s.kind == "project":
        h.update_pressure(s.p, s.phi)
        h.projection(s.u, dt=c["dt"], coeff=c["coeff"])
        return {"p": s.p, "phi": s.phi, "ucont": s.u, "maxdiv": h.divergence(s.u)}
    if s.kind == "velocity":
        h.contra2cart(s.u, s.ucat)
        for ibi, us in enumerate(s.us):
            V._check(V.load().vfs_poisson_ibm_interpolate(h.h, ibi, us.data_ptr(), 1, None, s.ucat.data_ptr(),
                                                          s.p.data_ptr(), s.u.data_ptr()))
        h.ib_bc(s.ucat, s.u)
        return {"ucat": s.ucat, "p": s.p, "ucont": s.u}
    loss = s.net.gradient(s.batch, s.grad)
    s.net.adam(c["lr"])
    return {"loss": loss, "grad": s.grad}


def work(case):
    """Bytes: inputs read once and outputs written once (per cell; FP64 words unless said otherwise)."""
    n = float(case["nx"] * case["ny"] * case["nz"])
    kind = case["kind"]
    if kind == "unet":
        ch = [(16, 16, 1), (16, 16, 1), (16, 32, 8), (32, 32, 8), (32, 64, 64), (64, 64, 64), (96, 32, 8), (32, 32, 8),
              (48, 16, 1), (16, 16, 1)]
        f = sum(2.0 * 27 * a * b / d for a, b, d in ch) * n  # forward; data and weight gradients the same each
        return {"bytes": n * 24.0 + 3 * 4.0 * 360e3, "flops": 3.0 * f}
    # the operator is known by its nine face coefficients (72 bytes per cell) and the blanking
    op, mask, vec, cmp_ = 72.0, 8.0, 8.0, 24.0
    per = {"solve": op + mask + cmp_ + vec, "history": op + mask + cmp_ + vec * (2 + 2 * case.get("keep", 0)),
           "mask": cmp_ + mask + 2 * vec + op, "rhs": mask + 2 * cmp_ + 2 * vec,
           "project": mask + 2 * vec + 2 * vec + 2 * cmp_ + op + vec,
           "velocity": mask + 3 * cmp_ + 4 * cmp_ + 2 * vec,
           "moving": cmp_ + mask + op + 2 * cmp_ + 4 * vec + 3 * cmp_ + 3 * cmp_}[kind]
    flops = {"solve": 60.0, "history": 60.0 + 4 * case.get("keep", 0), "mask": 40.0, "rhs": 15.0, "project": 80.0,
             "velocity": 150.0, "moving": 300.0}[kind]
    return {"bytes": n * per, "flops": n * flops}


# ---- what the calls return, in 64 bits and plain torch ------------------------------------------------------

def _sh(a, q, d):
    """a at index + d along axis q (0: i, 1: j, 2: k) of a DA array (the ends wrap and are not used)."""
    return torch.roll(a, -d, 2 - q)


class _Exact:
    """Metrics, face fluxes of grad phi and divergence on the DA grid."""

    def __init__(self, c, nv):
        self.c, self.nv = c, nv
        self.m = [c["nx"] + 2, c["ny"] + 2, c["nz"] + 2]
        self.per = [PERIODIC[c["grid"]][q] or PERIODIC[c["grid"]][q + 3] for q in range(3)]
        co = _coor(c)
        d = []
        for q in range(3):
            hi = co - _sh4(co, q)
            e, f = [r for r in range(3) if r != q]
            hi = hi + _sh4(hi, e)
            d.append(0.25 * (hi + _sh4(hi, f)))
        met = [torch.linalg.cross(d[1], d[2]), torch.linalg.cross(d[2], d[0]), torch.linalg.cross(d[0], d[1])]
        aj = 1.0 / (d[0] * met[0]).sum(-1)
        self.cell, self.aj = met, aj
        for a in met + [aj]:
            for q in range(3):
                ax = 2 - q
                a.select(ax, 0).copy_(a.select(ax, 1))
                a.select(ax, -1).copy_(a.select(ax, -2))
            _ghosts(c, a)
        self.face, self.faj = [], []
        for q in range(3):
            fm = [0.5 * (a + torch.roll(a, -1, 2 - q)) for a in met]
            self.face.append([(fm[e] * fm[q]).sum(-1) for e in range(3)])
            self.faj.append(2.0 / (1.0 / aj + 1.0 / _sh(aj, q, 1)))
        idx = [torch.arange(self.m[q], device=DEV).view([-1 if 2 - q == e else 1 for e in range(3)]) for q in range(3)]
        self.idx = idx
        self.inner = torch.ones_like(nv, dtype=torch.bool)
        for q in range(3):
            self.inner &= (idx[q] >= 1) & (idx[q] <= self.m[q] - 2)
        self.fluid = self.inner & (nv < 0.1)
        thr = 0.1
        self.rule = {}
        for q in range(3):
            N = nv + _sh(nv, q, 1)
            for t in range(3):
                if t == q:
                    continue
                Np, Nm = _sh(N, t, 1), _sh(N, t, -1)
                top = (idx[t] == self.m[t] - 2) & (not self.per[t])
                bot = (idx[t] == 1) & (not self.per[t])
                c1, c2 = top | (Np > thr), bot | (Nm > thr)
                self.rule[q, t] = (c1 & (Nm < thr) & (idx[t] != 1), ~c1 & c2 & (Np < thr), ~c1 & ~c2)
            self.rule[q] = self.inner & (N < thr) & ((idx[q] < self.m[q] - 2) | bool(self.per[q]))

    def flux(self, phi):
        """Metric-weighted grad phi at the i, j, k faces of each cell (phi with periodic ghosts, leading batch ok)."""
        out = []
        for q in range(3):
            f = (_sh(phi, q, 1) - phi) * self.face[q][q]
            S = phi + _sh(phi, q, 1)
            for t in range(3):
                if t == q:
                    continue
                lo, up, ce = self.rule[q, t]
                Sp, Sm = _sh(S, t, 1), _sh(S, t, -1)
                z = torch.zeros((), dtype=F64, device=DEV)
                dd = torch.where(lo, 0.5 * (S - Sm), torch.where(up, 0.5 * (Sp - S),
                                                                 torch.where(ce, 0.25 * (Sp - Sm), z)))
                f = f + dd * self.face[q][t]
            out.append(torch.where(self.rule[q], f * self.faj[q], torch.zeros((), dtype=F64, device=DEV)))
        return out

    def wrap_faces(self, u):
        """Each periodic direction's own component on its ghost layers (u: three DA arrays)."""
        for q in range(3):
            if self.per[q]:
                g = _ghosts(self.c, u[q].clone())
                u[q].select(2 - q, 0).copy_(g.select(2 - q, 0))
                u[q].select(2 - q, -1).copy_(g.select(2 - q, -1))
        return u

    def div(self, u):
        """Net outflow of each interior cell."""
        u = self.wrap_faces([x.clone() for x in u])
        return sum(u[q] - _sh(u[q], q, -1) for q in range(3))

    def rhs(self, u, dt, coeff):
        b = torch.where(self.fluid, self.div([u[..., q] for q in range(3)]) * (coeff / dt), 0.0)
        aj = torch.where(self.fluid, self.aj, 0.0)
        return b - b.sum() / aj.sum() * aj

    def solve(self, u):
        """phi by a dense solve over the fluid cells (one connected region, constants removed)."""
        b = self.rhs(u, 1.0, 1.0)
        cells = self.fluid.reshape(-1).nonzero()[:, 0]
        n = cells.numel()
        A = torch.empty((n, n), dtype=F64, device=DEV)
        # cells three apart in every direction share no stencil: one colour of 27 per product (more at wraps)
        pos = torch.stack([cells % self.m[0], (cells // self.m[0]) % self.m[1], cells // (self.m[0] * self.m[1])])
        A.zero_()
        number = torch.full((self.nv.numel(),), -1, dtype=torch.int64, device=DEV)
        number[cells] = torch.arange(n, device=DEV)
        number = _ghosts(self.c, number.view(self.nv.shape)).reshape(-1)
        col = [torch.where((pos[q] > self.m[q] - 2 - (self.m[q] - 2) % 3) & bool(self.per[q]), pos[q] % 3 + 3, pos[q] % 3)
               for q in range(3)]
        colour = (col[2] * 6 + col[1]) * 6 + col[0]
        for k in colour.unique().tolist():
            mine = cells[colour == k]
            phi = torch.zeros(self.nv.numel(), dtype=F64, device=DEV)
            phi[mine] = 1.0
            who = torch.full((self.nv.numel(),), -1, dtype=torch.int64, device=DEV)
            who[mine] = number[mine]
            who = _ghosts(self.c, who.view(self.nv.shape))
            r = self.div(self.flux(_ghosts(self.c, phi.view(self.nv.shape))))
            near = who.clone()  # the coloured cell within one point of each cell
            for q in range(3):
                near = torch.maximum(near, torch.maximum(_sh(near, q, 1), _sh(near, q, -1)))
            at = (self.fluid & (near >= 0)).reshape(-1).nonzero()[:, 0]
            A[number[at], near.reshape(-1)[at]] = r.reshape(-1)[at]
        scale = A.diagonal().abs().mean() / n
        x = torch.linalg.solve(A - scale, b.reshape(-1)[cells])
        phi = torch.zeros(self.nv.numel(), dtype=F64, device=DEV)
        phi[cells] = x - x.mean()
        return _ghosts(self.c, phi.view(self.nv.shape))


def _sh4(a, q):
    """a at index - 1 along axis q of a Cmpnts DA array."""
    return torch.roll(a, 1, 2 - q)


def _exact_unet(case, seed):
    """The loss and the gradient of the training step's forward pass, unrounded."""
    s = _prepare_unet(_fresh(case), seed)
    p = torch.from_numpy(s.net.get_params()).to(DEV).to(F64)
    ch = [(16, 16), (16, 16), (16, 32), (32, 32), (32, 64), (64, 64), (96, 32), (32, 32), (48, 16), (16, 16)]
    p.requires_grad_(True)
    off, ws = 0, []
    for a, b in ch:
        w = p[off:off + 27 * a * b].view(3, 3, 3, a, b).permute(4, 3, 0, 1, 2)
        off += 27 * a * b
        ws.append((w, p[off:off + b]))
        off += b
    F = torch.nn.functional

    def conv(i, x):
        w, b = ws[i]
        xp = F.pad(x, (1, 1, 1, 1, 1, 1))
        y = b.view(1, -1, 1, 1, 1)
        n = x.shape[2:]
        for t in range(27):
            dz, dy, dx = t // 9, t // 3 % 3, t % 3
            y = y + torch.einsum("oc,bczyx->bozyx", w[:, :, dz, dy, dx],
                                 xp[:, :, dz:dz + n[0], dy:dy + n[1], dx:dx + n[2]])
        return F.relu(y)

    def up(x):
        return x.repeat_interleave(2, 2).repeat_interleave(2, 3).repeat_interleave(2, 4)

    x = torch.zeros((1, 16) + tuple(s.feat.shape[1:]), dtype=F64, device=DEV)
    x[0, :4] = s.feat.to(F64)
    e0 = conv(1, conv(0, x))
    e1 = conv(3, conv(2, F.avg_pool3d(e0, 2)))
    e2 = conv(5, conv(4, F.avg_pool3d(e1, 2)))
    d1 = conv(7, conv(6, torch.cat([up(e2), e1], 1)))
    d0 = conv(9, conv(8, torch.cat([up(d1), e0], 1)))
    out = (d0[0] * p[off:off + 16].view(16, 1, 1, 1)).sum(0) + p[off + 16]
    wt = s.wt.to(F64)
    loss = (wt * (out - s.tgt.to(F64)) ** 2).sum() / wt.sum()
    g, = torch.autograd.grad(loss, p)
    return {"loss": float(loss), "grad": g}


def _fresh(case):
    s = _State()
    s.c, s.kind, s.t = dict(case), case["kind"], 0
    return s


def exact(case, seed):
    c, kind = case, case["kind"]
    n = c["nx"] * c["ny"] * c["nz"]
    if kind == "unet":
        return _exact_unet(case, seed) if n <= 64 ** 3 else None
    if kind not in ("solve", "rhs", "project") or (kind == "solve" and (n > 10000 or c["grid"] == "towers")):
        return None  # an independent solve (or ray cast) takes longer than the limit
    co = _coor(c)
    nv = _static_mask(c, co)
    X = _Exact(c, nv)
    flux = _Flux(c, seed)
    if kind == "solve":
        return {"phi": X.solve(_mask_faces(flux.at(1), nv))}
    u = flux.at()
    if kind == "rhs":
        ib = (nv > 0.1) & (nv < 1.1)
        fl = nv < 0.1
        tot = area = 0.0
        faces = []
        for q in range(3):
            a = X.cell[q].square().sum(-1).sqrt()
            for here, there, sign in ((fl, ib, 1.0), (ib, fl, -1.0)):
                f = X.inner & here & _sh(there, q, 1) & (X.idx[q] < X.m[q] - 2)
                v = u[..., q]
                v.masked_fill_(f & (v.abs() <= 1e-8), 0.0)
                g = f & (v.abs() > 1e-8)
                tot, area = tot + sign * v[g].sum(), area + a[g].sum()
                faces.append((q, f, g, a, sign))
        corr = tot / area if float(area) > 1e-15 else 0.0
        after = 0.0
        for q, f, g, a, sign in faces:
            u[..., q] -= torch.where(g, sign * a * corr, 0.0)
            after = after + a[f].sum()
        return {"ucont": u, "area": float(after), "b": torch.where(X.inner, X.rhs(u, c["dt"], c["coeff"]), 0.0)}
    rng = np.random.default_rng(seed + 1)
    phi = _field(c, _modes(rng), 0.0, (0.5, 0.5, 0.5)) * 0.01
    phi = _ghosts(c, phi.masked_fill_(nv > 0.1, 0.0))
    p = _ghosts(c, _field(c, _modes(rng), 0.0, (0.5, 0.5, 0.5)))
    p = torch.where(X.fluid, p + phi, p)
    p = _ghosts(c, torch.where(X.inner & (nv > 1.1), 0.0, p))
    f = X.flux(phi)
    comps = X.wrap_faces([u[..., q] - f[q] * (c["dt"] / c["coeff"]) for q in range(3)])
    near = nv + sum(_sh(nv, q, d) for q in range(3) for d in (1, -1))
    d = sum(comps[q] - _sh(comps[q], q, -1) for q in range(3)) * X.aj
    d = torch.where(X.inner & ~(near > 0.1), d.abs(), 0.0)
    return {"p": p, "phi": phi, "ucont": torch.stack(comps, -1), "maxdiv": float(d.max())}
