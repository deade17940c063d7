"""Timed work of the projection library, as its users run it: whole time steps on the grids of the
configurations and tests (launched and as one CUDA graph; mixed, FP64 and FP32-basis solves), a
step called with host fields, moving bodies, implicit momentum, the discrete adjoint, and the
entry points a program binds one by one (momentum operators, Poisson right-hand side and solve).

    listed()            the cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) a context with its grid, bodies and seeded flow
    run(state)          one pass through the public entry points; returns its outputs
    work(case)          bytes and flops a pass cannot do without
    exact(case, seed)   the outputs in plain 64-bit torch, where there is a direct formula

A case is a dict: `kind` (what a pass does), `grid` (channel, wavy, cylinders, wavy_cylinders),
nx/ny/nz (cells) and, for steps, `precision` (0 FP32 V-cycle in FP64 FGMRES, 1 all FP64, 2 FP32
basis), `graph` (1: the step as one CUDA graph), `les`, `sphere` (an immersed body with IB nodes).
"""
import ctypes
import functools
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "vfs-geophysics-3.1_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import vfs_b200 as vfs  # noqa: E402
from vfs_b200 import cases as grids  # noqa: E402

# Outer iterations a solve may take: the grids with odd cell counts coarsen little.
MAX_ITER = 400


def _case(name, kind, grid, nx, ny, nz, precision=0, graph=1, les=0, sphere=0, steps=0):
    return {"name": name, "kind": kind, "grid": grid, "nx": nx, "ny": ny, "nz": nz, "precision": precision,
            "graph": graph, "les": les, "sphere": sphere, "steps": steps}


def listed():
    return [
        # the smallest run: a first try of a set-up, a unit test, a parameter scan (launch latency)
        _case("step_channel_12x10x14", "step", "channel", 12, 10, 14),
        # the plain method: FP64 periodic channel
        _case("step_channel_64", "step", "channel", 64, 64, 64, precision=1),
        # a curvilinear grid whose cell counts are odd, kernels launched one by one (the default)
        _case("step_wavy_45x37x53", "step", "wavy", 45, 37, 53, graph=0),
        # dynamic-Smagorinsky LES over a wavy wall with an immersed sphere (IB nodes), FP64
        _case("step_les_sphere_128x96x128", "step", "wavy", 128, 96, 128, precision=1, les=2, sphere=1),
        # open channel with a cylinder array, inlet and outlet, mixed precision: production size
        _case("step_cylinders_256x192x256", "step", "cylinders", 256, 192, 256),
        # the same over a sinusoidal bottom: the 19-point operator
        _case("step_wavy_cylinders_192x128x192", "step", "wavy_cylinders", 192, 128, 192),
        # the step called from a host program that owns the fields: upload, step, download
        _case("hosted_cylinders_128x96x128", "hosted", "cylinders", 128, 96, 128, precision=2),
        # a moving body with the wall model: IB search, operator set-up and step every time step
        _case("moving_sphere_64x48x64", "moving", "channel", 64, 48, 64, graph=0, sphere=1),
        # implicit momentum (matrix-free Newton-Krylov) in place of the Runge-Kutta stages
        _case("implicit_channel_64x48x64", "implicit", "channel", 64, 48, 64, graph=0),
        # the gradient of the drag with respect to the inflow plane over a short window
        _case("adjoint_cylinders_64x48x64", "adjoint", "cylinders", 64, 48, 64, precision=1, graph=0, steps=4),
        # operators bound one by one: right-hand side and Poisson solve
        _case("poisson_channel_160x96x144", "poisson", "channel", 160, 96, 144, precision=1, graph=0),
        # operators bound one by one: velocities, eddy viscosity, momentum right-hand side, pressure gradient
        _case("momentum_wavy_176x120x200", "momentum", "wavy", 176, 120, 200, graph=0, les=2),
    ]


def _dims(rng, lo, hi, most):
    """Cells per direction, spread over the logarithm of [lo, hi], at most `most` cells in all:
    multiples of 8 (every direction coarsens three times), or any number on small grids."""
    while True:
        d = [int(round(np.exp(rng.uniform(np.log(lo), np.log(hi))))) for _ in range(3)]
        if min(d) >= 24 or rng.random() < 0.5:
            d = [max(16, 8 * round(v / 8)) for v in d]
        if d[0] * d[1] * d[2] <= most and max(d) <= 4 * min(d):
            return d


def draw(rng):
    kind = rng.choice(["step"] * 6 + ["hosted", "moving", "implicit", "adjoint", "poisson", "poisson", "momentum",
                                      "momentum"])
    if kind == "step":
        grid = rng.choice(["channel", "wavy", "cylinders", "wavy_cylinders"])
        lo = 32 if "cylinders" in grid else 10
        nx, ny, nz = _dims(rng, lo, 224, 4000000)
        les = rng.choice([0, 0, 1, 2]) if grid in ("channel", "wavy") else 0
        sphere = int(grid in ("channel", "wavy") and min(nx, ny, nz) >= 32 and rng.random() < 0.4)
        return _case("", "step", grid, nx, ny, nz, precision=rng.choice([0, 0, 1, 2]), graph=rng.choice([1, 1, 0]),
                     les=les, sphere=sphere)
    if kind == "hosted":
        d = _dims(rng, 32, 160, 2000000)
        return _case("", kind, "cylinders", *d, precision=rng.choice([0, 1, 2]))
    if kind == "moving":
        return _case("", kind, "channel", *_dims(rng, 32, 80, 300000), graph=0, sphere=1)
    if kind == "implicit":
        return _case("", kind, "channel", *_dims(rng, 24, 80, 300000), graph=0)
    if kind == "adjoint":
        return _case("", kind, "cylinders", *_dims(rng, 32, 80, 300000), precision=rng.choice([0, 1]), graph=0,
                     steps=rng.choice([2, 3, 4]))
    if kind == "poisson":
        return _case("", kind, "channel", *_dims(rng, 16, 200, 4000000), precision=rng.choice([0, 1, 2]), graph=0)
    return _case("", "momentum", rng.choice(["channel", "wavy", "wavy_cylinders"]), *_dims(rng, 32, 224, 6000000),
                 graph=0, les=rng.choice([0, 2]))


# ------------------------------------------------------------------ inputs
@functools.lru_cache(maxsize=2)
def _geometry(grid, nx, ny, nz):
    """The grid and its blocked cells (the same for every seed)."""
    if grid == "channel":
        return grids.channel(nx, ny, nz)
    if grid == "wavy":
        return grids.channel(nx, ny, nz, wavy=0.1)
    g = grids.inflow_outflow(grids.open_channel_cylinders(nx, ny, nz, wavy=0.05 if grid == "wavy_cylinders" else 0.0), 100)
    g.immersed = 0
    return g


def _geometry_of(case):
    g = _geometry(case["grid"], case["nx"], case["ny"], case["nz"])
    g.les = case["les"]
    g.immersed = case["sphere"]
    g.implicit = 4 if case["kind"] == "implicit" else 0
    g.moving = g.wallfunction = 1 if case["kind"] == "moving" else 0
    return g


class _Component:
    """One component of a field in device memory, shared without a copy."""

    def __init__(self, ctx, field, component):
        p = ctypes.c_void_p()
        ctx._check(ctx.lib.vfs_field_device_ptr(ctx.h, field, component, ctypes.byref(p)))
        self.ctx = ctx  # the memory is the context's
        self.__cuda_array_interface__ = {"shape": tuple(ctx.shape), "typestr": "<f8", "data": (p.value, False),
                                         "version": 3, "strides": None}


def _views(ctx, *fields):
    return {str(f): [torch.as_tensor(_Component(ctx, f, q), device="cuda") for q in range(vfs.FIELD_DOF[f])]
            for f in fields}


def _noise(shape, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    return torch.rand(shape, generator=gen, device="cuda", dtype=torch.float64) * 2 - 1


def _velocity(g, grid, nvert, seed):
    """Cartesian velocity at the cell centres (3, mz, my, mx): a channel's laminar parabola with
    uniform noise, or over cylinders a log law with random modes of a k^-5/3 spectrum."""
    mz, my, mx = g.da_shape
    nz, ny, nx = mz - 2, my - 2, mx - 2
    y = torch.from_numpy(np.ascontiguousarray(g.Y)).cuda()
    yc = 0.125 * sum(y[a:nz + a, b:ny + b, c:nx + c] for a in (0, 1) for b in (0, 1) for c in (0, 1))
    eta = (yc / g.Ly).clamp(1e-3, 1.0)
    u = torch.zeros((3, mz, my, mx), dtype=torch.float64, device="cuda")
    if "cylinders" in grid:
        mean = 1.0 + torch.log(eta / 0.2) / 0.41 * 0.0566
        mean /= mean.mean()
        kk = torch.sqrt(torch.fft.fftfreq(nz, device="cuda")[:, None] ** 2 +
                        torch.fft.rfftfreq(nx, device="cuda")[None, :] ** 2).double()
        amp = torch.where(kk > 0, kk.clamp(min=1e-9) ** (-5.0 / 6.0 - 0.5), torch.zeros_like(kk))[:, None, :]
        for c in range(3):
            f = _noise((nz, ny, nx), 1000003 * c + seed)
            f = torch.fft.irfft2(torch.fft.rfft2(f, dim=(0, 2)) * amp, s=(nz, nx), dim=(0, 2))
            u[c, 1:-1, 1:-1, 1:-1] = 0.05 * f / f.std()
    else:
        mean = 6.0 * eta * (1.0 - eta)
        for c in range(3):
            u[c, 1:-1, 1:-1, 1:-1] = 0.1 * _noise((nz, ny, nx), 1000003 * c + seed)
    u[2, 1:-1, 1:-1, 1:-1] += mean
    u[:, nvert > 0.1] = 0.0
    return u


def _fluxes(g, u, nvert, areas):
    """Face fluxes: the mean of the two cells dotted with the face area; zero on solid faces and
    on the upper wall of a direction that is not periodic."""
    out = torch.zeros_like(u)
    for c, ax in enumerate((2, 1, 0)):
        up = torch.roll(u, -1, dims=ax + 1)
        f = sum(0.5 * (u[q] + up[q]) * areas[c][q] for q in range(3))
        f[(nvert + torch.roll(nvert, -1, dims=ax)) > 0.1] = 0.0
        out[c, 1:-1, 1:-1, 1:-1] = f[1:-1, 1:-1, 1:-1]
        if not (g.i_periodic, g.j_periodic, g.k_periodic)[c]:
            out[c].select(ax, g.da_shape[ax] - 2).zero_()
    return out


def _host(v):
    return v.permute(1, 2, 3, 0).contiguous().cpu().numpy()


def _sphere(case):
    lz = 2 * np.pi
    return grids.icosphere((np.pi / 2, 1.0, lz / 2), 0.2 if case["nx"] >= 96 else 0.45, level=5 if case["nx"] >= 96 else 3)


def prepare(case, seed):
    g = _geometry_of(case)
    ctx = vfs.Context(g.config())
    ctx.form_metrics(g.X, g.Y, g.Z)
    nv = g.nvert if "cylinders" in case["grid"] else np.zeros(g.da_shape)
    ctx.set_field(vfs.NVERT, nv)
    s = {"ctx": ctx, "kind": case["kind"], "kw": {"precision": case["precision"], "rtol": 1e-10, "max_iter": MAX_ITER}}
    if case["sphere"]:
        s["body"] = _sphere(case)
        nv = ctx.ibm_search(*s["body"])
    ctx.synchronize()
    nvert = torch.from_numpy(nv).cuda()
    m = _views(ctx, vfs.ICSI, vfs.JETA, vfs.KZET)
    u = _velocity(g, case["grid"], nvert, seed)
    uc = _fluxes(g, u, nvert, [m[str(f)] for f in (vfs.ICSI, vfs.JETA, vfs.KZET)])
    del m
    u, uc = _host(u), _host(uc)
    ctx.set_field(vfs.UCONT, uc)
    ctx.set_field(vfs.UCAT, u)
    ctx.set_field(vfs.UCAT_O, u)
    ctx.set_field(vfs.UCONT_O, uc)
    _, area = ctx.calc_inlet_area()
    if "cylinders" in case["grid"]:
        ctx.set_inflow_plane(u[1])
        ctx.set_scalar(vfs.S_INLET_FLUX, area)  # bulk velocity 1
    ctx.contra2cart()
    if case["les"]:
        ctx.set_scalar(vfs.S_TI, 5)  # the model's coefficient is zero in the first two steps of a run
    if case["kind"] == "hosted":
        s["in"] = {f: torch.from_numpy(a).pin_memory().numpy() for f, a in
                   ((vfs.UCONT, uc), (vfs.UCAT, u), (vfs.P, ctx.get_field(vfs.P)))}
        s["out"] = {f: torch.empty(a.shape, dtype=torch.float64, pin_memory=True).numpy() for f, a in s["in"].items()}
    elif case["kind"] == "adjoint":
        ctx.adjoint_setup()
        s["steps"] = case["steps"]
    elif case["kind"] == "moving":
        s["pass"] = 0
    elif case["kind"] == "poisson":
        ctx.poisson_lhs()
    s["kw"]["graph"] = case["graph"]
    ctx.synchronize()
    torch.cuda.synchronize()
    return s


# ------------------------------------------------------------------ one pass
def run(s):
    ctx, kind, kw = s["ctx"], s["kind"], s["kw"]
    if kind == "step" or kind == "implicit":
        ctx.step(**kw)
        return _views(ctx, vfs.UCONT, vfs.UCAT, vfs.P, vfs.PHI)
    if kind == "hosted":
        for f, a in s["in"].items():
            ctx.set_field(f, a)
        ctx.step(**kw)
        for f, a in s["out"].items():
            ctx.get_field(f, out=a)
        return {str(f): a for f, a in s["out"].items()}
    if kind == "moving":
        # the body oscillates along the stream; its vertices move with it
        s["pass"] += 1
        x, y, z, tri = s["body"]
        t = 0.02 * s["pass"]
        ctx.ibm_search(x, y, z + 0.1 * np.sin(t), tri)
        ctx.ibm_set_velocity(np.zeros_like(x), np.zeros_like(x), np.full_like(x, 0.1 * np.cos(t)))
        ctx.step(**kw)
        return _views(ctx, vfs.UCONT, vfs.UCAT, vfs.P, vfs.PHI, vfs.NVERT)
    if kind == "adjoint":
        grad, st = ctx.adjoint_gradient(s["steps"], objective=vfs.OBJ_DRAG, control=vfs.CTRL_INFLOW_PLANE,
                                        checkpoint_every=2, **kw)
        return {"gradient": grad, "J": st.J}
    if kind == "poisson":
        ctx.poisson_rhs()
        ctx.poisson_solve(precision=kw["precision"], rtol=kw["rtol"], max_iter=kw["max_iter"], zero_guess=1)
        return _views(ctx, vfs.B, vfs.PHI)
    ctx.contra2cart()
    if ctx.cfg.les:
        ctx.smagorinsky_constant()
        ctx.eddy_viscosity()
    ctx.formfunction2(1.0)
    ctx.pressure_gradient()
    return _views(ctx, vfs.UCAT, vfs.NU_T, vfs.RHS, vfs.DP)


# ------------------------------------------------------------------ floors
def work(case):
    """Each operator's inputs read once and its outputs written once at their stored precision
    (metrics of a point 240 B of face and 72 B of centre vectors); a solve as nine Krylov
    iterations of one V-cycle, the operator and the orthogonalisation against the basis."""
    cells = float(case["nx"] * case["ny"] * case["nz"])
    wide = case["grid"].startswith("wavy")
    vc = 293.0 * (1 if case["precision"] != 1 else 2)
    basis = 4.0 if case["precision"] == 2 else 8.0
    apply_ = 169.0 if wide else 73.0
    its = 9
    solve = its * (apply_ + vc + 2 * basis) + sum(2 * basis * (j + 1) for j in range(its)) + 64.0
    solve_f = its * ((38 if wide else 14) + 250.0) + sum(8.0 * (j + 1) for j in range(its))
    momentum = 433.0 + 121.0
    correct = 169.0 + 129.0 + 121.0 + 96.0
    les = {0: 0.0, 1: 130.0, 2: 250.0}[case["les"]]
    les_f = {0: 0.0, 1: 120.0, 2: 5373.0}[case["les"]]
    step = 4 * momentum + 129.0 + 58.0 + solve + correct + les
    step_f = 4 * 900.0 + 300.0 + solve_f + les_f
    kind = case["kind"]
    if kind == "poisson":
        b, f = solve + 58.0, solve_f
    elif kind == "momentum":
        b, f = 121.0 + 417.0 + 129.0 + les, 1000.0 + les_f
    elif kind == "adjoint":  # the forward window, its recomputation and the transposed steps
        b, f = case["steps"] * 3.0 * step, case["steps"] * 3.0 * step_f
    elif kind == "hosted":
        b, f = step + 4 * 56.0, step_f
    elif kind == "moving":  # the operator and the solver's levels again every step
        b, f = step + 320.0 + 152.0 + 200.0, step_f + 400.0
    elif kind == "implicit":  # about ten residuals in place of the four stages
        b, f = step + 6 * momentum, step_f + 6 * 900.0
    else:
        b, f = step, step_f
    return {"bytes": cells * b, "flops": cells * f}


# ------------------------------------------------------------------ direct values
def exact(case, seed):
    """Right-hand side and solution of the Poisson problem on the periodic channel (uniform in x
    and z): Fourier transforms in x and z, a tridiagonal solve in y per mode.  The other passes
    are time steps and operators of a whole discretisation, which have no formula short of it."""
    if case["kind"] != "poisson":
        return None
    g = _geometry_of(case)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    x, y, z = (np.ascontiguousarray(a) for a in (g.X[0, 0, :], g.Y[0, :, 0], g.Z[:, 0, 0]))
    dx, dz = x[-1] / nx, z[-1] / nz
    dy = torch.from_numpy(np.diff(y)).cuda()
    gap = 0.5 * (dy[1:] + dy[:-1])
    # face areas at the cells' upper faces, in the DA layout
    mz, my, mx = g.da_shape
    zero = torch.zeros((mz, my, mx), dtype=torch.float64, device="cuda")
    ax, ay, az = zero.clone(), zero + dx * dz, zero.clone()
    ax[:, 1:-1, :] = (dy * dz)[None, :, None]
    az[:, 1:-1, :] = (dy * dx)[None, :, None]
    u = _velocity(g, "channel", zero, seed)
    uc = _fluxes(g, u, zero, [(ax, zero, zero), (zero, ay, zero), (zero, zero, az)])[:, 1:-1, 1:-1, 1:-1]
    b = uc[0] - torch.roll(uc[0], 1, 2) + uc[2] - torch.roll(uc[2], 1, 0)
    b += uc[1]
    b[:, 1:] -= uc[1][:, :-1]
    b = b / g.dt * g.st
    aj = (1.0 / (dx * dy * dz))[None, :, None].expand(nz, ny, nx)
    b = b - b.sum() * aj / aj.sum()
    # conductances and the modes' eigenvalues
    cx, cz, cy = dy * dz / dx, dy * dx / dz, dx * dz / gap
    lx = 2 - 2 * torch.cos(2 * np.pi * torch.arange(nx // 2 + 1, device="cuda", dtype=torch.float64) / nx)
    lz = 2 - 2 * torch.cos(2 * np.pi * torch.arange(nz, device="cuda", dtype=torch.float64) / nz)
    f = torch.fft.rfft2(b, dim=(0, 2))
    up = torch.cat([cy, cy.new_zeros(1)])
    lo = torch.cat([cy.new_zeros(1), cy])
    d, e = [], []
    for j in range(ny):
        diag = -(up[j] + lo[j]) - cx[j] * lx[None, :] - cz[j] * lz[:, None]
        if j == ny - 1:
            diag[0, 0] -= cy[-1]  # the mean is free: fixed here, removed below
        den = diag - (lo[j] * e[-1] if j else 0.0)
        e.append(up[j] / den)
        d.append((f[:, j, :] - (lo[j] * d[-1] if j else 0.0)) / den)
    for j in range(ny - 2, -1, -1):
        d[j] = d[j] - e[j] * d[j + 1]
    phi = torch.fft.irfft2(torch.stack(d, 1), s=(nz, nx), dim=(0, 2))
    phi = phi - phi.mean()
    out_b, out_p = zero.clone(), zero.clone()
    out_b[1:-1, 1:-1, 1:-1] = b
    out_p[1:-1, 1:-1, 1:-1] = phi
    out_p[:, :, 0], out_p[:, :, -1] = out_p[:, :, -2].clone(), out_p[:, :, 1].clone()
    out_p[0], out_p[-1] = out_p[-2].clone(), out_p[1].clone()
    return {str(vfs.B): [out_b], str(vfs.PHI): [out_p]}
