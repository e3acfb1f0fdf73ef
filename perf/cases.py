"""Performance cases of the library: what its users have it do.

A case is one of
  step       one LES time step (falm_step) of a running simulation: forcing,
             pseudo-velocity, Poisson solve, projection, boundary conditions, SGS
  adjoint    one reverse step of the power gradient (falm_step_adjoint)
  operators  the solver classes called one by one, as a program ported from the
             reference's own main loop calls them (FalmCFD, AlmHandler)
  solve      one pressure solve through FalmEq on a caller's right-hand side,
             with the Poisson operator or a caller's 7-column matrix
on a channel with an actuator-line rotor, or a lid-driven cavity, in FP64 or
mixed precision (FP32 fields).  Sizes and settings are those of
falm_b200/cases.py, of the tests and of bench.py, with the time step at the CFL
number 0.05 at which the explicit scheme runs indefinitely.

Fields start as a flow in progress: a mean velocity plus a smooth solenoidal
perturbation drawn from the seed, with the face velocity and the eddy viscosity
that belong to it.  `exact` restates every stage in FP64 torch.
"""
import math

import numpy as np
import torch
import torch.nn.functional as F

from falm_b200 import cases as C
from falm_b200.api import Context

GC = 2
ALPHA4 = {"Upwind3": 1.0 / 24.0, "UTOPIA": 1.0 / 12.0, "KK": 0.25}
W_POWER = 1.0 / 200.0   # a 200-step averaging window


# ---------------------------------------------------------------- the cases
def _case(name, kind, nx, ny, nz, precision, bc="channel", cpr=20, inflow=0.0, tol=1e-6, maxit=1000, adv="Upwind3", stretch=1.0,
          pitching=False, matrix=False):
    c = {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "precision": precision, "bc": bc, "cells_per_radius": cpr, "inflow": inflow,
         "tol": tol, "maxit": maxit, "adv": adv, "stretch": stretch, "pitching": pitching, "matrix": matrix}
    return dict(c, name=name) if name else c


def _tol(nx, ny, nz):
    """channel_large's tolerance of 1e-6 on ||r||_2 / N, as the same root mean square residual on any grid"""
    return 5.8e-3 / math.sqrt(nx * ny * nz)


def listed():
    # Solves end after the same number of iterations at every step, so that passes are alike: mixed
    # steps meet channel_large's tolerance after one, FP64 steps and solves run a fixed number.
    return [
        # the smallest configuration: a 64^3 lid-driven cavity, some thirty kernels of a few microseconds
        _case("cavity_64_fp64", "step", 64, 64, 64, "fp64", bc="cavity", cpr=64, tol=1e-30, maxit=3),
        # the same problem in FP32 on a mesh that no tile divides
        _case("cavity_101_mixed", "step", 101, 101, 101, "mixed", bc="cavity", cpr=101, tol=_tol(101, 101, 101)),
        # the forward step of a gradient window (R = 10 cells), a solve of many iterations
        _case("channel_128_fp64", "step", 128, 64, 64, "fp64", cpr=10, tol=1e-30, maxit=20),
        # the turbine in a turbulent inflow on the 256x128x128 channel
        _case("channel_256_inflow_mixed", "step", 256, 128, 128, "mixed", inflow=0.05, tol=_tol(256, 128, 128)),
        # the 512x256x256 production step in both precisions
        _case("channel_512_mixed", "step", 512, 256, 256, "mixed", tol=1e-6),
        _case("channel_512_fp64", "step", 512, 256, 256, "fp64", tol=1e-6),
        # a channel cut to fit a site: odd sizes in every direction
        _case("channel_ragged_mixed", "step", 301, 157, 131, "mixed", inflow=0.05, tol=_tol(301, 157, 131)),
        # the largest: a floating turbine, the platform pitching, 67 M cells
        _case("floating_1024_mixed", "step", 1024, 256, 256, "mixed", cpr=24, inflow=0.08, tol=1e-6, pitching=True),
        # the reverse step of a gradient window
        _case("adjoint_128_fp64", "adjoint", 128, 64, 64, "fp64", cpr=10),
        # a ported main loop's operator calls on a stretched mesh
        _case("operators_stretched_fp64", "operators", 192, 96, 90, "fp64", stretch=1.01, adv="UTOPIA"),
        # pressure solves of their own: FP64 on a stretched mesh, and the FP32 recursion with its
        # restarts from the FP64 residual (five passes of four iterations)
        _case("solve_stretched_fp64", "solve", 200, 120, 96, "fp64", stretch=1.01, tol=1e-30, maxit=20),
        _case("solve_256_mixed", "solve", 256, 128, 128, "mixed", tol=1e-30, maxit=4),
    ]


def draw(rng):
    """One more case: grids of 32^3 to 16 M cells of any aspect and parity, every kind, both precisions."""
    kind = rng.choice(["step", "step", "step", "step", "adjoint", "operators", "solve"])
    precision = rng.choice(["fp64", "mixed"])
    top = {"step": 1.6e7, "adjoint": 1e6, "operators": 4e6, "solve": 4e6}[kind]
    cells = math.exp(rng.uniform(math.log(3.2e4), math.log(top if precision == "mixed" else top / 2)))
    if kind != "adjoint" and rng.random() < 0.25:
        n = max(32, round(min(cells, 2e6) ** (1 / 3)) + rng.randint(-3, 3))
        nx, ny, nz, cpr, bc = n, max(32, n + rng.choice([0, 0, -1, 3])), n, n, "cavity"
    else:
        a, b = rng.uniform(1.2, 3.0), rng.uniform(0.8, 1.25)
        ny = max(30, round((cells / a * b) ** (1 / 3)))
        nz = max(30, round(ny / b))
        nx = max(40, round(ny * a))
        cpr, bc = max(4, min(24, int(min(ny, nz) / rng.uniform(2.6, 6.4)))), "channel"
    if kind == "solve" or (kind == "step" and precision == "fp64"):
        tol, maxit = 1e-30, rng.randint(1, 12) if precision == "fp64" else rng.randint(2, 4)
    else:
        tol, maxit = _tol(nx, ny, nz), 1000
    adv = rng.choice(["Upwind3", "Upwind3", "UTOPIA", "KK"] + ([] if kind == "adjoint" else ["QUICK", "Upwind1"]))
    return _case(None, kind, nx, ny, nz, precision, bc=bc, cpr=cpr, inflow=rng.choice([0.0, 0.05, 0.08]) if bc == "channel" else 0.0,
                 adv=adv, tol=tol, maxit=maxit, stretch=rng.choice([1.0, 1.0, 1.005]) if kind in ("operators", "solve") else 1.0,
                 pitching=bc == "channel" and rng.random() < 0.3, matrix=kind == "solve" and rng.random() < 0.4)


# ---------------------------------------------------------------- set-up shared by prepare and exact
def _setup(case):
    """the grid, the rotor and the scalars of a case (falm_b200.cases objects)"""
    h = 1.0 / case["cells_per_radius"]
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    grid = C.uniform_grid(nx, ny, nz, h) if case["stretch"] == 1.0 else C.stretched_grid(nx, ny, nz, h, case["stretch"])
    if case["bc"] == "cavity":
        return C.Case("cavity", grid, 1, Re=1000.0, dt=0.064 * h, tol=case["tol"], maxit=case["maxit"], adv=case["adv"], u_inlet=0.0)
    mid = [0.5 * (float(a[GC - 1 + n // 2]) + float(a[GC + n // 2])) for a, n in ((grid.y, ny), (grid.z, nz))]
    hub = (min(3.2, 0.35 * nx * h), mid[0], mid[1])
    if case["pitching"]:
        rotor = C.make_rotor(hub, h, tsr=9.0, pitch=3.0, platform_pitch_deg=3.0, platform_period=10.0, tower=1.0)
    else:
        rotor = C.make_rotor(hub, h)
    return C.Case("channel", grid, 0, Re=1e4, dt=0.05 * h, tol=case["tol"], maxit=case["maxit"], adv=case["adv"], alm=rotor,
                  intensity=case["inflow"])


def _smooth(shape, ncomp, gen, every=6):
    """ncomp smooth random fields: normal values on every sixth cell, interpolated"""
    low = [max(2, s // every + 2) for s in shape]
    v = torch.randn(1, ncomp, *low, generator=gen, device="cuda", dtype=torch.float32)
    return F.interpolate(v, size=shape, mode="trilinear", align_corners=True)[0].double()


def _solenoidal(m, gen, rms):
    """curl of a smooth random vector potential by central differences: free of
    divergence in the interior of a uniform grid"""
    a = F.pad(_smooth(m.shape, 3, gen), (1, 1, 1, 1, 1, 1), mode="replicate")
    d = lambda c, ax: (torch.roll(a[c], -1, 2 - ax) - torch.roll(a[c], 1, 2 - ax))[1:-1, 1:-1, 1:-1]  # noqa: E731
    u = torch.stack([d(2, 1) - d(1, 2), d(0, 2) - d(2, 0), d(1, 0) - d(0, 1)])
    return u * (rms / u.square().mean().sqrt())


def _inputs(case, seed, setup, m):
    """the fields of a flow in progress (FP64; a mixed context rounds them)"""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    mixed = case["precision"] == "mixed"
    r32 = (lambda t: t.float().double()) if mixed else (lambda t: t)
    cavity = case["bc"] == "cavity"
    u = _solenoidal(m, gen, 0.02 if cavity else 0.05)
    if not cavity:
        u[0] += 1.0
    u = r32(u)
    _ubc_cavity(m, u) if cavity else None
    p = torch.zeros(m.shape, dtype=torch.float64, device="cuda")
    out = {"u": u, "uu": r32(_face_velocity(m, u, torch.zeros_like(u), cavity)), "p": p,
           "nut": r32(_smagorinsky(m, u, torch.zeros_like(p), setup.Cs)), "box": None}
    if case["inflow"]:
        nb, (nz, ny) = 64, (case["nz"], case["ny"])
        box = _smooth((nb, nz, ny), 3, gen, every=4)
        out["box"] = box * (case["inflow"] / box.square().mean().sqrt())
    kind = case["kind"]
    if kind == "adjoint":
        out["u_after"] = r32(u + setup.dt * 0.2 * _smooth(m.shape, 3, gen))
        out["au"], out["auu"] = 1e-4 * _smooth(m.shape, 3, gen), 1e-4 * _smooth(m.shape, 3, gen)
        out["anut"] = 1e-5 * _smooth(m.shape, 1, gen)[0]
    elif kind == "operators":
        out["p"] = r32(0.1 * _smooth(m.shape, 1, gen)[0])
    elif kind == "solve":
        b = torch.zeros_like(p)
        b[m.inner] = 1e-2 * _smooth(m.shape, 1, gen)[0][m.inner]
        if cavity:
            b[m.inner] -= b[m.inner].mean()   # the singular operator's range
        out["b"] = r32(b)
        out["x0"] = p
    return out


# ---------------------------------------------------------------- prepare, run
def prepare(case, seed):
    setup = _setup(case)
    m = _Mesh(setup.grid)
    f = _inputs(case, seed, setup, m)
    ctx = Context(setup.grid, case["precision"])
    ctx.cfd_init(setup.Re, setup.adv, setup.sgs, setup.Cs)
    ctx.eq_init(setup.maxit, setup.tol, setup.pc, setup.pc_maxit, setup.pc_relax)
    ctx.bc_init(setup.bc, setup.u_inlet)
    maxdiag = ctx.poisson_operator(setup.bc)
    if f["box"] is not None:
        ctx.set_inflow(f.pop("box").cpu().numpy(), float(setup.grid.hx[GC]))
    if setup.alm is not None:
        ctx.alm_init(setup.alm)
    own = lambda k, t=ctx.dtype: f.pop(k).to(t).contiguous().view(-1)  # noqa: E731
    s = {"ctx": ctx, "kind": case["kind"], "dt": setup.dt, "it": 0}
    for k in ("u", "uu", "p", "nut"):
        s[k] = own(k)
    if case["kind"] == "adjoint":
        s["u_after"] = own("u_after")
        for k in ("au", "auu", "anut"):
            s[k] = own(k, torch.float64)
        ctx.adjoint_set_tol(1e-9)   # a gradient to be compared with differences of the step
        s["grad"] = torch.zeros(1 + 2 * setup.alm.apcount, dtype=torch.float64, device="cuda")
    elif case["kind"] == "operators":
        s["maxdiag"] = maxdiag
        for k, ncol in (("ff", 3), ("ua", 3), ("uu1", 3), ("u2", 3), ("uu2", 3), ("rhs", 1), ("nut2", 1), ("div", 1)):
            s[k] = ctx.field(ncol)
    elif case["kind"] == "solve":
        if case["matrix"]:
            s["A"] = _Poisson(m, setup.bc).columns().to(ctx.dtype).contiguous().view(-1)
            ctx.set_matrix(s["A"])
        s["b"], s["x0"], s["x"], s["r"] = own("b"), own("x0"), ctx.field(1), ctx.field(1)
    return s


def run(s):
    ctx, dt = s["ctx"], s["dt"]
    if s["kind"] == "step":
        s["it"] += 1
        st = ctx.step(s["u"], s["uu"], s["p"], s["nut"], None, dt, s["it"] * dt)
        return {"u": s["u"], "uu": s["uu"], "p": s["p"], "nut": s["nut"], "torque": st["torque"], "thrust": st["thrust"]}
    if s["kind"] == "adjoint":
        ctx.step_adjoint(s["u"], s["uu"], s["p"], s["nut"], dt, dt, W_POWER, s["au"], s["auu"], s["anut"], s["grad"],
                         u_after=s["u_after"])
        return {"au": s["au"], "auu": s["auu"], "anut": s["anut"], "grad": s["grad"]}
    if s["kind"] == "operators":
        out = {}
        if ctx.alm_on:
            out["torque"], out["thrust"] = ctx.alm_run(s["u"], s["ff"], dt)
        ctx.pseudo_u(s["u"], s["u"], s["uu"], s["ua"], s["nut"], s["ff"], dt)
        ctx.utouu(s["ua"], s["uu1"])
        ctx.poisson_rhs(s["uu1"], s["rhs"], dt, s["maxdiag"])
        ctx.project_p(s["u2"], s["ua"], s["uu2"], s["uu1"], s["p"], dt)
        ctx.ubc(s["u2"], s["u"], dt, dt)
        ctx.sgs(s["u2"], s["nut2"])
        ctx.divergence(s["uu2"], s["div"])
        return dict(out, **{k: s[k] for k in ("ff", "ua", "uu1", "rhs", "u2", "uu2", "nut2", "div")})
    s["x"].copy_(s["x0"])
    ctx.solve(s["x"], s["b"], s["r"])
    return {"x": s["x"], "r": s["r"]}


def work(case):
    """each field read once and written once; the operations of the stages (a nominal solver iteration 150 a cell)"""
    n = case["nx"] * case["ny"] * case["nz"]
    size = 8 if case["precision"] == "fp64" else 4
    if case["kind"] == "step":
        return {"bytes": 16 * size * n, "flops": (420 + 2 * 150) * n}
    if case["kind"] == "adjoint":   # the state and the velocity after it, and the FP64 adjoint fields in and out
        return {"bytes": (11 * size + 14 * 8) * n, "flops": (1200 + 20 * 150) * n}
    if case["kind"] == "operators":  # u, uu, nut, p in; ff, ua, uu1, rhs, u2, uu2, nut2, div out
        return {"bytes": (8 + 18) * size * n, "flops": 450 * n}
    a = 7 if case["matrix"] else 0
    return {"bytes": (4 + a) * size * n, "flops": min(case["maxit"], 20) * 150 * n}


def tolerance(case):
    """about four times the distance to the FP64 restatement: rounding, which a solve carries
    through the scalars of its iterations into the pressure (and most into a residual)"""
    mixed = case["precision"] == "mixed"
    if case["kind"] == "adjoint":
        return {"rel": 1e-5, "max": 1e-3}    # the transposed solve stops at a relative residual of 1e-9
    if case["kind"] == "operators":
        return {"rel": 4e-6, "max": 1e-3} if mixed else {"rel": 1e-13, "max": 1e-10}
    if case["kind"] == "solve":
        return {"rel": 3e-3, "max": 0.2} if mixed else {"rel": 1e-8, "max": 1e-5}
    return {"rel": 3e-4, "max": 0.02} if mixed else {"rel": 1e-8, "max": 1e-5}


# ---------------------------------------------------------------- the stages in FP64 torch
class _Mesh:
    """1D metric tables and shifted views of fields shaped [..., sz, sy, sx]"""

    def __init__(self, grid):
        self.grid = grid
        self.shape = (grid.sz, grid.sy, grid.sx)
        t = lambda a: torch.as_tensor(a, dtype=torch.float64, device="cuda")  # noqa: E731
        self.x = [t(a) for a in (grid.x, grid.y, grid.z)]
        self.h = [t(a) for a in (grid.hx, grid.hy, grid.hz)]
        self.dims = (grid.sx, grid.sy, grid.sz)
        self.lo = (GC, GC, GC)
        self.hi = tuple(s - GC for s in self.dims)
        self.inner = self.box(self.lo, self.hi)
        self.faces = ((GC - 1,) * 3, self.hi)   # cells that own a computed plus face

    def box(self, lo, hi, off=(0, 0, 0)):
        return (Ellipsis,) + tuple(slice(lo[d] + off[d], hi[d] + off[d]) for d in (2, 1, 0))

    def axis(self, v, d, lo, hi, off=0):
        s = [1, 1, 1]
        s[2 - d] = hi[d] - lo[d]
        return v[lo[d] + off:hi[d] + off].view(s)

    def volume(self, lo, hi, off=(0, 0, 0)):
        return self.axis(self.h[0], 0, lo, hi, off[0]) * self.axis(self.h[1], 1, lo, hi, off[1]) * self.axis(self.h[2], 2, lo, hi, off[2])

    def metric(self, d, lo, hi, off=(0, 0, 0)):
        return self.volume(lo, hi, off) / self.axis(self.h[d], d, lo, hi, off[d]) ** 2


def _unit(d, n=1):
    return tuple(n if a == d else 0 for a in range(3))


def _face_velocity(m, u, uu, cavity):
    """contravariant velocity averaged onto the plus faces"""
    lo, hi = m.faces
    out = uu.clone()
    for d in range(3):
        e = _unit(d)
        c = lambda off: m.volume(lo, hi, off) / m.axis(m.h[d], d, lo, hi, off[d]) * u[d][m.box(lo, hi, off)]  # noqa: E731
        out[d][m.box(lo, hi)] = 0.5 * (c((0, 0, 0)) + c(e))
        if cavity:
            wall = [slice(GC, m.dims[a] - GC) for a in (2, 1, 0)]
            for at in (GC - 1, m.dims[d] - GC - 1):
                wall[2 - d] = at
                out[(d,) + tuple(wall)] = 0.0
    return out


def _divergence(m, uu):
    lo, hi = m.lo, m.hi
    return sum(uu[d][m.box(lo, hi)] - uu[d][m.box(lo, hi, _unit(d, -1))] for d in range(3)) / m.volume(lo, hi)


def _smagorinsky(m, u, nut, Cs):
    lo, hi = m.lo, m.hi
    g = [[0.5 / m.axis(m.h[a], a, lo, hi) * (u[c][m.box(lo, hi, _unit(a))] - u[c][m.box(lo, hi, _unit(a, -1))]) for a in range(3)]
         for c in range(3)]
    s = 2 * (g[0][0] ** 2 + g[1][1] ** 2 + g[2][2] ** 2) + (g[0][1] + g[1][0]) ** 2 + (g[1][2] + g[2][1]) ** 2 + (g[0][2] + g[2][0]) ** 2
    out = nut.clone()
    out[m.inner] = (Cs * m.volume(lo, hi) ** (1.0 / 3.0)) ** 2 * torch.sqrt(s)
    return out


def _pseudo(m, u, uu, nut, ff, Re, dt, adv):
    """u + dt (-advection + diffusion + force) on the interior; guide cells keep u"""
    lo, hi = m.lo, m.hi
    jac = m.volume(lo, hi)
    at = lambda f, d, n: f[m.box(lo, hi, _unit(d, n))]  # noqa: E731
    out = u.clone()
    speed = [(u[a][m.inner] / m.axis(m.h[a], a, lo, hi)).abs() for a in range(3)]
    for d in range(3):
        f = u[d]
        c = f[m.inner]
        acc = torch.zeros_like(c) if ff is None else ff[d][m.inner].clone()
        for a in range(3):
            jp, jm = uu[a][m.inner], at(uu[a], a, -1)
            p1, m1 = at(f, a, 1), at(f, a, -1)
            if adv == "Upwind1":
                acc = acc - 0.5 * (jp * (p1 + c) - jp.abs() * (p1 - c) - jm * (c + m1) + jm.abs() * (c - m1)) / jac
            else:
                p2, m2 = at(f, a, 2), at(f, a, -2)
                if adv == "QUICK":
                    acc = acc - (jp * (-p2 + 9 * p1 + 9 * c - m1) + jp.abs() * (p2 - 3 * p1 + 3 * c - m1)
                                 - jm * (-p1 + 9 * c + 9 * m1 - m2) - jm.abs() * (p1 - 3 * c + 3 * m1 - m2)) / (16 * jac)
                else:
                    acc = acc - 0.5 * (jp * (-p2 + 27 * p1 - 27 * c + m1) + jm * (-p1 + 27 * c - 27 * m1 + m2)) / (24 * jac)
                    acc = acc - ALPHA4[adv] * speed[a] * (p2 - 4 * p1 + 6 * c - 4 * m1 + m2)
            gc, gp, gm = m.metric(a, lo, hi), m.metric(a, lo, hi, _unit(a)), m.metric(a, lo, hi, _unit(a, -1))
            nc = nut[m.inner]
            acc = acc + ((gc + gp) * (1 / Re + 0.5 * (nc + at(nut, a, 1))) * (p1 - c)
                         - (gc + gm) * (1 / Re + 0.5 * (nc + at(nut, a, -1))) * (c - m1)) / (2 * jac)
        out[d][m.inner] = c + dt * acc
    return out


class _Poisson:
    """the scaled 7-point operator as 1D coefficient tables: Neumann on every face but a channel's outlet"""

    def __init__(self, m, bc):
        self.m = m
        up, dn = [], []
        for d in range(3):
            h, n = m.h[d], m.dims[d]
            q = torch.arange(GC, n - GC, device="cuda")
            plus, minus = 0.5 * (1 / h[q] + 1 / h[q + 1]) / h[q], 0.5 * (1 / h[q] + 1 / h[q - 1]) / h[q]
            minus[0] = 0.0
            if not (d == 0 and bc == 0):
                plus[-1] = 0.0
            s = [1, 1, 1]
            s[2 - d] = -1
            up.append(plus.view(s))
            dn.append(minus.view(s))
        diag = -sum(up) - sum(dn)
        self.maxdiag = float(diag.abs().max())
        self.up, self.dn, self.diag = [v / self.maxdiag for v in up], [v / self.maxdiag for v in dn], diag / self.maxdiag
        i = [torch.arange(GC, n - GC, device="cuda") for n in m.dims]
        self.colour = (i[2].view(-1, 1, 1) + i[1].view(1, -1, 1) + i[0].view(1, 1, -1)) & 1

    def columns(self):
        """the seven columns c, w, e, s, n, b, t over the whole box"""
        A = torch.zeros((7,) + self.m.shape, dtype=torch.float64, device="cuda")
        for col, v in enumerate((self.diag, self.dn[0], self.up[0], self.dn[1], self.up[1], self.dn[2], self.up[2])):
            A[col][self.m.inner] = v.expand(self.diag.shape)
        return A

    def apply(self, x):
        """A x on the interior of a field with guide cells"""
        m = self.m
        y = self.diag * x[m.inner]
        for d in range(3):
            y += self.up[d] * x[m.box(m.lo, m.hi, _unit(d))] + self.dn[d] * x[m.box(m.lo, m.hi, _unit(d, -1))]
        return y

    def sor(self, b, sweeps=2, omega=1.2):
        z = torch.zeros(self.m.shape, dtype=torch.float64, device="cuda")
        zi = z[self.m.inner]
        for half in range(2 * sweeps):
            zi += torch.where(self.colour == (half & 1), omega * (b - self.apply(z)) / self.diag, 0.0)
        return z

    def bicgstab(self, x, b, tol, maxit):
        """right-preconditioned BiCGStab in place on x; b and the residual on the interior"""
        m, n = self.m, self.diag.numel()
        xi = x[m.inner]
        r = b - self.apply(x)
        rr, p, q = r.clone(), None, None
        rho = float((r * rr).sum())
        for _ in range(maxit):
            if abs(rho) < 1.17549435e-38:
                break
            p = r.clone() if p is None else r + beta * (p - omega * q)  # noqa: F821
            pp = self.sor(p)
            q = self.apply(pp)
            alpha = rho / float((rr * q).sum())
            s = r - alpha * q
            ss = self.sor(s)
            t = self.apply(ss)
            omega = float((t * s).sum()) / float((t * t).sum())
            xi += alpha * pp[m.inner] + omega * ss[m.inner]
            r = s - omega * t
            if math.sqrt(float((r * r).sum())) / n <= tol:
                break
            new = float((r * rr).sum())
            beta = new * alpha / (rho * omega)
            rho = new
        return r

    def transposed(self, b):
        """A^T y = b to rounding: diag(volume) A is symmetric, so CG on it with y = volume w"""
        m = self.m
        v = m.volume(m.lo, m.hi)
        w = torch.zeros(m.shape, dtype=torch.float64, device="cuda")
        wi, r = w[m.inner], -b.clone()
        d = torch.zeros_like(w)
        d[m.inner] = r
        rs = float((r * r).sum())
        stop = 1e-22 * rs
        for _ in range(20000):
            if rs <= stop:
                break
            q = -v * self.apply(d)
            a = rs / float((d[m.inner] * q).sum())
            wi += a * d[m.inner]
            r -= a * q
            new = float((r * r).sum())
            d[m.inner] = r + (new / rs) * d[m.inner]
            rs = new
        return v * wi


class _PressureOf(torch.autograd.Function):
    """a pressure with the derivative of the exact solve (its value does not enter the gradient)"""

    @staticmethod
    def forward(ctx, rhs, op):
        ctx.op = op
        return torch.zeros_like(rhs)

    @staticmethod
    def backward(ctx, g):
        return ctx.op.transposed(g), None


def _pbc(m, p, bc):
    """Neumann guide values, zero at a channel's outlet"""
    out = p.clone()
    for d in range(3):
        for at, src in ((GC - 1, GC), (m.dims[d] - GC, m.dims[d] - GC - 1)):
            lo, hi = list(m.lo), list(m.hi)
            lo[d], hi[d] = at, at + 1
            v = p[m.box(lo, hi, _unit(d, src - at))]
            out[m.box(lo, hi)] = torch.zeros_like(v) if bc == 0 and d == 0 and at > GC else v
    return out


def _project(m, u, ua, uu, p, dt):
    """cell velocity on the interior of ua into u, face velocity on the face map"""
    u, uu = u.clone(), uu.clone()
    lo, hi = m.lo, m.hi
    for d in range(3):
        k = 0.5 / m.axis(m.h[d], d, lo, hi)
        u[d][m.inner] = ua[d][m.inner] - dt * k * (p[m.box(lo, hi, _unit(d))] - p[m.box(lo, hi, _unit(d, -1))])
    lo, hi = m.faces
    for d in range(3):
        g = 0.5 * (m.metric(d, lo, hi) + m.metric(d, lo, hi, _unit(d)))
        uu[d][m.box(lo, hi)] = uu[d][m.box(lo, hi)] - dt * g * (p[m.box(lo, hi, _unit(d))] - p[m.box(lo, hi)])
    return u, uu


def _ubc_cavity(m, u):
    """reflection about the wall value, the lid on y+"""
    for d in range(3):
        n = m.dims[d]
        for g, s in ((GC - 1, GC), (GC - 2, GC + 1), (n - GC, n - GC - 1), (n - GC + 1, n - GC - 2)):
            lo, hi = list(m.lo), list(m.hi)
            lo[d], hi[d] = g, g + 1
            to, fr = m.box(lo, hi), m.box(lo, hi, _unit(d, s - g))
            for c in range(3):
                u[c][to] = (2.0 if c == 0 and d == 1 and g >= n - GC else 0.0) - u[c][fr]


def _ubc_channel(m, u, before, dt, inlet):
    """given inlet, convective outlet, slip sides and top, no-slip bottom"""
    def at(d, i):
        lo, hi = list(m.lo), list(m.hi)
        lo[d], hi[d] = i, i + 1
        return m.box(lo, hi)
    n = m.dims[0]
    k = 0.5 / (m.x[0][n - GC] - m.x[0][n - GC - 1])
    for c in range(3):
        u[c][at(0, GC - 1)] = inlet[c].unsqueeze(-1)
        u[c][at(0, GC - 2)] = inlet[c].unsqueeze(-1)
        o, i1, i2 = (before[c][at(0, n - GC - q)] for q in (0, 1, 2))
        out = o - dt * k * (3 * o - 4 * i1 + i2)
        u[c][at(0, n - GC)] = out
        u[c][at(0, n - GC + 1)] = 2 * out - u[c][at(0, n - GC - 1)]
    for d, sides in ((1, ((GC, -1, True), (m.dims[1] - GC - 1, 1, True))), (2, ((GC, -1, False), (m.dims[2] - GC - 1, 1, True)))):
        for i, s, slip in sides:
            for c in range(3):
                v = u[c][at(d, i)].clone()
                w = v if slip and c != d else torch.zeros_like(v)
                u[c][at(d, i + s)] = w
                u[c][at(d, i + 2 * s)] = 2 * w - v


def _inlet(setup, box, t, like):
    """the inlet plane [3, nz, ny] at time t: the inflow box carried by the mean velocity"""
    nx, ny, nz = setup.grid.interior
    plane = torch.zeros((3, nz, ny), dtype=torch.float64, device=like.device)
    if box is not None:
        x = setup.u_inlet * t / float(setup.grid.hx[GC])
        s, f = int(math.floor(x)), x - math.floor(x)
        plane += (1.0 - f) * box[:, s % box.shape[1]] + f * box[:, (s + 1) % box.shape[1]]
    plane[0] += setup.u_inlet
    return plane


def _rotor(m, alm, u, t, table=None):
    """actuator forces at time t: positions, force vectors, |tangential force| radius and thrust of each point.
    table: pitch, chord, twist to use in place of the rotor's own"""
    dev = u.device
    n = alm.n_blade * alm.n_ap_per_blade
    tip, base, hub = float(alm.tip_rate[0]), alm.base[0], alm.hub[0]
    apr = torch.as_tensor(alm.aps["r"], device=dev)
    own = (torch.tensor(alm.pitch, dtype=torch.float64, device=dev), torch.as_tensor(alm.aps["chord"], device=dev),
           torch.as_tensor(alm.aps["twist"], device=dev))
    pitch, chord, twist = table or own
    theta = tip * t + (2 * math.pi / alm.n_blade) * (torch.arange(n, device=dev) // alm.n_ap_per_blade).double()
    ang = rate = 0.0
    if alm.angle_type[0] == 2:   # platform pitch, about y
        amp, freq, phase = alm.motion[0]
        ang, rate = amp * math.sin(freq * t + phase), amp * freq * math.cos(freq * t + phase)
    cs, sn = math.cos(ang), math.sin(ang)
    cx, cy, cz = torch.full_like(apr, hub[0]), hub[1] + apr * torch.cos(theta), hub[2] + apr * torch.sin(theta)
    rel = (cs * cx + sn * cz, cy, -sn * cx + cs * cz)
    pos = [rel[d] + base[d] for d in range(3)]
    idx, w = [], []
    for d in range(3):
        i = torch.searchsorted(m.x[d], pos[d].contiguous(), right=True) - 1
        idx.append(i)
        w.append((pos[d] - m.x[d][i]) / (m.x[d][i + 1] - m.x[d][i]))
    vel = [0.0, 0.0, 0.0]
    for a in (0, 1):
        for b in (0, 1):
            for c in (0, 1):
                wt = (w[0] if a else 1 - w[0]) * (w[1] if b else 1 - w[1]) * (w[2] if c else 1 - w[2])
                for d in range(3):
                    vel[d] = vel[d] + wt * u[d][idx[2] + c, idx[1] + b, idx[0] + a]
    vx = rate * (-sn * rel[0] - cs * rel[2]) + cs * vel[0] - sn * vel[2]
    vz = rate * (cs * rel[0] - sn * rel[2]) + sn * vel[0] + cs * vel[2]
    ut = tip * apr + vel[1] * torch.sin(theta) - vz * torch.cos(theta)
    u2, phi = vx * vx + ut * ut, torch.atan(vx / ut)
    attack = phi * 180.0 / math.pi - (twist + pitch)
    at = torch.as_tensor(alm.stations["attack"], device=dev)
    na = len(at)
    lo = (torch.searchsorted(at, attack.detach().contiguous(), right=True) - 1).clamp(0, na - 2)
    f = ((attack - at[lo]) / (at[lo + 1] - at[lo])).clamp(0.0, 1.0)
    pts = torch.arange(n, device=dev)
    polar = lambda k: torch.as_tensor(alm.aps[k], device=dev).view(na, n)  # noqa: E731
    cl, cd = ((1 - f) * polar(k)[lo, pts] + f * polar(k)[lo + 1, pts] for k in ("cl", "cd"))
    dr = (alm.radius - alm.hub_radius) / alm.n_ap_per_blade
    lift, drag = 0.5 * cl * u2 * chord * dr, 0.5 * cd * u2 * chord * dr
    fx = lift * torch.cos(phi) + drag * torch.sin(phi)
    ft = (lift - drag) * torch.sin(phi) * math.copysign(1.0, tip)
    fr = (-fx, ft * torch.sin(theta), -ft * torch.cos(theta))
    force = (cs * fr[0] + sn * fr[2], fr[1], -sn * fr[0] + cs * fr[2])
    return pos, force, ft.abs() * apr, fx


def _spread(m, alm, pos, force):
    """Gaussian projection onto the interior, truncated at six widths"""
    eps = alm.euler_eps
    eta, cut = 1.0 / (math.sqrt(math.pi) * eps) ** 3, 6.0 * eps
    ff = torch.zeros((3,) + m.shape, dtype=torch.float64, device="cuda")
    xyz = [p.detach().cpu().numpy() for p in pos]
    tables = [m.grid.x, m.grid.y, m.grid.z]
    for a in range(len(xyz[0])):
        lo = [max(GC, int(np.searchsorted(tables[d], xyz[d][a] - cut))) for d in range(3)]
        hi = [min(m.dims[d] - GC, int(np.searchsorted(tables[d], xyz[d][a] + cut, side="right"))) for d in range(3)]
        if any(h <= l for l, h in zip(lo, hi)):
            continue
        r2 = sum((m.axis(m.x[d], d, lo, hi) - float(xyz[d][a])) ** 2 for d in range(3))
        w = torch.where(r2 < cut * cut, eta * torch.exp(-r2 / eps ** 2), 0.0)
        for d in range(3):
            ff[d][m.box(lo, hi)] += force[d][a] * w
    return ff


def _exact_step(case, setup, m, f):
    u, uu, p, nut, dt = f["u"], f["uu"], f["p"], f["nut"], setup.dt
    cavity = setup.bc == 1
    torque, thrust, ff = [], [], None
    if setup.alm is not None:
        pos, force, tq, th = _rotor(m, setup.alm, u, dt)
        ff = _spread(m, setup.alm, pos, force)
        torque, thrust = [float(tq.sum())], [float(th.sum())]
    ua = _pseudo(m, u, uu, nut, ff, setup.Re, dt, setup.adv)
    del ff
    uu = _face_velocity(m, ua, uu, cavity)
    op = _Poisson(m, setup.bc)
    op.bicgstab(p, _divergence(m, uu) / (dt * op.maxdiag), setup.tol, setup.maxit)
    p = _pbc(m, p, setup.bc)
    new, uu = _project(m, u, ua, uu, p, dt)
    _ubc_cavity(m, new) if cavity else _ubc_channel(m, new, u, dt, _inlet(setup, f["box"], dt, u))
    return {"u": new, "uu": uu, "p": p, "nut": _smagorinsky(m, new, nut, setup.Cs), "torque": torque, "thrust": thrust}


def _exact_operators(case, setup, m, f):
    u, uu, p, nut, dt = f["u"], f["uu"], f["p"], f["nut"], setup.dt
    out = {}
    zero = torch.zeros_like(u)
    ff = zero
    if setup.alm is not None:
        pos, force, tq, th = _rotor(m, setup.alm, u, dt)
        ff = _spread(m, setup.alm, pos, force)
        out["torque"], out["thrust"] = [np.array([float(v.sum())]) for v in (tq, th)]
    ua = zero.clone()
    ua[m.inner] = _pseudo(m, u, uu, nut, ff, setup.Re, dt, setup.adv)[m.inner]
    uu1 = _face_velocity(m, ua, zero, False)
    op = _Poisson(m, setup.bc)
    u2, uu2 = _project(m, zero, ua, uu1, p, dt)
    _ubc_cavity(m, u2) if setup.bc == 1 else _ubc_channel(m, u2, u, dt, _inlet(setup, f["box"], dt, u))
    return dict(out, ff=ff, ua=ua, uu1=uu1, rhs=_embed(m, _divergence(m, uu1) / (dt * op.maxdiag)), u2=u2, uu2=uu2, nut2=_smagorinsky(m, u2, torch.zeros_like(p), setup.Cs),
                div=_embed(m, _divergence(m, uu2)))


def _embed(m, v):
    out = torch.zeros(m.shape, dtype=torch.float64, device=v.device)
    out[m.inner] = v
    return out


def _exact_adjoint(case, setup, m, f):
    """reverse-mode differentiation of the step's stages, the solve taken as exact"""
    alm, dt, t = setup.alm, setup.dt, setup.dt
    u, uu, nut = (f[k].clone().requires_grad_() for k in ("u", "uu", "nut"))
    table = [torch.tensor(alm.pitch, dtype=torch.float64, device="cuda").requires_grad_(),
             torch.as_tensor(alm.aps["chord"], device="cuda").clone().requires_grad_(),
             torch.as_tensor(alm.aps["twist"], device="cuda").clone().requires_grad_()]
    pos, force, tq, _ = _rotor(m, alm, u, t, table)
    ua = _pseudo(m, u, uu, nut, _spread(m, alm, pos, force), setup.Re, dt, setup.adv)
    uu1 = _face_velocity(m, ua, uu, False)
    op = _Poisson(m, setup.bc)
    p = _pbc(m, _embed(m, _PressureOf.apply(_divergence(m, uu1) / (dt * op.maxdiag), op)), setup.bc)
    new, uu1 = _project(m, u, ua, uu1, p, dt)
    _ubc_channel(m, new, u, dt, _inlet(setup, f["box"], dt, new).detach())
    at = f["u_after"] + (new - new.detach())   # the eddy viscosity is linearised at the velocity given
    nut1 = _smagorinsky(m, at, nut, setup.Cs)
    goal = (f["au"] * new).sum() + (f["auu"] * uu1).sum() + (f["anut"] * nut1).sum() + W_POWER * float(alm.tip_rate[0]) * tq.sum()
    g = torch.autograd.grad(goal, [u, uu, nut] + table)
    return {"au": g[0], "auu": g[1], "anut": g[2], "grad": torch.cat([g[3].view(1), g[4], g[5]])}


def _exact_solve(case, setup, m, f):
    x = f["x0"].clone()
    op = _Poisson(m, setup.bc)
    mixed = case["precision"] == "mixed"
    b = f["b"][m.inner]
    # a mixed solve restarts from its true residual after each pass that misses the tolerance, five passes at most
    for _ in range(5 if mixed else 1):
        op.bicgstab(x, b, setup.tol, setup.maxit)
    return {"x": x, "r": _embed(m, b - op.apply(x))}


def exact(case, seed):
    setup = _setup(case)
    m = _Mesh(setup.grid)
    f = _inputs(case, seed, setup, m)
    out = {"step": _exact_step, "adjoint": _exact_adjoint, "operators": _exact_operators, "solve": _exact_solve}[case["kind"]](case, setup, m, f)
    return {k: v.reshape(-1) if isinstance(v, torch.Tensor) else v for k, v in out.items()}
