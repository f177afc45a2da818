"""Performance cases: the work a user of the engine has it do, through its public entry
points, over the sizes, forms and options it is used with.

A case is a dict of plain values; listed() gives the standing ones, draw(rng) one more of
the same ranges, prepare() what a program holds before the call, run() one pass of the
call, work() the bytes and operations it cannot do without, exact() the outputs in plain
64-bit torch.  Kinds:

  rhs        du = rhs!(u, t) on caller-owned device arrays (2D Euler, periodic cloud)
  rhs3d      the same on a periodic cube (3D Euler, plain flux divergence)
  igr        rhs! with the IGR source (a conjugate-gradient solve per evaluation)
  steps      solve() with SSP-RK3 and the HistoryCallback, host state in and out
  advance    a few more steps of a host-held state (pinned arrays, in place)
  channel    solve() with inlet, outlet and slip walls (the reference's boundary set-up)
  ensemble   solve() over independent clouds of different sizes in one context
  gradient   d loss(u(T)) / d u0 through torch.autograd (record and reverse sweep)
  stencils   k nearest neighbours and first-derivative weights of a new cloud
  weights    one batch of uneven 2D and 3D weight systems (host arrays in and out)
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "meshfreetrixi.jl_gb300"))

import meshfree_gb300 as M  # noqa: E402
from meshfree_gb300 import _lib as L  # noqa: E402
from meshfree_gb300 import autodiff  # noqa: E402
from meshfree_gb300 import workloads as W  # noqa: E402

GAMMA = 1.4


def listed():
    return [
        # the reference's test clouds hold about 2,000 nodes: one evaluation from a host
        # loop, where launches and latency count
        dict(name="rhs_small", kind="rhs", nx=46, ny=46, k=35, deg=3, visc="rv", hv=True, prec="fp64"),
        # an odd, ragged size with another stencil, upwind viscosity, no hyperviscosity
        dict(name="rhs_odd", kind="rhs", nx=317, ny=211, k=24, deg=2, visc="upwind", hv=False, prec="fp64"),
        # the headline problem size: 1M nodes, residual viscosity and hyperviscosity
        dict(name="rhs_1m", kind="rhs", nx=1024, ny=1024, k=35, deg=3, visc="rv", hv=True, prec="fp64"),
        # time stepping of the vortex benchmark (262,144 nodes, residual viscosity)
        dict(name="steps_vortex", kind="steps", nx=512, ny=512, k=35, deg=3, hv=False, prec="fp64", nsteps=32),
        # the FP32-apply form on the 1M problem, a caller's loop that looks at the state
        # every eight steps
        dict(name="advance_1m_fp32", kind="advance", nx=1024, ny=1024, k=35, deg=3, hv=True, prec="fp32", nsteps=8),
        # the reference's boundary set-up: Dirichlet inlet (host callback), outlet, walls
        dict(name="channel", kind="channel", n=64, k=20, deg=3, nsteps=20),
        # 3D Euler on a cube of 64^3 nodes
        dict(name="rhs3d", kind="rhs3d", n=64, k=30, deg=2),
        # IGR regularisation of the vortex
        dict(name="igr", kind="igr", nx=512, ny=512, k=35, deg=3),
        # a parameter study: sixteen vortices of different sizes in one context
        dict(name="ensemble", kind="ensemble", members=16, lo=32, hi=160, k=35, deg=3, nsteps=16),
        # gradient of a density misfit with respect to the initial state
        dict(name="gradient", kind="gradient", nx=256, ny=256, k=35, deg=3, nsteps=20),
        # set-up of a new cloud: neighbours and weights
        dict(name="stencils", kind="stencils", nx=512, ny=512, k=35, deg=3),
        # mixed weight batch: boundary stencils of 40..60, a tenth in 3D with 60..90
        dict(name="weights", kind="weights", total=131072),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rhs", "rhs", "rhs", "steps", "advance", "channel", "rhs3d", "igr", "ensemble",
                       "gradient", "stencils", "weights"])
    k, deg = rng.choice([(35, 3), (35, 3), (28, 3), (24, 2), (20, 2)])
    if kind == "rhs":
        prec = rng.choice(["fp64", "fp64", "fp32"])
        return dict(kind=kind, nx=_log(rng, 33, 1000), ny=_log(rng, 33, 1000), k=k, deg=deg,
                    visc=rng.choice(["rv", "rv", "upwind", "none"]), hv=rng.random() < 0.5, prec=prec)
    if kind == "steps":
        return dict(kind=kind, nx=_log(rng, 33, 900), ny=_log(rng, 33, 900), k=k, deg=deg,
                    hv=rng.random() < 0.5, prec=rng.choice(["fp64", "fp64", "fp32"]),
                    nsteps=rng.randint(4, 32))
    if kind == "advance":
        return dict(kind=kind, nx=_log(rng, 33, 1000), ny=_log(rng, 33, 1000), k=k, deg=deg,
                    hv=rng.random() < 0.5, prec=rng.choice(["fp64", "fp32"]), nsteps=rng.randint(1, 8))
    if kind == "channel":
        return dict(kind=kind, n=_log(rng, 32, 250), k=rng.choice([20, 24, 35]), deg=3,
                    nsteps=rng.randint(4, 20))
    if kind == "rhs3d":
        return dict(kind=kind, n=_log(rng, 12, 64), k=rng.choice([24, 30, 35]), deg=2)
    if kind == "igr":
        return dict(kind=kind, nx=_log(rng, 33, 512), ny=_log(rng, 33, 512), k=k, deg=deg)
    if kind == "ensemble":
        return dict(kind=kind, members=rng.randint(2, 16), lo=32, hi=_log(rng, 40, 160), k=k, deg=deg,
                    nsteps=rng.randint(4, 16))
    if kind == "gradient":
        return dict(kind=kind, nx=_log(rng, 33, 256), ny=_log(rng, 33, 256), k=k, deg=deg,
                    nsteps=rng.randint(4, 20))
    if kind == "stencils":
        return dict(kind=kind, nx=_log(rng, 33, 512), ny=_log(rng, 33, 512), k=k, deg=deg)
    return dict(kind=kind, total=_log(rng, 2000, 131072))


# ------------------------------------------------------------------ inputs


def _cloud(c, seed):
    """Jittered nodes of the periodic box [0, nx h] x [0, ny h], h = 10 / max(nx, ny)."""
    nx, ny = c["nx"], c["ny"]
    h = 10.0 / max(nx, ny)
    pts, _ = W.jittered_grid(nx, ny, hi=(nx * h, ny * h), seed=1000 + seed)
    return pts, (nx * h, ny * h), h


def _waves(pts, per, seed):
    """A smooth periodic 2D Euler state: seeded density, velocity and pressure waves."""
    g = np.random.default_rng(seed)
    a = 2 * np.pi * pts / np.asarray(per)
    ph = g.uniform(0, 2 * np.pi, 8)
    amp = g.uniform(0.05, 0.2, 4)
    rho = 1.0 + amp[0] * np.sin(a[:, 0] + ph[0]) * np.cos(2 * a[:, 1] + ph[1])
    u = 0.5 + amp[1] * np.sin(a[:, 1] + ph[2]) * np.cos(a[:, 0] + ph[3])
    v = -0.3 + amp[2] * np.cos(2 * a[:, 0] + ph[4]) * np.sin(a[:, 1] + ph[5])
    p = 1.0 + amp[3] * np.sin(a[:, 0] + ph[6]) * np.sin(a[:, 1] + ph[7])
    e = p / (GAMMA - 1.0) + 0.5 * rho * (u * u + v * v)
    return np.ascontiguousarray(np.stack([rho, rho * u, rho * v, e]))


def _solver(c, dim=2, prec="fp64"):
    basis = M.PointCloudBasis(M.Point3D() if dim == 3 else M.Point2D(), c["deg"], nv=c["k"])
    return M.PointCloudSolver(basis, M.RBFFDEngineGB300(precision=prec))


def _euler(c, pts, per, prec, visc, hv, igr=None):
    solver = _solver(c, prec=prec)
    dom = M.PointCloudDomain(solver, pts, period=per)
    eq = M.CompressibleEulerEquations2D(GAMMA)
    src = M.SourceTerms()
    if visc == "rv":
        src["rv"] = M.SourceResidualViscosityTominec(solver, eq, dom)
    elif visc == "upwind":
        src["uw"] = M.SourceUpwindViscosityTominec(solver, eq, dom)
    if hv:
        src["hv"] = M.SourceHyperviscosityTominec(solver, eq, dom)
    if igr is not None:
        src["igr"] = M.SourceIGR(solver, eq, dom, alpha=igr)
    return M.SemidiscretizationHyperbolic(dom, eq, None, solver, source_terms=src)


def _channel(c, seed):
    """n x n jittered nodes on the unit square and n nodes on each edge; inlet left,
    outlet right, slip walls bottom and top."""
    pts, tags, h = W.advection_cloud(c["n"], seed=1000 + seed)
    (inflow, nin), (outflow, nout) = tags["inflow"], tags["outflow"]
    n = c["n"]
    bt = dict(inlet=M.BoundaryData(inflow[:n], nin[:n]), outlet=M.BoundaryData(outflow[:n], nout[:n]),
              bottom=M.BoundaryData(inflow[n:], nin[n:]), top=M.BoundaryData(outflow[n:], nout[n:]))
    return pts, bt, h


def _channel_state(pts, seed):
    """Flow along x with a transverse part that vanishes at the walls and a seeded smooth
    bump of density and pressure."""
    g = np.random.default_rng(seed)
    cx, cy = g.uniform(0.35, 0.65, 2)
    b = 0.2 * np.exp(-((pts[:, 0] - cx) ** 2 + (pts[:, 1] - cy) ** 2) / 0.02)
    rho, u, v, p = 1.0 + b, np.full(len(b), 0.4), 0.1 * np.sin(np.pi * pts[:, 1]), 1.0 + b
    return np.ascontiguousarray(np.stack([rho, rho * u, rho * v, p / (GAMMA - 1.0) + 0.5 * rho * (u * u + v * v)]))


_INLET = np.array([1.0, 0.4, 0.0, 1.0 / (GAMMA - 1.0) + 0.5 * 0.16])


def _members(c, seed):
    sides = np.random.default_rng(5).permutation(np.geomspace(c["lo"], c["hi"], c["members"]).round().astype(int))
    return [W.vortex_cloud(int(s), seed=1000 + 37 * seed + i) for i, s in enumerate(sides)]


def _batch(c, seed):
    """The two point clouds of a weight batch and their stencil sizes: 2D with k = 35, and
    40..60 for the 8 % nearest the square's edge; 3D with 60..90."""
    n3 = max(c["total"] // 10, 200)
    p2, p3 = W.halton_points(c["total"] - n3, 2, seed=seed), W.halton_points(n3, 3, seed=seed + 1)
    g = np.random.default_rng(5)
    k2, k3 = np.full(len(p2), 35), g.integers(60, 91, n3)
    edge = np.argsort(np.minimum(p2, 1 - p2).min(1), kind="stable")[:len(p2) * 8 // 100]
    k2[edge] = g.integers(40, 61, len(edge))
    return (p2, k2, 3), (p3, k3, 2)


def _ragged(idx, ks):
    keep = np.arange(idx.shape[1])[None, :] < ks[:, None]
    return np.concatenate([[0], np.cumsum(ks)]).astype(np.int64), idx[keep].astype(np.int32)


def prepare(case, seed):
    c, kind = case, case["kind"]
    dev = torch.device("cuda:0")
    if kind in ("rhs", "igr"):
        pts, per, h = _cloud(c, seed)
        visc, hv = (c["visc"], c["hv"]) if kind == "rhs" else ("none", False)
        semi = _euler(c, pts, per, c.get("prec", "fp64"), visc, hv, igr=h * h if kind == "igr" else None)
        u = _waves(pts, per, seed)
        if visc == "rv":  # the history's time derivative, as after a few accepted steps
            semi.domain.ctx.set_rv_state(_approx_du(u), 3)
        ut = torch.from_numpy(u).to(dev)
        return dict(kind=kind, semi=semi, u=ut, du=torch.empty_like(ut))
    if kind == "rhs3d":
        pts, _h = W.jittered_grid3(c["n"], seed=1000 + seed)
        solver = _solver(c, dim=3)
        dom = M.PointCloudDomain(solver, pts, period=(1.0, 1.0, 1.0))
        semi = M.SemidiscretizationHyperbolic(dom, M.CompressibleEulerEquations3D(GAMMA), None, solver)
        ut = torch.from_numpy(_state3(pts, seed)).to(dev)
        return dict(kind="rhs", semi=semi, u=ut, du=torch.empty_like(ut))
    if kind == "steps":
        pts, per, h = _cloud(c, seed)
        semi = _euler(c, pts, per, c["prec"], "rv", c["hv"])
        dt = 0.1 * h
        return dict(kind=kind, ode=M.ODEProblem(_waves(pts, per, seed), (0.0, c["nsteps"] * dt), semi), dt=dt)
    if kind == "advance":
        pts, per, h = _cloud(c, seed)
        semi = _euler(c, pts, per, c["prec"], "rv", c["hv"])
        semi.domain.ctx.history_init(3)
        u = torch.from_numpy(_waves(pts, per, seed)).pin_memory()
        return dict(kind=kind, semi=semi, u=u, t=0.0, dt=0.1 * h, nsteps=c["nsteps"])
    if kind == "channel":
        pts, bt, h = _channel(c, seed)
        solver = _solver(c)
        dom = M.PointCloudDomain(solver, pts, bt)
        eq = M.CompressibleEulerEquations2D(GAMMA)
        wall = M.boundary_condition_slip_wall
        bcs = dict(inlet=M.BoundaryConditionDirichlet(lambda x, t, e: np.tile(_INLET, (len(x), 1))),
                   outlet=M.BoundaryConditionDoNothing(), bottom=wall, top=wall)
        src = M.SourceTerms(rv=M.SourceResidualViscosityTominec(solver, eq, dom),
                            hv=M.SourceHyperviscosityTominec(solver, eq, dom))
        semi = M.SemidiscretizationHyperbolic(dom, eq, None, solver, bcs, src)
        dt = 0.05 * h
        return dict(kind="steps", ode=M.ODEProblem(_channel_state(pts, seed), (0.0, c["nsteps"] * dt), semi),
                    dt=dt)
    if kind == "ensemble":
        clouds = _members(c, seed)
        solver = _solver(c)
        dom = M.PointCloudEnsemble(solver, [x[0] for x in clouds], period=clouds[0][1])
        eq = M.CompressibleEulerEquations2D(GAMMA)
        src = M.SourceTerms(rv=M.SourceResidualViscosityTominec(solver, eq, dom))
        semi = M.SemidiscretizationHyperbolic(dom, eq, None, solver, source_terms=src)
        dt = 0.1 * min(x[2] for x in clouds)
        u0 = np.ascontiguousarray(np.concatenate([W.isentropic_vortex(x[0], 0.0) for x in clouds], axis=1))
        return dict(kind="steps", ode=M.ODEProblem(u0, (0.0, c["nsteps"] * dt), semi), dt=dt)
    if kind == "gradient":
        pts, per, h = _cloud(c, seed)
        semi = _euler(c, pts, per, "fp64", "none", False)
        u0 = torch.from_numpy(_waves(pts, per, seed)).to(dev)
        target = torch.from_numpy(_waves(pts, per, seed + 1)[0]).to(dev)
        return dict(kind=kind, semi=semi, u0=u0, target=target, dt=0.1 * h, nsteps=c["nsteps"])
    if kind == "stencils":
        pts, per, _h = _cloud(c, seed)
        return dict(kind=kind, ctx=L.Context(0), pts=pts, per=per, k=c["k"], deg=c["deg"])
    groups = []
    for pts, ks, deg in _batch(c, seed):
        ctx = L.Context(0)
        ctx.set_points(pts)
        rp, cols = _ragged(ctx.knn(int(ks.max()))[0], ks)
        groups.append((pts, rp, cols, 3, deg, 1))
        if pts.shape[1] == 2:
            keep = ctx
        else:
            ctx.close()
    return dict(kind=kind, ctx=keep, groups=groups)


def run(state):
    kind = state["kind"]
    if kind in ("rhs", "igr"):
        state["semi"].domain.ctx.rhs_device(state["du"].data_ptr(), state["u"].data_ptr(), 0.0)
        return state["du"]
    if kind == "steps":
        sol = M.solve(state["ode"], M.SSPRK33(), dt=state["dt"], callback=M.HistoryCallback(3))
        return sol.u, sol.t
    if kind == "advance":
        u = state["u"].numpy()
        state["t"] = state["semi"].domain.ctx.ssprk33_host(u, state["t"], state["dt"], state["nsteps"])
        return u
    if kind == "gradient":
        u0 = state["u0"].clone().requires_grad_(True)
        uT = autodiff.ssprk33_solve(u0, state["semi"], 0.0, state["dt"], state["nsteps"])
        loss = 0.5 * (uT[0] - state["target"]).square().sum()
        loss.backward()
        return uT.detach(), u0.grad
    if kind == "stencils":
        ctx = state["ctx"]
        ctx.set_points(state["pts"], state["per"])
        idx, dist, dmin, davg = ctx.knn(state["k"], want_dist=True)
        w, _ = ctx.weights(L.OP_GRAD, 3, state["deg"], 1, want_w=True)
        return idx, dist, dmin, davg, w
    (w2, w3), _ = state["ctx"].weights_batch(state["groups"])
    return w2, w3


# ------------------------------------------------------------------ necessary work


def _npoly(deg, dim):
    return math.comb(deg + dim, dim)


def work(case):
    """bytes: operator values and indices once per evaluation, states, results; flops: two
    per product of a weight with a flux or state (per system: the factorisation)."""
    c, kind = case, case["kind"]
    k = c.get("k", 0)
    if kind in ("rhs", "steps", "advance", "channel", "ensemble", "igr", "gradient"):
        s = 4 if c.get("prec") == "fp32" else 8
        if kind == "channel":
            n = c["n"] ** 2 + 4 * c["n"]
        elif kind == "ensemble":
            n = c["members"] * 0.5 * (c["hi"] ** 2 - c["lo"] ** 2) / math.log(c["hi"] / c["lo"])
        else:
            n = c["nx"] * c["ny"]
        visc = {"rhs": c.get("visc"), "igr": "none", "gradient": "none"}.get(kind, "rv")
        hv = bool(c.get("hv")) or kind == "channel"
        per = k * (4 + 2 * s + (s if hv else 0)) + 64 + (32 if visc == "rv" else 0)
        prod = 8 * k + (16 * k if visc != "none" else 0) + (8 * k if hv else 0)
        if kind == "igr":
            return dict(bytes=n * (per + 20 * 2 * (k * 20 + 24)), flops=n * 2 * (prod + 20 * 4 * k + 7 * k))
        evals = 1 if kind == "rhs" else 3 * c["nsteps"] * (2 if kind == "gradient" else 1)
        return dict(bytes=n * per * evals, flops=n * 2 * prod * evals)
    if kind == "rhs3d":
        n = c["n"] ** 3
        return dict(bytes=n * (k * 28 + 80), flops=n * 30 * k)
    if kind == "stencils":
        n, m = c["nx"] * c["ny"], k + _npoly(c["deg"], 2)
        return dict(bytes=n * (16 + 12 * k + 16 * k), flops=n * (m ** 3 / 3 + 4 * m * m))
    n3 = max(c["total"] // 10, 200)
    n2, m2, m3 = c["total"] - n3, 46.5, 85.0
    return dict(bytes=n2 * 36.5 * 20 + n3 * 75 * 28,
                flops=n2 * (m2 ** 3 / 3 + 4 * m2 ** 2) + n3 * (m3 ** 3 / 3 + 6 * m3 ** 2))


def _approx_du(u):
    """A stand-in for the history's du/dt: smooth, of the size of the flux divergence."""
    return np.ascontiguousarray(0.1 * np.roll(u, 1, axis=0) - 0.05)


def _state3(pts, seed):
    u = W.euler3d_wave(pts)
    g = np.random.default_rng(seed)
    return np.ascontiguousarray(u * (1.0 + 0.01 * np.sin(2 * np.pi * pts[:, 0] + g.uniform(0, 6, (5, 1)))))


# ------------------------------------------------------------------ 64-bit results


def _dev():
    return torch.device("cuda:0" if torch.cuda.is_available() else "cpu")


def _wrap(d, per):
    return d if per is None else d - per * torch.round(d / per)


def _neighbours(pts, kmax, per=None, grid=None):
    """k nearest nodes by (distance, index) and squared distances, in row chunks.  grid:
    lattice shape (x fastest) of a jittered periodic lattice, whose candidates are the
    lattice points near each node; else all nodes are candidates."""
    n, dim = pts.shape
    off = None
    if grid is not None and min(grid) >= 11:
        r = 5 if dim == 2 else 3
        axes = [torch.arange(-r, r + 1, device=pts.device)] * dim
        off = torch.cartesian_prod(*axes)
    idx, d2 = [], []
    step = max(1, int(6e7) // (len(off) if off is not None else n))
    for a in range(0, n, step):
        i = torch.arange(a, min(n, a + step), device=pts.device)
        if off is not None:
            cand, mul, rest = torch.zeros(len(i), len(off), dtype=torch.int64, device=pts.device), 1, i
            for d in range(dim):
                cand += (rest % grid[d])[:, None].add(off[:, d]).remainder(grid[d]) * mul
                mul, rest = mul * grid[d], rest // grid[d]
        else:
            cand = None
        s = 0
        for d in range(dim):
            q = (pts[cand, d] if cand is not None else pts[None, :, d]) - pts[i, d][:, None]
            q = _wrap(q, None if per is None else per[d])
            s = s + q * q
        v, j = torch.topk(s, kmax, dim=1, largest=False, sorted=True)
        d2.append(v)
        idx.append(j if cand is None else torch.gather(cand, 1, j))
    return torch.cat(idx), torch.cat(d2)


def _solve_weights(pts, nb, per, deg, orders):
    """First (1) and second (2) derivative weights of PHS r^3 + degree-deg polynomials for
    stencils nb (n, k): a list of (n, k, dim), by dense solves in the scaled coordinates."""
    n, k = nb.shape
    dim = pts.shape[1]
    mono = [e for e in _exponents(dim, deg)]
    m = k + len(mono)
    outs = [torch.empty(n, k, dim, dtype=torch.float64, device=pts.device) for _ in orders]
    step = max(1, int(2.5e8) // (m * m))
    for a in range(0, n, step):
        b = min(n, a + step)
        x = pts[nb[a:b]] - pts[nb[a:b, :1]]
        if per is not None:
            x = torch.stack([_wrap(x[..., d], per[d]) for d in range(dim)], -1)
        s = 1.0 / x.abs().amax(1)
        x = x * s[:, None, :]
        A = torch.zeros(b - a, m, m, dtype=torch.float64, device=pts.device)
        A[:, :k, :k] = (x[:, :, None] - x[:, None]).square().sum(-1).sqrt().pow(3)
        P = torch.stack([torch.stack([x[..., d] ** e[d] for d in range(dim)]).prod(0) for e in mono], -1)
        A[:, :k, k:] = P
        A[:, k:, :k] = P.transpose(1, 2)
        r = x.square().sum(-1).sqrt()
        B = torch.zeros(b - a, m, dim * len(orders), dtype=torch.float64, device=pts.device)
        for q, o in enumerate(orders):
            for d in range(dim):
                col = q * dim + d
                B[:, :k, col] = -3 * r * x[..., d] if o == 1 else torch.where(
                    r > 0, 3 * r + 3 * x[..., d] ** 2 / r.clamp_min(1e-300), torch.zeros_like(r))
                for p, e in enumerate(mono):
                    if sum(e) == o and e[d] == o:
                        B[:, k + p, col] = math.factorial(o)
        w = torch.linalg.solve(A, B)[:, :k]
        for q, o in enumerate(orders):
            outs[q][a:b] = w[..., q * dim:(q + 1) * dim] * (s ** o)[:, None, :]
    return outs


def _exponents(dim, deg):
    grids = np.stack(np.meshgrid(*[np.arange(deg + 1)] * dim, indexing="ij"), -1).reshape(-1, dim)
    return [tuple(int(v) for v in e) for e in grids if e.sum() <= deg]


class _Exact:
    """rhs! of the Euler equations on one cloud, from the definitions, in float64 torch."""

    def __init__(self, pts, k, deg, per=None, grid=None, visc="none", hv=False, bcs=None):
        dev = _dev()
        x = torch.from_numpy(pts).to(dev)
        self.nb, d2 = _neighbours(x, k, per, grid)
        near = d2[:, 1].sqrt()
        self.h, self.gam = float(near.mean()), float(near.min()) ** 4.5
        ws = _solve_weights(x, self.nb, per, deg, (1, 2) if hv else (1,))
        self.D = ws[0].unbind(-1)
        self.lap = ws[1].sum(-1) if hv else None
        self.visc, self.bcs = visc, bcs
        self.approx_du, self.si, self.n = None, 0, len(pts)

    def apply(self, w, f):
        return (w * f[..., self.nb]).sum(-1)

    def transpose(self, w, s):
        out = torch.zeros_like(s)
        return out.index_add_(-1, self.nb.reshape(-1), (w * s[..., None]).reshape(*s.shape[:-1], -1))

    def _bc(self, u, du=None):
        """The strong BC pass: on the state, and on du after the sources."""
        if self.bcs is None:
            return
        inlet, walls = self.bcs
        u[:, inlet] = torch.from_numpy(_INLET).to(u)[:, None]
        u[2, walls] = 0.0
        if du is not None:
            du[:, inlet] = 0.0
            du[1:3, walls] = 0.0

    def rhs(self, u):
        self._bc(u)
        g, dim = GAMMA, len(self.D)
        rho, m, en = u[0], u[1:1 + dim], u[1 + dim]
        v = m / rho
        p = (g - 1) * (en - 0.5 * (m * v).sum(0))
        du = 0
        for d in range(dim):
            rows = [m[d]] + [m[a] * v[d] + p if a == d else m[a] * v[d] for a in range(dim)] + [(en + p) * v[d]]
            du = du - torch.stack([self.apply(self.D[d], r) for r in rows])
        if self.visc != "none":
            eps = 0.5 * self.h * (v.square().sum(0).sqrt() + (g * p / rho).sqrt())
            if self.visc == "rv" and self.si:
                y = (u - u.sum(1, keepdim=True) / (self.n * len(u))).abs()
                ok = torch.ones_like(y[0], dtype=torch.bool)
                for a in range(len(u)):  # the lexicographic maximum of the nodes' vectors
                    ok &= y[a] == y[a][ok].max()
                norm = y[:, ok][:, :1]
                eps = torch.minimum(0.5 * self.h ** 2 * ((self.approx_du - du).abs() / norm).amax(0), eps)
            part = [torch.stack([self.apply(w, u[a]) for a in range(len(u))]) * eps for w in self.D]
            du = du - sum(self.transpose(w, s) for w, s in zip(self.D, part))
        if self.lap is not None:
            q = torch.stack([self.apply(self.lap, u[a]) for a in range(len(u))])
            du = du - self.gam * self.transpose(self.lap, q)
        self._bc(u, du)
        return du

    def solve(self, u, dt, nsteps, history=True):
        """SSP-RK3 with first-same-as-last and the order-3 history."""
        hist = [(0.0, u)]
        k = self.rhs(u)
        for step in range(nsteps):
            un = u
            u = un + dt * k
            u = (3 * un + u + dt * self.rhs(u)) / 4
            u = (un + 2 * u + 2 * dt * self.rhs(u)) / 3
            k = self.rhs(u)
            if history:
                hist = ([((step + 1) * dt, u.clone())] + hist)[:4]
                t = np.array([x[0] for x in hist])
                z = (t - t[0]) / dt
                w = np.linalg.solve(np.vander(z, increasing=True).T, np.eye(len(t))[1]) / dt
                self.approx_du, self.si = sum(a * x for a, (_, x) in zip(w, hist)), step + 1
        return u


def _exact_igr(e, u, alpha, maxiter=20):
    """du of rhs! with the IGR source: conjugate gradients from zero."""
    du, (dx, dy) = e.rhs(u), e.D
    rho, v1, v2 = u[0], u[1] / u[0], u[2] / u[0]
    A = lambda w, f: e.apply(w, f)  # noqa: E731
    tr = A(dx, rho) + A(dy, v1)
    b = alpha * (tr ** 2 + A(dx, v1) ** 2 + 2 * A(dy, v1) * A(dx, v2) + A(dy, v2) ** 2)
    x, r, p = torch.zeros_like(b), b.clone(), torch.zeros_like(b)
    res, prev = r.norm(), torch.ones_like(b[0])
    tol, it = math.sqrt(2.0 ** -52) * res, 0
    while it < maxiter and res > tol:
        p = r + (res / prev) ** 2 * p
        c = p / rho - alpha * (A(dx, A(dx, p) / rho) + A(dy, A(dy, p) / rho))
        a = res ** 2 / (p * c).sum()
        x, r = x + a * p, r - a * c
        prev, res, it = res, r.norm(), it + 1
    du[1] -= A(dx, x)
    du[2] -= A(dy, x)
    return du


def exact(case, seed):
    c, kind = case, case["kind"]
    dev = _dev()
    up = lambda a: torch.from_numpy(a).to(dev)  # noqa: E731
    if kind in ("rhs", "steps", "advance", "igr", "gradient"):
        pts, per, h = _cloud(c, seed)
        visc = "rv" if kind in ("steps", "advance") else c.get("visc", "none")
        e = _Exact(pts, c["k"], c["deg"], per, (c["nx"], c["ny"]), visc, c.get("hv", False))
        u = up(_waves(pts, per, seed))
        if kind == "igr":
            return _exact_igr(e, u, h * h)
        if kind == "rhs":
            e.approx_du, e.si = up(_approx_du(u.cpu().numpy())), 3
            return e.rhs(u)
        dt = 0.1 * h
        if kind in ("steps", "advance"):
            uT = e.solve(u, dt, c["nsteps"]).cpu()
            return (uT, c["nsteps"] * dt) if kind == "steps" else uT
        u.requires_grad_(True)
        uT = e.solve(u, dt, c["nsteps"], history=False)
        (0.5 * (uT[0] - up(_waves(pts, per, seed + 1)[0])).square().sum()).backward()
        return uT.detach(), u.grad
    if kind == "rhs3d":
        pts, _h = W.jittered_grid3(c["n"], seed=1000 + seed)
        e = _Exact(pts, c["k"], c["deg"], (1.0,) * 3, (c["n"],) * 3)
        return e.rhs(up(_state3(pts, seed)))
    if kind == "channel":
        pts, bt, h = _channel(c, seed)
        walls = np.concatenate([bt["bottom"].idx, bt["top"].idx])
        e = _Exact(pts, c["k"], c["deg"], visc="rv", hv=True, bcs=(up(bt["inlet"].idx), up(walls)))
        return e.solve(up(_channel_state(pts, seed)), 0.05 * h, c["nsteps"]).cpu(), c["nsteps"] * 0.05 * h
    if kind == "ensemble":
        clouds = _members(c, seed)
        dt, outs = 0.1 * min(x[2] for x in clouds), []
        for pts, per, _h in clouds:
            side = int(round(math.sqrt(len(pts))))
            e = _Exact(pts, c["k"], c["deg"], per, (side, side), "rv")
            outs.append(e.solve(up(W.isentropic_vortex(pts, 0.0)), dt, c["nsteps"]).cpu())
        return torch.cat(outs, 1), c["nsteps"] * dt
    if kind == "stencils":
        pts, per, _h = _cloud(c, seed)
        x = up(pts)
        nb, d2 = _neighbours(x, c["k"], per, (c["nx"], c["ny"]))
        d = d2.sqrt()
        w = _solve_weights(x, nb, per, c["deg"], (1,))[0]
        return (None, d.cpu(), float(d[:, 1].min()), float(d[:, 1].mean()), w.reshape(-1, 2).cpu())
    outs = []
    for pts, ks, deg in _batch(c, seed):
        x = up(pts)
        nb, _ = _neighbours(x, int(ks.max()))
        rp = np.concatenate([[0], np.cumsum(ks)])
        w = np.empty((rp[-1], pts.shape[1]))
        for k in np.unique(ks):
            rows = np.nonzero(ks == k)[0]
            v = _solve_weights(x, nb[up(rows)][:, :int(k)], None, deg, (1,))[0].cpu().numpy()
            w[(rp[rows][:, None] + np.arange(k)).reshape(-1)] = v.reshape(-1, pts.shape[1])
        outs.append(w)
    return tuple(outs)
