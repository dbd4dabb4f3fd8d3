"""The workloads the speed of this framework is judged by.

Each case is one pass of a program that uses the package through its public
entry points (:class:`Context`, :class:`Batch`).  The flows, sizes and solver
settings are those of ``configs.py``, ``bench.py``, ``ensemble.py`` and the
tests: the lid-driven cavity, the static droplet, the rising bubble and the
two-phase channel, on grids from 32 x 32 to 768 x 768, in FP64 and in the
mixed form, with the solver settings the configurations use and with the
reference's own solver.

A time-stepping pass resumes a run: it uploads the state a checkpoint holds
(velocity, pressure, colour, previous velocity), takes a few steps on the
device and downloads the resulting state.  So every pass does the same work
and the copies are a small part of it.

``listed`` names the cases, ``draw`` makes more of the same ranges,
``prepare`` makes what a program has in hand before the call, ``run`` is one
pass, ``work`` the bytes and operations it cannot do without and ``exact``
the 64-bit value of the outputs where plain numpy gives it.
"""
from __future__ import annotations

import math

import numpy as np

from coupled_codefort_2d_b200 import cases
from coupled_codefort_2d_b200._lib import FIELD_KIND, FP64, MIXED
from coupled_codefort_2d_b200.batch import Batch, ensemble_params, initial_bubble_state
from coupled_codefort_2d_b200.context import Context
from coupled_codefort_2d_b200.layout import Grid, at
from coupled_codefort_2d_b200.params import Params

# the state of a checkpoint and the state a program looks at after its steps
CHECKPOINT = ("u_vel", "v_vel", "p_field", "c_field", "u_prev", "v_prev")
RESULT = ("u_vel", "v_vel", "p_field", "c_field")
STATE = CHECKPOINT + ("rho_c", "rho_u", "rho_v", "kappa", "zeta", "eta", "kappa_curv", "f_sigma_u", "f_sigma_v")

# flexible GMRES inside the FP64 defect correction, as the configurations and
# the benchmark set it; the bubble adds the red-black smoother
FAST = dict(refine=2, refine_inner_tol=1e-2, refine_max_inner=30, refine_max_outer=60, krylov_bc_fix=1,
            pcg_cap_start=80, pcd_sweeps=6, pcd_sweeps_max=24, pcd_visc_scale=1.0, graphs=1)
BUBBLE = dict(FAST, pcd_smoother=1, pcd_sor_omega=1.5)
# the ensemble's settings (ensemble.SOLVER) and the gradient runs' (adjoint.RisingBubble)
ENSEMBLE = dict(BUBBLE, pcg_cap_start=40, tol_bicgstab2=1e-8, max_iter_bicgstab2=500)
GRADIENT = dict(refine=2, refine_inner_tol=1e-2, refine_max_inner=30, refine_max_outer=100, krylov_bc_fix=1,
                svof_tol=0.0)


def listed():
    return [
        # the smallest call: one coupled operator on a small box, as a host code calls it
        dict(name="matvec_32", kind="matvec", nx=32, ny=32),
        # colour transport, filter, curvature and force of one step, called routine by routine
        dict(name="transport_256", kind="transport", nx=256, ny=256),
        # the pressure Poisson solve of a projection code, FP64, an odd size
        dict(name="poisson_203x125", kind="poisson", nx=203, ny=125),
        # the reference's own solver and defaults on the size of its tests
        dict(name="plain_droplet_64", kind="steps", flow="droplet", solver="plain", nx=64, ny=64, mixed=False, steps=2),
        # lid-driven cavity, FP64 to 1e-10 (configs c1)
        dict(name="cavity_128_fp64", kind="steps", flow="cavity", solver="fast", nx=128, ny=128, mixed=False, steps=3),
        # the benchmark's droplet (configs c2) in both precisions
        dict(name="droplet_256_mixed", kind="steps", flow="droplet", solver="fast", nx=256, ny=256, mixed=True,
             steps=4),
        dict(name="droplet_256_fp64", kind="steps", flow="droplet", solver="fast", nx=256, ny=256, mixed=False,
             steps=2),
        # a Fortran host's drop-in call: all state arrays up and down on every step
        dict(name="dropin_bubble_64x128", kind="dropin", flow="bubble", solver="fast", nx=64, ny=128, mixed=True),
        # the rising bubble of configs c3
        dict(name="bubble_320x640_mixed", kind="steps", flow="bubble", solver="fast", nx=320, ny=640, mixed=True,
             steps=2),
        # the droplet on a large box (configs scale)
        dict(name="droplet_768_mixed", kind="steps", flow="droplet", solver="fast", nx=768, ny=768, mixed=True,
             steps=1),
        # a shard of the ensemble (configs c4): many uneven cases on one GPU
        dict(name="ensemble_16", kind="batch", cases=16, steps=2, lockstep=False),
        # the gradient of one rising-bubble step (configs c5), at its smaller size
        dict(name="vjp_80x160", kind="vjp", nx=80, ny=160),
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["matvec", "transport", "poisson", "steps", "steps", "steps", "steps", "steps", "dropin",
                       "batch", "vjp"])
    if kind in ("matvec", "transport"):
        return dict(kind=kind, nx=_size(rng, 32, 640), ny=_size(rng, 32, 640))
    if kind == "poisson":
        return dict(kind=kind, nx=_size(rng, 48, 400), ny=_size(rng, 48, 400))
    if kind == "batch":
        return dict(kind=kind, cases=rng.randint(4, 16), steps=rng.randint(1, 2), lockstep=rng.random() < 0.3)
    if kind == "vjp":
        nx = _size(rng, 32, 80)
        return dict(kind=kind, nx=nx, ny=2 * nx + rng.randint(0, 3))
    flow = rng.choice(["cavity", "droplet", "bubble", "channel"])
    if kind == "dropin":
        n = _size(rng, 32, 256)
        return dict(kind=kind, flow=flow, solver="fast", nx=n, ny=2 * n if flow == "bubble" else n,
                    mixed=rng.random() < 0.6)
    plain = rng.random() < 0.15
    n = _size(rng, 32, 96) if plain else _size(rng, 48, 640)
    mixed = not plain and rng.random() < 0.6
    ny = 2 * n if flow == "bubble" and n <= 320 else n + rng.randint(-8, 8)
    return dict(kind="steps", flow=flow, solver="plain" if plain else "fast", nx=n, ny=ny, mixed=mixed,
                steps=rng.randint(1, 4) if n < 400 else 1)


# ------------------------------------------------------------------ inputs
def _grid(case):
    nx, ny, flow = case["nx"], case["ny"], case.get("flow")
    if flow == "channel":
        return Grid(nx, ny, periodic_x=True)
    if flow == "bubble" or case["kind"] == "vjp":
        return Grid(nx, ny, 1.0, ny / nx)
    return Grid(nx, ny)


def _flow(case):
    """Physics, time step, lid and boundaries of a flow (configs.py)."""
    flow = case.get("flow", "droplet")
    if flow == "cavity":
        return dict(rho1=1.0, rho2=1.0, mu1=1e-3, mu2=1e-3, sigma=0.0, gx=0.0, gy=0.0, time_order=1,
                    tol_bicgstab2=1e-10), 1e-2 * 128 / max(128, case["nx"]), 1.0
    if flow == "bubble":
        return dict(rho1=1000.0, rho2=100.0, mu1=10.0, mu2=1.0, sigma=24.5, gx=0.0, gy=-0.98, time_order=2,
                    free_slip_x=1, tol_bicgstab2=1e-8), 5e-4, None
    if flow == "channel":
        return dict(rho1=1.0, rho2=1.0, mu1=1.0, mu2=0.1, sigma=0.0, gx=1.0, gy=0.0, time_order=2,
                    tol_bicgstab2=1e-8), 1e-3, None
    return dict(rho1=1.0, rho2=0.1, mu1=0.1, mu2=0.01, sigma=1.0, gx=0.0, gy=0.0, time_order=2,
                tol_bicgstab2=1e-8), 1e-4, None


def _params(case):
    phys, dt, lid = _flow(case)
    if case.get("solver") == "plain":  # the reference's algorithm and tolerance (params.py's defaults)
        phys = dict(phys, tol_bicgstab2=1e-6)
        return Params(max_iter_bicgstab2=60, **phys), dt, lid
    solver = BUBBLE if case.get("flow") == "bubble" else FAST
    return Params(max_iter_bicgstab2=500, **phys, **solver), dt, lid


def _colour(case, g, rng):
    flow = case.get("flow", "droplet")
    if flow == "cavity":
        return g.full("cell", 1.0)
    if flow == "channel":
        return cases.poiseuille_layers(g)
    xc, r = 0.5 + 0.02 * rng.uniform(-1, 1), 0.25 + 0.01 * rng.uniform(-1, 1)
    if flow == "bubble":
        return cases.binary_circle(g, xc, 0.5, r, inside=0.0)
    return cases.circle_fraction(g, xc, 0.5 + 0.02 * rng.uniform(-1, 1), r, inside=1.0, ns=4)


def _velocity(case, g, rng):
    """A smooth solenoidal field: face differences of a vertex stream function
    that vanishes on the walls, a few seeded modes, of the size the flow has
    after some steps."""
    i, j = np.arange(-2, g.nx + 3) / g.nx, np.arange(-2, g.ny + 3) / g.ny
    X, Y = np.meshgrid(i, j, indexing="ij")
    psi = np.zeros_like(X)
    for m in (1, 2, 3):
        for n in (1, 2, 3):
            a, ph = rng.standard_normal() / (m * n), rng.uniform(0, 2 * np.pi)
            sx = np.cos(2 * np.pi * m * X + ph) if g.periodic_x else np.sin(np.pi * m * X) * np.sin(np.pi * X)
            psi += a * sx * np.sin(np.pi * n * Y) * np.sin(np.pi * Y)
    size = {"cavity": 0.1, "droplet": 0.02, "bubble": 0.05, "channel": 0.05}[case.get("flow", "droplet")]
    psi *= size / (2 * np.pi)
    u, v = g.zeros("u"), g.zeros("v")
    u[:, :] = (psi[:, 1:] - psi[:, :-1]) / g.dy
    v[:, :] = -(psi[1:, :] - psi[:-1, :]) / g.dx
    return u, v


def _pressure(phys, c, g):
    """The pressure the step before left, near enough: hydrostatic in the
    outer fluid and the capillary jump across a circle of radius 0.25."""
    j = np.arange(-1, g.ny + 3, dtype=np.float64)
    y = ((j - 0.5) * g.dy)[None, :]
    inside = 1.0 - c if phys["gy"] else c
    return phys["rho1"] * phys["gy"] * (y - g.Ly) + 4.0 * phys["sigma"] * inside


def _state(case, g, ctx, lid, seed):
    rng = np.random.default_rng(seed)
    st = {k: g.zeros(FIELD_KIND[k]) for k in STATE}
    st["c_field"][...] = _colour(case, g, rng)
    st["p_field"][...] = _pressure(_flow(case)[0], st["c_field"], g)
    for pair in (("u_vel", "v_vel"), ("u_prev", "v_prev")):
        st[pair[0]][...], st[pair[1]][...] = _velocity(case, g, np.random.default_rng(seed + 1))
        if g.periodic_x:
            ctx.halo("u", st[pair[0]])
            ctx.halo("v", st[pair[1]])
        ctx.apply_velocity_bcs(st[pair[0]], st[pair[1]], lid)
    return st


def _random(rng, g, kind, lo=-1.0, hi=1.0):
    return np.asfortranarray(rng.uniform(lo, hi, g.shape(kind)))


def prepare(case, seed):
    kind, rng = case["kind"], np.random.default_rng(seed)
    if kind == "batch":
        specs = cases.bubble_ensemble(case["cases"])
        for s in specs:  # the same cases with other bubbles
            s["radius"] *= 1.0 + 0.05 * rng.uniform(-1, 1)
            s["xc"] += 0.02 * rng.uniform(-1, 1)
        b = Batch([(s["grid"], ensemble_params(s, **ENSEMBLE), MIXED) for s in specs], lockstep=case["lockstep"])
        for k, s in enumerate(specs):
            initial_bubble_state(b.case(k), s)
        start = [{f: b.case(k).download(f) for f in CHECKPOINT} for k in range(len(specs))]
        out = [{f: s["grid"].zeros(FIELD_KIND[f]) for f in RESULT} for s in specs]
        return dict(kind=kind, batch=b, start=start, out=out, steps=case["steps"], opts=Context.step_opts())
    g = _grid(case)
    if kind == "matvec":
        ctx = Context(g, Params())
        x = [_random(rng, g, k) for k in ("u", "v", "cell")]
        coef = [_random(rng, g, k) for k in ("u", "v")]
        coef += [_random(rng, g, k, lo, hi) for k, lo, hi in (
            ("cell", 1.0, 10.0), ("u", 1.0, 10.0), ("v", 1.0, 10.0), ("cell", 0.1, 2.0), ("vert", 0.2, 2.0),
            ("vert", 0.1, 1.0))]
        return dict(kind=kind, ctx=ctx, x=x, y=[g.zeros(k) for k in ("u", "v", "cell")], coef=coef, dt=1e-3)
    if kind == "transport":
        prm, dt, _ = _params(case)
        ctx = Context(g, prm)
        st = _state(case, g, ctx, None, seed)
        work = {k: g.zeros(kd) for k, kd in (("c", "cell"), ("cs", "cell"), ("kc", "cell"), ("fu", "u"), ("fv", "v"))}
        return dict(kind=kind, ctx=ctx, st=st, out=work, dt=dt, delta=prm.svof_delta_h * min(g.dx, g.dy),
                    iters=prm.svof_max_iter, tol=prm.svof_tol)
    if kind == "poisson":
        ctx = Context(g, Params())
        rhs, ru, rv = _poisson_inputs(g, seed)
        return dict(kind=kind, ctx=ctx, rhs=rhs, ru=ru, rv=rv, phi=g.zeros("cell"), tol=1e-10, iters=4000)
    if kind == "vjp":
        prm = Params(rho1=1000.0, rho2=100.0, mu1=10.0, mu2=1.0, sigma=24.5, gx=0.0, gy=-0.98, time_order=2,
                     tol_bicgstab2=1e-12, max_iter_bicgstab2=500, **GRADIENT)
        ctx = Context(g, prm)
        case = dict(case, flow="bubble")
        st = _state(case, g, ctx, None, seed)
        st["c_field"][...] = cases.circle_fraction(g, 0.5 + 0.02 * rng.uniform(-1, 1), 0.5, 0.25, inside=0.0, ns=8)
        _, Y = cases.cell_centres_interior(g)
        bar = {k: g.zeros(FIELD_KIND[k]) for k in ("u_vel", "v_vel", "c_field")}
        at(bar["c_field"], "cell", slice(1, g.nx), slice(1, g.ny))[...] = (0.5 - Y) * g.dx * g.dy
        for k in ("u_vel", "v_vel"):  # what the steps after this one pass back
            bar[k][...] = st[k] * g.dx * g.dy
        return dict(kind=kind, ctx=ctx, st=st, bar=bar, dt=2.5e-3, opts=Context.step_opts())
    prm, dt, lid = _params(case)
    ctx = Context(g, prm, precision=MIXED if case["mixed"] else FP64)
    st = _state(case, g, ctx, lid, seed)
    # the plain form of the tests steps with BiCGStab (the reference's BiCGStab(2)
    # does not converge on them)
    opts = Context.step_opts(use_bicgstab2=case["solver"] != "plain", u_top_lid=lid)
    out = {k: g.zeros(FIELD_KIND[k]) for k in RESULT}
    live = {k: a.copy(order="F") for k, a in st.items()}
    return dict(kind=kind, ctx=ctx, st=st, live=live, out=out, dt=dt, lid=lid, opts=opts,
                steps=case.get("steps", 1))


# --------------------------------------------------------------------- run
def run(s):
    kind = s["kind"]
    if kind == "batch":
        b = s["batch"]
        for k, st in enumerate(s["start"]):
            b.case(k).upload_state(st)
        b.run(s["steps"], 5e-4, 2, s["opts"])
        for k, out in enumerate(s["out"]):
            for f in RESULT:
                b.case(k).download(f, out[f])
        return s["out"]
    ctx = s["ctx"]
    if kind == "matvec":
        ctx.matvec_coupled(*s["x"], *s["y"], *s["coef"], s["dt"])
        return s["y"]
    if kind == "transport":
        st, o = s["st"], s["out"]
        ctx.vof_advection_tvd(st["c_field"], o["c"], st["u_vel"], st["v_vel"], s["dt"])
        ctx.svof_helmholtz_filter(o["c"], o["cs"], s["delta"], s["iters"], s["tol"])
        ctx.compute_interface_curvature(o["cs"], o["kc"])
        ctx.compute_csf_force(o["c"], o["kc"], o["fu"], o["fv"])
        return o
    if kind == "poisson":
        s["phi"][...] = 0.0
        ctx.solve_poisson_pressure(s["phi"], s["rhs"], s["ru"], s["rv"], s["tol"], s["iters"])
        return s["phi"]
    if kind == "vjp":
        ctx.upload_state({k: s["st"][k] for k in CHECKPOINT})
        bar, theta, _ = ctx.step_vjp(s["dt"], 2, s["opts"], s["bar"])
        return dict(bar, theta=theta)
    if kind == "dropin":
        live = s["live"]
        for k in STATE:
            live[k][...] = s["st"][k]
        ctx.advance_coupled_step(*[live[k] for k in STATE], s["dt"], 2, u_top_lid=s["lid"])
        return {k: live[k] for k in RESULT}
    ctx.upload_state({k: s["st"][k] for k in CHECKPOINT})
    for q in range(s["steps"]):
        ctx.step(s["dt"], 2 + q, s["opts"])
    for k in RESULT:
        ctx.download(k, s["out"][k])
    return s["out"]


def work(case):
    """Bytes of the inputs and outputs of a pass (each state field once per
    step) and the operations of one operator application per step; the
    iterations of the solves are not counted, since their number is the
    solver's own affair."""
    kind = case["kind"]
    if kind == "batch":
        cells = case["cases"] * 62000.0 * case["steps"]  # the ensemble's mean grid
        return {"bytes": 21 * 8 * cells, "flops": 150 * cells}
    cells = float(case["nx"] * case["ny"])
    fields = {"matvec": 14, "transport": 8, "poisson": 4, "vjp": 21}.get(kind, 21 * case.get("steps", 1))
    flops = {"matvec": 110, "transport": 250, "poisson": 20, "vjp": 600}.get(kind, 400 * case.get("steps", 1))
    return {"bytes": 8 * fields * cells, "flops": flops * cells}


# ------------------------------------------------------------------- exact
def _poisson_inputs(g, seed):
    rng = np.random.default_rng(seed)
    c = cases.circle_fraction(g, 0.5 + 0.02 * rng.uniform(-1, 1), 0.5, 0.25, inside=1.0, ns=4)
    rho = 1.0 * c + 0.1 * (1.0 - c)
    ru, rv = g.full("u", 1.0), g.full("v", 1.0)
    ru[1:-1, :] = 0.5 * (rho[:-1, :] + rho[1:, :])
    rv[:, 1:-1] = 0.5 * (rho[:, :-1] + rho[:, 1:])
    ru[0, :], ru[-1, :] = ru[1, :], ru[-2, :]
    rv[:, 0], rv[:, -1] = rv[:, 1], rv[:, -2]
    X, Y = cases.cell_centres_interior(g)
    rhs = g.zeros("cell")
    f = sum(rng.standard_normal() * np.cos(np.pi * m * X) * np.cos(np.pi * n * Y)
            for m in range(4) for n in range(4) if m + n)
    at(rhs, "cell", slice(1, g.nx), slice(1, g.ny))[...] = f
    return rhs, ru, rv


def _exact_poisson(case, seed):
    g = _grid(case)
    rhs, ru, rv = _poisson_inputs(g, seed)
    cx = 1.0 / (g.dx * g.dx) / at(ru, "u", slice(0, g.nx), slice(1, g.ny))
    cy = 1.0 / (g.dy * g.dy) / at(rv, "v", slice(1, g.nx), slice(0, g.ny))
    cx[0, :] = cx[-1, :] = 0.0
    cy[:, 0] = cy[:, -1] = 0.0
    cE, cW, cN, cS = cx[1:, :], cx[:-1, :], cy[:, 1:], cy[:, :-1]
    diag = cE + cW + cN + cS

    def apply(p):
        q = np.pad(p, 1, mode="edge")
        return diag * p - (cE * q[2:, 1:-1] + cW * q[:-2, 1:-1] + cN * q[1:-1, 2:] + cS * q[1:-1, :-2])

    b = at(rhs, "cell", slice(1, g.nx), slice(1, g.ny)).copy()
    b -= b.mean()
    x, r = np.zeros_like(b), b.copy()
    z = r / diag
    p, rz, nb = z.copy(), float(np.sum(r * z)), float(np.sqrt(np.sum(b * b)))
    for _ in range(6000):
        ap = apply(p)
        a = rz / float(np.sum(p * ap))
        x += a * p
        r -= a * ap
        if float(np.sqrt(np.sum(r * r))) < 1e-13 * nb:
            break
        z = r / diag
        rz, old = float(np.sum(r * z)), rz
        p = z + (rz / old) * p
    # the ghosts hold the initial guess's mirror, zero here
    out = g.zeros("cell")
    at(out, "cell", slice(1, g.nx), slice(1, g.ny))[...] = x - x.mean()
    return out


def _exact_matvec(case, seed):
    g = _grid(case)
    rng = np.random.default_rng(seed)
    U, V, Pr = (_random(rng, g, k) for k in ("u", "v", "cell"))
    ua, va = (_random(rng, g, k) for k in ("u", "v"))
    rc, ru, rv, ka, ze, et = (_random(rng, g, k, lo, hi) for k, lo, hi in (
        ("cell", 1.0, 10.0), ("u", 1.0, 10.0), ("v", 1.0, 10.0), ("cell", 0.1, 2.0), ("vert", 0.2, 2.0),
        ("vert", 0.1, 1.0)))
    nx, ny, idx, idy, dt, h = g.nx, g.ny, 1.0 / g.dx, 1.0 / g.dy, 1e-3, 0.5

    def view(a, kind, i0, i1, j0, j1):
        return lambda di, dj: at(a, kind, slice(i0 + di, i1 + di), slice(j0 + dj, j1 + dj))

    def views(i0, i1, j0, j1):
        return [view(a, k, i0, i1, j0, j1) for a, k in ((U, "u"), (V, "v"), (Pr, "cell"), (ua, "u"), (va, "v"),
                                                        (rc, "cell"), (ru, "u"), (rv, "v"), (ka, "cell"),
                                                        (ze, "vert"), (et, "vert"))]

    def shear(u, v, z, e, di, dj):
        dudy, dvdx = (u(di, dj + 1) - u(di, dj)) * idy, (v(di + 1, dj) - v(di, dj)) * idx
        zz, ee = z(di, dj), e(di, dj)
        return (zz - ee) * dudy + ee * dvdx, ee * dudy + (zz - ee) * dvdx

    Yu, Yv, Yp = g.zeros("u"), g.zeros("v"), g.zeros("cell")
    u, v, p, a, b, c, du, dv, k, z, e = views(1, nx - 1, 1, ny)
    adv = (c(1, 0) * h * (a(0, 0) + a(1, 0)) * h * (u(0, 0) + u(1, 0)) -
           c(0, 0) * h * (a(-1, 0) + a(0, 0)) * h * (u(-1, 0) + u(0, 0))) * idx
    adv += (h * (dv(0, 0) + dv(1, 0)) * h * (b(0, 0) + b(1, 0)) * h * (u(0, 0) + u(0, 1)) -
            h * (dv(0, -1) + dv(1, -1)) * h * (b(0, -1) + b(1, -1)) * h * (u(0, -1) + u(0, 0))) * idy
    vis = -((k(1, 0) * (u(1, 0) - u(0, 0)) - k(0, 0) * (u(0, 0) - u(-1, 0))) * idx * idx +
            (shear(u, v, z, e, 0, 0)[0] - shear(u, v, z, e, 0, -1)[0]) * idy)
    at(Yu, "u", slice(1, nx - 1), slice(1, ny))[...] = (du(0, 0) / dt * u(0, 0) + adv + vis +
                                                        (p(1, 0) - p(0, 0)) * idx)
    u, v, p, a, b, c, du, dv, k, z, e = views(1, nx, 1, ny - 1)
    adv = (h * (du(0, 0) + du(0, 1)) * h * (a(0, 0) + a(0, 1)) * h * (v(0, 0) + v(1, 0)) -
           h * (du(-1, 0) + du(-1, 1)) * h * (a(-1, 0) + a(-1, 1)) * h * (v(-1, 0) + v(0, 0))) * idx
    adv += (c(0, 1) * h * (b(0, 0) + b(0, 1)) * h * (v(0, 0) + v(0, 1)) -
            c(0, 0) * h * (b(0, -1) + b(0, 0)) * h * (v(0, -1) + v(0, 0))) * idy
    vis = -((shear(u, v, z, e, 0, 0)[1] - shear(u, v, z, e, -1, 0)[1]) * idx +
            (k(0, 1) * (v(0, 1) - v(0, 0)) - k(0, 0) * (v(0, 0) - v(0, -1))) * idy * idy)
    at(Yv, "v", slice(1, nx), slice(1, ny - 1))[...] = (dv(0, 0) / dt * v(0, 0) + adv + vis +
                                                        (p(0, 1) - p(0, 0)) * idy)
    for q in (0, nx):  # wall faces keep their value
        at(Yu, "u", q, slice(1, ny))[...] = at(U, "u", q, slice(1, ny))
    for q in (0, ny):
        at(Yv, "v", slice(1, nx), q)[...] = at(V, "v", slice(1, nx), q)
    u, v = views(1, nx, 1, ny)[:2]
    at(Yp, "cell", slice(1, nx), slice(1, ny))[...] = (u(0, 0) - u(-1, 0)) * idx + (v(0, 0) - v(0, -1)) * idy
    return [Yu, Yv, Yp]


def exact(case, seed):
    """The matrix-vector product and the Poisson solution in 64 bits.  The
    coupled steps have none (a Krylov solve to a residual tolerance), nor has
    the transport chain, whose filter stops by its own test."""
    if case["kind"] == "matvec":
        return _exact_matvec(case, seed)
    if case["kind"] == "poisson":
        return _exact_poisson(case, seed)
    return None
