"""The velocity smoother's quotient (``csrc/smooth_tile.cuh``) where it is not
simply the division: numerators that are a zero with a sign or outside the
exact range, in both modes and for both components in FP64 (bit for bit the
oracle's, signs of zeros included), and a diagonal outside the range in FP32 (bit
for bit the lockstep batch's sweeps, which divide)."""
import numpy as np
import pytest

from conftest import rfield, two_phase_params
from coupled_codefort_2d_b200 import cases
from coupled_codefort_2d_b200._lib import MIXED
from coupled_codefort_2d_b200.batch import STATE_FIELDS, Batch, ensemble_params, initial_bubble_state
from coupled_codefort_2d_b200.context import Context
from coupled_codefort_2d_b200.layout import Grid

pytestmark = pytest.mark.gpu


def same_bits(a, b, what):
    np.testing.assert_array_equal(a, b, err_msg=what)
    num = ~np.isnan(a)
    np.testing.assert_array_equal(np.signbit(a) & num, np.signbit(b) & num, err_msg=what + ", signs")


@pytest.mark.parametrize("smoother", [0, 1])
@pytest.mark.parametrize("kind", ["u", "v"])
@pytest.mark.parametrize("scale", [-0.0, 0.0, 1e-310, 1e-200, 1e-140, 1e250, 1e306, np.inf])
def test_fp64_extreme_numerators(gpu, oracle_mod, kind, smoother, scale):
    g = Grid(33, 20)
    rng = np.random.default_rng(3)
    prm = two_phase_params(pcd_smoother=smoother, pcd_sor_omega=0.9)
    o = oracle_mod.Oracle(g, prm)
    pr = o.properties(np.asfortranarray(rng.uniform(0.0, 1.0, g.shape("cell"))))
    rho = pr["rho_u"] if kind == "u" else pr["rho_v"]
    with np.errstate(all="ignore"):
        rhs = rfield(rng, g, kind) * scale if scale else g.full(kind, scale)
        sol = g.full(kind, np.copysign(0.0, scale))
        with Context(g, prm) as ctx:
            for n in (3, 6):
                s, r = sol.copy(order="F"), sol.copy(order="F")
                gfn, ofn = (ctx.solve_helmholtz_u, o.helmholtz_u) if kind == "u" else (ctx.solve_helmholtz_v, o.helmholtz_v)
                gfn(s, rhs, rho, pr["kappa"], pr["zeta"], pr["eta"], 2e-3, n, None)
                ofn(r, rhs, pr, 2e-3, n, None)
                same_bits(s, r, f"{n} sweeps")


@pytest.mark.parametrize("smoother", [0, 1])
def test_fp32_diagonal_outside_the_exact_range(gpu, smoother):
    grids = ((40, 81), (64, 64))
    specs = cases.bubble_ensemble(2, grids=grids)
    for s, (nx, ny) in zip(specs, grids):
        s["grid"] = Grid(nx, ny, 1.0, ny / nx)
    solver = dict(tol_bicgstab2=1e-6, max_iter_bicgstab2=200, refine=2, refine_inner_tol=1e-1, refine_max_inner=12,
                  refine_max_outer=2, krylov_bc_fix=1, pcg_cap_start=20, pcd_sweeps=3, pcd_smoother=smoother,
                  pcd_sor_omega=1.5, graphs=1, pcd_visc_scale=1.0)
    out = []
    for lockstep in (False, True):
        with Batch([(s["grid"], ensemble_params(s, **solver), MIXED) for s in specs], max_cluster=16,
                   lockstep=lockstep) as b:
            for k, s in enumerate(specs):
                initial_bubble_state(b.case(k), s)
            b.run(1, 1e-11, 1, b.case(0).step_opts())  # rho / dt above 2^40 in the heavy fluid
            out.append([b.case(k).download_state(list(STATE_FIELDS)) for k in range(2)])
    for k in range(2):
        for f in STATE_FIELDS:
            same_bits(out[0][k][f], out[1][k][f], f"case {k} {f}")
