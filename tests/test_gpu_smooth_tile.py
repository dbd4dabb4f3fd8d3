"""The PCD's velocity smoother with several sweeps per launch
(``csrc/smooth_tile.cuh``) at the sizes where its layout can go wrong: boxes
smaller than a tile, one row or column more or less than whole tiles, odd and
even sizes, each ring (2, 4, 6, 12 faces) with as many passes as it takes, with
fewer and with a second launch.

FP64 equals the oracle bit for bit.  FP32 equals one sweep per launch bit for
bit: the lockstep batch runs those, the thread-pool batch the tiles.
"""
import numpy as np
import pytest

from conftest import rfield, two_phase_params
from coupled_codefort_2d_b200 import cases
from coupled_codefort_2d_b200._lib import MIXED
from coupled_codefort_2d_b200.batch import STATE_FIELDS, Batch, ensemble_params, initial_bubble_state
from coupled_codefort_2d_b200.context import Context
from coupled_codefort_2d_b200.layout import Grid

pytestmark = pytest.mark.gpu

# tiles keep 60 x 26, 56 x 22, 52 x 18 or 40 x 6 faces; the box is nx + 5 padded by ny + 5
GRIDS = [(4, 4), (5, 7), (35, 13), (47, 66), (64, 32), (129, 130), (420, 430)]
SWEEPS = [(1, False), (2, True), (3, False), (6, False), (7, True)]  # and with penalisation


@pytest.mark.parametrize("smoother", [0, 1])
@pytest.mark.parametrize("nx,ny", GRIDS)
def test_fp64_sweeps_equal_the_oracle(gpu, oracle_mod, nx, ny, smoother):
    g = Grid(nx, ny)
    rng = np.random.default_rng(nx + 7 * ny)
    prm = two_phase_params(pcd_smoother=smoother, pcd_sor_omega=1.5)
    o = oracle_mod.Oracle(g, prm)
    pr = o.properties(np.asfortranarray(rng.uniform(0.0, 1.0, g.shape("cell"))))
    with Context(g, prm) as ctx:
        for kind, gfn, ofn in (("u", ctx.solve_helmholtz_u, o.helmholtz_u), ("v", ctx.solve_helmholtz_v, o.helmholtz_v)):
            sol, rhs, pen = rfield(rng, g, kind), rfield(rng, g, kind), rfield(rng, g, kind, 0, 1e6)
            rho = pr["rho_u"] if kind == "u" else pr["rho_v"]
            for n, penalised in SWEEPS:
                p = pen if penalised else None
                s, r = sol.copy(order="F"), sol.copy(order="F")
                gfn(s, rhs, rho, pr["kappa"], pr["zeta"], pr["eta"], 2e-3, n, p)
                ofn(r, rhs, pr, 2e-3, n, p)
                np.testing.assert_array_equal(s, r, err_msg=f"{kind} {n}")


@pytest.mark.parametrize("smoother", [0, 1])
def test_fp32_sweeps_equal_one_sweep_per_launch(gpu, smoother):
    specs = cases.bubble_ensemble(4, grids=((40, 81), (129, 130), (200, 301), (256, 512)))
    for s, grid in zip(specs, ((40, 81), (129, 130), (200, 301), (256, 512))):
        s["grid"] = Grid(*grid, 1.0, grid[1] / grid[0])
    solver = dict(tol_bicgstab2=1e-6, max_iter_bicgstab2=200, refine=2, refine_inner_tol=1e-1, refine_max_inner=12,
                  refine_max_outer=2, krylov_bc_fix=1, pcg_cap_start=20, pcd_sweeps=3, pcd_sweeps_max=6,
                  pcd_smoother=smoother, pcd_sor_omega=1.5, graphs=1, pcd_visc_scale=1.0)
    out = []
    for lockstep in (False, True):
        with Batch([(s["grid"], ensemble_params(s, **solver), MIXED) for s in specs], max_cluster=16,
                   lockstep=lockstep) as b:
            for k, s in enumerate(specs):
                initial_bubble_state(b.case(k), s)
            b.run(1, 5e-4, 1, b.case(0).step_opts())
            out.append([b.case(k).download_state(list(STATE_FIELDS)) for k in range(len(specs))])
    for k in range(len(specs)):
        for f in STATE_FIELDS:
            np.testing.assert_array_equal(out[0][k][f], out[1][k][f], err_msg=f"case {k} {f}")


def test_extreme_values_take_the_division(gpu, oracle_mod):
    """Numerators outside the exact quotient's range, zeros and infinities."""
    g = Grid(33, 20)
    rng = np.random.default_rng(3)
    prm = two_phase_params(pcd_smoother=1, pcd_sor_omega=1.5)
    o = oracle_mod.Oracle(g, prm)
    pr = o.properties(np.asfortranarray(rng.uniform(0.0, 1.0, g.shape("cell"))))
    for scale in (0.0, 1e-310, 1e-200, 1e250, 1e306):
        sol, rhs = rfield(rng, g, "u") * 0.0, rfield(rng, g, "u") * scale
        if scale == 0.0:
            rhs[rhs.shape[0] // 2, rhs.shape[1] // 2] = np.inf
        with Context(g, prm) as ctx, np.errstate(all="ignore"):
            s, r = sol.copy(order="F"), sol.copy(order="F")
            ctx.solve_helmholtz_u(s, rhs, pr["rho_u"], pr["kappa"], pr["zeta"], pr["eta"], 2e-3, 3, None)
            o.helmholtz_u(r, rhs, pr, 2e-3, 3, None)
            np.testing.assert_array_equal(s, r, err_msg=f"{scale}")
