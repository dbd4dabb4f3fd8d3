"""Narrow boxes of an odd or tiny width, as tall as a thread-block cluster
holds (16 CTAs of 4,096 cells): their FP64 pressure solve runs in the cluster and
equals the oracle bit for bit, and a lockstep batch, which needs the cluster,
takes them."""
import numpy as np
import pytest

from conftest import rfield, two_phase_params
from coupled_codefort_2d_b200 import cases
from coupled_codefort_2d_b200._lib import FP64
from coupled_codefort_2d_b200.batch import STATE_FIELDS, Batch, ensemble_params, initial_bubble_state
from coupled_codefort_2d_b200.context import Context
from coupled_codefort_2d_b200.layout import Grid

pytestmark = pytest.mark.gpu


# the first and the last height of each width whose segments or pitched rows did not fit four segments per thread
@pytest.mark.parametrize("nx,ny", [(4, 14433), (4, 16384), (5, 10913), (5, 13056), (7, 9344), (25, 2560), (85, 753),
                                   (85, 768)])
def test_cluster_takes_narrow_boxes(gpu, oracle_mod, monkeypatch, nx, ny):
    monkeypatch.setenv("FUGU_PCG", "cluster")
    g, prm = Grid(nx, ny, 1.0, ny / nx), two_phase_params()
    o = oracle_mod.Oracle(g, prm)
    rng = np.random.default_rng(nx + ny)
    pr = o.properties(np.asfortranarray(rng.uniform(0.0, 1.0, g.shape("cell"))))
    rhs, phi0 = rfield(rng, g, "cell"), rfield(rng, g, "cell", -0.1, 0.1)
    po, pg = phi0.copy(order="F"), phi0.copy(order="F")
    want = o.poisson(po, rhs, pr["rho_u"], pr["rho_v"], 1e-5, 24)
    with Context(g, prm) as ctx:
        assert ctx.profile()["pcg_cluster_fp64"] == 16
        assert ctx.solve_poisson_pressure(pg, rhs, pr["rho_u"], pr["rho_v"], 1e-5, 24) == want
    np.testing.assert_array_equal(pg, po)


def test_lockstep_takes_narrow_boxes(gpu):
    grids = ((51, 160), (85, 96))
    specs = cases.bubble_ensemble(2, grids=grids)
    for s, (nx, ny) in zip(specs, grids):
        s["grid"] = Grid(nx, ny, 1.0, ny / nx)
    solver = dict(tol_bicgstab2=1e-6, max_iter_bicgstab2=200, refine=2, refine_inner_tol=1e-1, refine_max_inner=12,
                  refine_max_outer=2, krylov_bc_fix=1, pcg_cap_start=20, graphs=1, pcd_visc_scale=1.0)
    out = []
    for lockstep in (False, True):
        with Batch([(s["grid"], ensemble_params(s, **solver), FP64) for s in specs], max_cluster=2,
                   lockstep=lockstep) as b:
            for k, s in enumerate(specs):
                initial_bubble_state(b.case(k), s)
            b.run(1, 5e-4, 1, b.case(0).step_opts())
            out.append([b.case(k).download_state(list(STATE_FIELDS)) for k in range(2)])
    for k in range(2):
        for f in STATE_FIELDS:
            np.testing.assert_array_equal(out[0][k][f], out[1][k][f], err_msg=f"case {k} {f}")
