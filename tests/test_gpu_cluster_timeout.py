"""The waits of the kernels that exchange within a thread-block cluster are
bounded: armed (every CTA expects bytes that nobody sends) the launch gives up,
the call reports FUGU_ETIMEOUT, and the same context then gives the bits of
one that never failed."""
import numpy as np
import pytest

from conftest import rfield, two_phase_params
from coupled_codefort_2d_b200._lib import MIXED, FuguError
from coupled_codefort_2d_b200.context import Context
from coupled_codefort_2d_b200.layout import Grid
from coupled_codefort_2d_b200.params import Params

pytestmark = pytest.mark.gpu


def times_out(fn):
    with pytest.raises(FuguError) as ei:
        fn()
    assert ei.value.code == -5 and "gave up" in str(ei.value)


# two CTAs and sixteen
@pytest.mark.parametrize("nx,ny,py", [(12, 10, 1), (130, 121, 0)])
def test_fp64_solve(gpu, oracle_mod, nx, ny, py):
    g, prm = Grid(nx, ny, periodic_y=bool(py)), two_phase_params()
    o = oracle_mod.Oracle(g, prm)
    rng = np.random.default_rng(nx)
    pr = o.properties(np.asfortranarray(rng.uniform(0.0, 1.0, g.shape("cell"))))
    rhs, phi0 = rfield(rng, g, "cell"), rfield(rng, g, "cell", -0.1, 0.1)

    def solve(ctx, phi):
        return ctx.solve_poisson_pressure(phi, rhs, pr["rho_u"], pr["rho_v"], 1e-5, 24)

    po, pg = phi0.copy(order="F"), phi0.copy(order="F")
    want = o.poisson(po, rhs, pr["rho_u"], pr["rho_v"], 1e-5, 24)
    with Context(g, prm) as ctx:
        ctx.arm_cluster_timeout(1000)
        times_out(lambda: solve(ctx, phi0.copy(order="F")))
        assert solve(ctx, pg) == want
    np.testing.assert_array_equal(pg, po)


@pytest.mark.parametrize("nx,ny", [(17, 15), (130, 121)])
def test_fp32_solve_inside_a_step(gpu, oracle_mod, nx, ny):
    g = Grid(nx, ny)
    p = Params(rho1=1.0, rho2=1.0, mu1=0.01, mu2=0.01, sigma=0.0, gx=0.0, gy=0.0, time_order=1, tol_bicgstab2=1e-8,
               max_iter_bicgstab2=100, refine=2, refine_inner_tol=1e-2, refine_max_inner=30, refine_max_outer=60,
               krylov_bc_fix=1, pcd_visc_scale=1.0)
    st = oracle_mod.new_state(g, g.full("cell", 1.0), p)
    out = []
    for fail in (False, True):
        with Context(g, p, precision=MIXED) as ctx:
            o = ctx.step_opts(u_top_lid=1.0)
            ctx.upload_state(st)
            if fail:
                ctx.arm_cluster_timeout(1000)
                times_out(lambda: ctx.step(1e-3, 1, o))
                ctx.upload_state(st)
            out.append((ctx.step(1e-3, 1, o), ctx.download_state(["u_vel", "v_vel", "p_field"])))
    assert out[0][0] == out[1][0] and out[0][0]["status"] == 0
    for k, a in out[0][1].items():
        np.testing.assert_array_equal(a, out[1][1][k], err_msg=k)


@pytest.mark.parametrize("nx,ny,py", [(33, 29, 1), (256, 250, 0)])
def test_svof_filter(gpu, oracle_mod, nx, ny, py):
    g, prm = Grid(nx, ny, periodic_y=bool(py)), two_phase_params()
    c = np.asfortranarray(np.random.default_rng(nx).uniform(0.0, 1.0, g.shape("cell")))
    h = 1.5 * min(g.dx, g.dy)
    so, sg = g.zeros("cell"), g.zeros("cell")
    ko = oracle_mod.Oracle(g, prm).svof(c, so, h, 23, 0.0)
    with Context(g, prm) as ctx:
        ctx.arm_cluster_timeout(1000)
        times_out(lambda: ctx.svof_helmholtz_filter(c, sg, h, 23, 0.0))
        assert ctx.svof_helmholtz_filter(c, sg, h, 23, 0.0) == ko
    np.testing.assert_array_equal(sg, so)
