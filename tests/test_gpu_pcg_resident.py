"""The PCG pressure solve resident on chip (``csrc/pcg_resident.cuh``,
``csrc/pcg_cluster.cuh``) at the sizes where its layout can go wrong: partly
filled segments and strips, one row per CTA, a last CTA with fewer rows, every
kernel shape and both exchanges; its bounded waits; and two host threads whose
whole-device solves share the GPU.

FP64 equals the oracle bit for bit (error-free sums, the reference's
expressions).  FP32 over the whole device equals the grid-wide kernel it
replaces bit for bit (``FUGU_PCG=grid``: same expressions, error-free sums);
FP32 in a cluster sums in another order than that kernel, so the mixed form
solved to 1e-10 agrees to 1e-7 (two FP32 inner paths, one FP64 tolerance).
"""
import threading

import numpy as np
import pytest

from conftest import rfield, two_phase_params
from coupled_codefort_2d_b200 import cases
from coupled_codefort_2d_b200._lib import FuguError
from coupled_codefort_2d_b200.context import Context
from coupled_codefort_2d_b200.layout import Grid
from coupled_codefort_2d_b200.params import Params

pytestmark = pytest.mark.gpu

# cluster: 1 x 256 (smallest, partial segments, one row per CTA), 2 x 256,
# 4 x 256 with a short last CTA; grid: 2 x 256, 4 x 256, 3 x 512, 4 x 512
FP64_GRIDS = [(4, 4, 0, 0), (5, 67, 0, 1), (31, 29, 1, 0), (130, 121, 0, 0), (203, 157, 0, 0), (255, 129, 1, 1),
              (256, 257, 0, 0), (511, 301, 0, 0), (641, 300, 0, 1), (1030, 296, 0, 0), (1023, 590, 0, 0)]


def poisson_inputs(o, g, seed):
    rng = np.random.default_rng(seed)
    pr = o.properties(np.asfortranarray(rng.uniform(0.0, 1.0, size=g.shape("cell"))))
    return pr, rfield(rng, g, "cell"), rfield(rng, g, "cell", -0.1, 0.1)


@pytest.mark.parametrize("nx,ny,px,py", FP64_GRIDS)
def test_fp64_solve_equals_the_oracle(gpu, oracle_mod, nx, ny, px, py):
    g = Grid(nx, ny, periodic_x=bool(px), periodic_y=bool(py))
    o = oracle_mod.Oracle(g, two_phase_params())
    pr, rhs, phi0 = poisson_inputs(o, g, nx + ny)
    po, pg = phi0.copy(order="F"), phi0.copy(order="F")
    want = o.poisson(po, rhs, pr["rho_u"], pr["rho_v"], 1e-5, 24)
    with Context(g, two_phase_params()) as ctx:
        for _ in range(2):  # the exchange's numbers continue from solve to solve
            pg[...] = phi0
            got = ctx.solve_poisson_pressure(pg, rhs, pr["rho_u"], pr["rho_v"], 1e-5, 24)
            assert got == want
            np.testing.assert_array_equal(pg, po)
        zero = g.zeros("cell")  # a zero right-hand side ends at once
        assert ctx.solve_poisson_pressure(pg, zero, pr["rho_u"], pr["rho_v"], 1e-5, 24) == (0, 0.0)
        assert not np.any(pg)


def droplet(nx, ny):
    g = Grid(nx, ny, 1.0, ny / nx)
    p = Params(rho1=1.0, rho2=0.1, mu1=0.1, mu2=0.01, sigma=1.0, gx=0.0, gy=0.0, time_order=2, tol_bicgstab2=1e-10,
               max_iter_bicgstab2=500, refine=2, refine_inner_tol=1e-2, refine_max_inner=30, refine_max_outer=60,
               krylov_bc_fix=1, pcg_cap_start=40, pcd_sweeps=6, pcd_sweeps_max=24, graphs=1, pcd_visc_scale=1.0)
    return g, p, cases.circle_fraction(g, 0.5, 0.5 * ny / nx, 0.2 * min(1.0, ny / nx), inside=1.0, ns=4)


def mixed_steps(oracle_mod, nx, ny, precision=1):
    g, p, c0 = droplet(nx, ny)
    st = oracle_mod.new_state(g, c0, p)
    with Context(g, p, precision=precision) as ctx:
        ctx.upload_state(st)
        stats = [ctx.step(1e-4, s, ctx.step_opts()) for s in (1, 2)]
        return stats, ctx.download_state(["u_vel", "v_vel", "p_field"])


@pytest.mark.parametrize("nx,ny", [(514, 20), (515, 150), (600, 301), (770, 296)])
def test_fp32_whole_device_solve_equals_the_grid_wide_kernel(gpu, oracle_mod, monkeypatch, nx, ny):
    s1, a = mixed_steps(oracle_mod, nx, ny)
    monkeypatch.setenv("FUGU_PCG", "grid")
    s2, b = mixed_steps(oracle_mod, nx, ny)
    assert s1 == s2
    for k in a:
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)


# strips of 1, 2, 4, 8 and 16 cells; partly filled strips and last CTAs
@pytest.mark.parametrize("nx,ny", [(17, 15), (33, 61), (130, 121), (255, 250), (500, 201)])
def test_fp32_cluster_solve_agrees_with_the_grid_wide_kernel(gpu, oracle_mod, monkeypatch, nx, ny):
    s1, a = mixed_steps(oracle_mod, nx, ny)
    monkeypatch.setenv("FUGU_PCG", "grid")
    s2, b = mixed_steps(oracle_mod, nx, ny)
    assert [s["status"] for s in s1 + s2] == [0] * 4
    for k in ("u_vel", "v_vel"):
        assert np.linalg.norm(a[k] - b[k]) <= 1e-7 * np.linalg.norm(b[k]), k


def test_whole_device_wait_is_bounded_and_the_context_recovers(gpu, oracle_mod):
    g = Grid(300, 200)
    o = oracle_mod.Oracle(g, two_phase_params())
    pr, rhs, phi0 = poisson_inputs(o, g, 5)
    with Context(g, two_phase_params()) as ctx:
        ctx.arm_barrier_timeout(1000)
        with pytest.raises(FuguError) as ei:
            ctx.solve_poisson_pressure(phi0.copy(order="F"), rhs, pr["rho_u"], pr["rho_v"], 1e-5, 24)
        assert ei.value.code == -5 and "gave up" in str(ei.value)
        pg = phi0.copy(order="F")
        got = ctx.solve_poisson_pressure(pg, rhs, pr["rho_u"], pr["rho_v"], 1e-5, 24)
    po = phi0.copy(order="F")
    assert got == o.poisson(po, rhs, pr["rho_u"], pr["rho_v"], 1e-5, 24)
    np.testing.assert_array_equal(pg, po)


def test_two_threads_share_the_device(gpu, oracle_mod):
    """Two contexts stepped by two host threads, each with whole-device solves
    of its own: the same states as one after the other."""
    sizes = [(530, 90), (300, 260)]
    want = [mixed_steps(oracle_mod, *s, precision=q) for s, q in zip(sizes, (1, 0))]
    got = [None, None]

    def work(k):
        for _ in range(3):
            got[k] = mixed_steps(oracle_mod, *sizes[k], precision=(1, 0)[k])

    ts = [threading.Thread(target=work, args=(k,)) for k in (0, 1)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for w, h in zip(want, got):
        assert h is not None and w[0] == h[0]
        for k in w[1]:
            np.testing.assert_array_equal(w[1][k], h[1][k], err_msg=k)
