"""The SVOF filter in one thread-block cluster (``csrc/svof_cluster.cuh``) at the
sizes where its groups of sweeps can go wrong: the fewest rows a CTA may own,
a last CTA with fewer rows, padding rows, periodic wraps, sweep counts that
are no multiple of the group, and stops inside a group (which repeat its
sweeps).  Equal to the oracle bit for bit, sweep count included; 512 columns
are the widest, 513 take the grid-wide kernel."""
import numpy as np
import pytest

from conftest import two_phase_params
from coupled_codefort_2d_b200.context import Context
from coupled_codefort_2d_b200.layout import Grid

pytestmark = pytest.mark.gpu

GRIDS = [(4, 4, 0, 0), (5, 9, 1, 1), (33, 29, 0, 1), (64, 67, 0, 0), (100, 66, 1, 0), (255, 61, 0, 0), (256, 250, 0, 1),
         (512, 40, 0, 0), (513, 20, 0, 0)]


@pytest.mark.parametrize("nx,ny,px,py", GRIDS)
def test_filter_equals_the_oracle(gpu, oracle_mod, nx, ny, px, py):
    g = Grid(nx, ny, periodic_x=bool(px), periodic_y=bool(py))
    o = oracle_mod.Oracle(g, two_phase_params())
    rng = np.random.default_rng(nx * 1000 + ny)
    c = np.asfortranarray(rng.uniform(0.0, 1.0, g.shape("cell")))
    h = 1.5 * min(g.dx, g.dy)
    with Context(g, two_phase_params()) as ctx:
        # tolerances that stop at every position of a group, then plain counts
        for iters, tol in [(40, t) for t in (3e-2, 1.5e-2, 8e-3, 5e-3, 2e-3)] + [(k, 0.0) for k in (0, 1, 4, 7)]:
            so, sg = g.zeros("cell"), g.zeros("cell")
            ko = o.svof(c, so, h, iters, tol)
            kg = ctx.svof_helmholtz_filter(c, sg, h, iters, tol)
            assert kg == ko, (iters, tol)
            np.testing.assert_array_equal(sg, so, err_msg=f"{iters} {tol}")


@pytest.mark.parametrize("nx,ny,px,py", [(33, 29, 0, 1), (256, 250, 0, 1)])
def test_filter_beyond_the_exact_quotient(gpu, oracle_mod, nx, ny, px, py):
    """Infinities, NaN, denormals, -0, huge values and a diagonal beyond 2^100: the bits of a division."""
    g = Grid(nx, ny, periodic_x=bool(px), periodic_y=bool(py))
    o = oracle_mod.Oracle(g, two_phase_params())
    rng = np.random.default_rng(ny)
    c = np.asfortranarray(rng.uniform(-0.5, 1.0, g.shape("cell")))
    marked = c.copy(order="F")
    marked[nx // 2, ny // 2], marked[nx // 3, ny // 4] = np.inf, np.nan
    h = 1.5 * min(g.dx, g.dy)
    with Context(g, two_phase_params()) as ctx:
        for field, width in [(marked, h), (c * 1e-310, h), (c * 1e-296, h), (c * 1e303, h), (c * -0.0, h),
                             (c, 1e20 * h)]:
            # a NaN change counts for nothing here and resets the oracle's maximum: plain counts there
            for iters, tol in [(7, 0.0)] + [(40, 8e-3)] * (field is not marked):
                field = np.asfortranarray(field)
                so, sg = g.zeros("cell"), g.zeros("cell")
                ko = o.svof(field, so, width, iters, tol)
                assert ctx.svof_helmholtz_filter(field, sg, width, iters, tol) == ko
                np.testing.assert_array_equal(sg, so)
                finite = ~np.isnan(so)
                np.testing.assert_array_equal(np.signbit(sg[finite]), np.signbit(so[finite]))
