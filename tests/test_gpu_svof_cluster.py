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
