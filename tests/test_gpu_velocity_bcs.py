"""The wall conditions without phases (``k_velocity_bcs``) at the sizes
where their fixed expressions could go wrong: the smallest box they take, one
below it (the phases), and every combination of walls; bit for bit the oracle's
four phases, ghosts and corners included."""
import numpy as np
import pytest

from conftest import rfield, two_phase_params
from coupled_codefort_2d_b200.context import Context
from coupled_codefort_2d_b200.layout import Grid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("px,py", [(0, 0), (1, 0), (0, 1)])
@pytest.mark.parametrize("nx,ny", [(4, 4), (4, 33), (27, 4), (60, 71)])
@pytest.mark.parametrize("free_slip", [0, 1])
def test_faces_equal_the_phases(gpu, oracle_mod, nx, ny, px, py, free_slip):
    g = Grid(nx, ny, periodic_x=bool(px), periodic_y=bool(py))
    prm = two_phase_params(free_slip_x=free_slip)
    rng = np.random.default_rng(10 * nx + ny)
    o = oracle_mod.Oracle(g, prm)
    with Context(g, prm) as ctx:
        for lid in (None, 0.75):
            u, v = rfield(rng, g, "u"), rfield(rng, g, "v")
            ru, rv = u.copy(order="F"), v.copy(order="F")
            ctx.apply_velocity_bcs(u, v, lid)
            o.velocity_bcs(ru, rv, lid)
            np.testing.assert_array_equal(u, ru, err_msg=f"u {lid}")
            np.testing.assert_array_equal(v, rv, err_msg=f"v {lid}")
