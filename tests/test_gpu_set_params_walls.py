"""``fugu_set_params`` may turn a periodic direction of a context into walls:
what the periodic case left in the ghost cells of the context's work arrays must
not reach the results, which are those of a context made with walls."""
import numpy as np
import pytest

from conftest import rfield, two_phase_params
from coupled_codefort_2d_b200.context import Context
from coupled_codefort_2d_b200.layout import Grid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("px,py", [(1, 0), (0, 1), (1, 1)])
def test_walls_after_periodic_directions(gpu, oracle_mod, px, py):
    per, walls, prm = Grid(24, 20, periodic_x=bool(px), periodic_y=bool(py)), Grid(24, 20), two_phase_params()
    rng = np.random.default_rng(17)
    pr = oracle_mod.Oracle(walls, prm).properties(np.asfortranarray(rng.uniform(0.0, 1.0, walls.shape("cell"))))
    z = [rfield(rng, walls, k) for k in ("u", "v", "cell")]
    coef = [rfield(rng, walls, k) for k in ("u", "v")] + [pr[k] for k in ("rho_u", "rho_v", "kappa", "zeta", "eta")]

    def apply(ctx):
        r = [walls.zeros(k) for k in ("u", "v", "cell")]
        ctx.apply_pcd_precond(*z, *r, *coef, 2e-3)
        return r

    with Context(walls, prm) as ctx:
        want = apply(ctx)
    with Context(per, prm) as ctx:
        apply(ctx)
        ctx.g = walls
        ctx.set_params(prm)
        got = apply(ctx)
    for k, a, b in zip("uvp", got, want):
        np.testing.assert_array_equal(a, b, err_msg=k)
