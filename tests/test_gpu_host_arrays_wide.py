"""Host arrays of few rows: alone they go by the driver's copy (no launch), as
do very large ones with others; the values are the same by every way."""
import numpy as np
import pytest

from conftest import rfield, two_phase_params
from coupled_codefort_2d_b200.context import Context
from coupled_codefort_2d_b200.layout import Grid

pytestmark = pytest.mark.gpu


# a cell array has ny + 4 rows
@pytest.mark.parametrize("nx,ny,staged", [(4000, 20, 0), (1000, 21, 1), (600, 8, 1), (1100, 8, 0), (800, 92, 0), (800, 93, 1)])
def test_an_array_alone(gpu, nx, ny, staged):
    g = Grid(nx, ny, 1.0, ny / nx)
    a = rfield(np.random.default_rng(ny), g, "cell")
    with Context(g, two_phase_params()) as ctx:
        k = ctx.profile()["kernel_launches"]
        ctx.upload("c_field", a)
        assert ctx.profile()["kernel_launches"] - k == staged
        np.testing.assert_array_equal(ctx.download("c_field"), a)


# 120 KB: square, tall, and tall no more
@pytest.mark.parametrize("nx,ny,staged", [(116, 116, 0), (55, 256, 1), (80, 172, 1), (84, 160, 0)])
def test_an_array_down_alone(gpu, nx, ny, staged):
    g = Grid(nx, ny, 1.0, ny / nx)
    a = rfield(np.random.default_rng(ny), g, "cell")
    with Context(g, two_phase_params()) as ctx:
        ctx.upload("c_field", a)
        k = ctx.profile()["kernel_launches"]
        b = ctx.download("c_field")
        assert ctx.profile()["kernel_launches"] - k == staged
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("nx,ny", [(5900, 16), (800, 124), (800, 125)])
def test_arrays_together(gpu, oracle_mod, nx, ny):
    g, prm = Grid(nx, ny, 1.0, ny / nx), two_phase_params()
    rng = np.random.default_rng(ny)
    o = oracle_mod.Oracle(g, prm)
    pr = o.properties(np.asfortranarray(rng.uniform(0.0, 1.0, g.shape("cell"))))
    x = [rfield(rng, g, k) for k in ("u", "v", "cell")]
    adv = [rfield(rng, g, k) for k in ("u", "v")]
    xo, y, yo = [a.copy(order="F") for a in x], *[[g.zeros(k) for k in ("u", "v", "cell")] for _ in range(2)]
    o.matvec(*xo, *yo, *adv, pr, 2e-3)
    with Context(g, prm) as ctx:
        ctx.matvec_coupled(*x, *y, *adv, *[pr[k] for k in ("rho_c", "rho_u", "rho_v", "kappa", "zeta", "eta")], 2e-3)
    for a, b in zip(x + y, xo + yo):
        np.testing.assert_array_equal(a, b)
