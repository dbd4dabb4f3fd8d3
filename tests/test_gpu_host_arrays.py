"""How a context moves host arrays: through its staging area (a launch), or by
the driver's copy (none) where the array is page-locked and large, or comes down
alone and is small.  The values are the same by every way."""
import numpy as np
import pytest
import torch

from conftest import rfield, two_phase_params
from coupled_codefort_2d_b200.context import Context
from coupled_codefort_2d_b200.layout import Grid

pytestmark = pytest.mark.gpu


def pinned(a):
    t = torch.empty(a.size, dtype=torch.float64, pin_memory=True)
    out = t.numpy().reshape(a.shape, order="F")
    out[...] = a
    return out


# a cell array of 10 KB, 139 KB, 205 KB, 302 KB and 541 KB
@pytest.mark.parametrize("n", [32, 128, 156, 190, 256])
def test_ways_of_one_array(gpu, n):
    g = Grid(n, n)
    a = rfield(np.random.default_rng(n), g, "cell")
    with Context(g, two_phase_params()) as ctx:
        def launches(fn):
            k = ctx.profile()["kernel_launches"]
            fn()
            return ctx.profile()["kernel_launches"] - k

        for host in (a, pinned(a)):
            lock = host is not a
            up = launches(lambda: ctx.upload("c_field", host))
            back = pinned(np.zeros_like(a)) if lock else np.zeros_like(a)
            dn = launches(lambda: ctx.download("c_field", back))
            np.testing.assert_array_equal(back, a)
            assert up == (0 if lock and host.nbytes > 256 << 10 else 1)
            assert dn == (0 if lock or host.nbytes <= 160 << 10 else 1)


@pytest.mark.parametrize("n", [20, 256, 400])
def test_operator_with_mixed_arrays(gpu, n):
    """Pageable and page-locked arrays in one call, both beyond the staging
    area's wrap and with arrays that never stage (400^2)."""
    g = Grid(n, n)
    rng = np.random.default_rng(n)
    kinds = ("u", "v", "cell", "u", "v", "cell", "u", "v", "cell", "vert", "vert")
    lo = (-1, -1, -1, -1, -1, 1, 1, 1, 0.1, 0.2, 0.1)
    arrays = [rfield(rng, g, k, a, a + 2) for k, a in zip(kinds, lo)]
    out = []
    with Context(g, two_phase_params()) as ctx:
        for lock in ("", "even", "all"):
            pin = [pinned(a) if lock == "all" or lock and q % 2 == 0 else a.copy(order="F") for q, a in enumerate(arrays)]
            y = [g.zeros(k) for k in ("u", "v", "cell")]
            y = [pinned(a) if lock == "all" or lock and q % 2 else a for q, a in enumerate(y)]
            ctx.matvec_coupled(*pin[:3], *y, *pin[3:], 1e-3)
            out.append(pin[:3] + y)
    for got in out[1:]:
        for a, b in zip(got, out[0]):
            np.testing.assert_array_equal(a, b)
