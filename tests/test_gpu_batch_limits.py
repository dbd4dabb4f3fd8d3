"""``fugu_batch_opts.max_coop`` bounds the CTAs of every grid-wide persistent
kernel of a batch, the SVOF filter's too, and the filter's result does not depend
on them; ``fugu_profile`` reports the CTAs of the kernel that runs."""
import numpy as np
import pytest

from coupled_codefort_2d_b200 import cases
from coupled_codefort_2d_b200._lib import MIXED
from coupled_codefort_2d_b200.batch import STATE_FIELDS, Batch, ensemble_params, initial_bubble_state
from coupled_codefort_2d_b200.context import Context
from coupled_codefort_2d_b200.layout import Grid
from coupled_codefort_2d_b200.params import Params

pytestmark = pytest.mark.gpu

SOLVER = dict(tol_bicgstab2=1e-6, max_iter_bicgstab2=200, refine=2, refine_inner_tol=1e-1, refine_max_inner=12,
              refine_max_outer=2, krylov_bc_fix=1, pcg_cap_start=20, graphs=1, pcd_visc_scale=1.0)


def run(max_coop):
    specs = cases.bubble_ensemble(2, grids=((32, 64), (64, 128)))
    for s, (nx, ny) in zip(specs, ((32, 64), (64, 128))):
        s["grid"] = Grid(nx, ny, 1.0, 2.0)
    with Batch([(s["grid"], ensemble_params(s, **SOLVER), MIXED) for s in specs], max_cluster=8,
               max_coop=max_coop) as b:
        for k, s in enumerate(specs):
            initial_bubble_state(b.case(k), s)
        b.run(1, 5e-4, 1, b.case(0).step_opts())
        return ([b.case(k).profile() for k in range(2)],
                [b.case(k).download_state(list(STATE_FIELDS)) for k in range(2)])


def test_max_coop_bounds_the_filter(gpu):
    want = run(0)
    assert [p["svof_grid"] for p in want[0]] == [4, 16]  # 512 cells per CTA
    for limit in (1, 3, 8):
        prof, got = run(limit)
        for p, a, b in zip(prof, got, want[1]):
            assert 1 <= p["svof_grid"] <= limit and p["pcg_grid"] <= limit
            for f in STATE_FIELDS:
                np.testing.assert_array_equal(a[f], b[f], err_msg=f)


def test_profile_reports_the_kernels_that_run(gpu):
    with Context(Grid(256, 256), Params()) as ctx:
        p = ctx.profile()
        assert p["svof_grid"] == 16 and p["pcg_grid"] == 64  # a cluster; 1,024 cells per CTA
