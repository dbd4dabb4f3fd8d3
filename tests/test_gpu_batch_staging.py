"""The cases of a batch share one page-locked staging area: a batch's locked
memory does not grow by an area per case, and host threads that move arrays of
different cases at the same time, where one of them finds the area taken, get
their own values."""
import threading

import numpy as np
import pytest

from conftest import rfield
from coupled_codefort_2d_b200 import cases
from coupled_codefort_2d_b200._lib import MIXED
from coupled_codefort_2d_b200.batch import Batch, ensemble_params
from coupled_codefort_2d_b200.layout import Grid

pytestmark = pytest.mark.gpu

SOLVER = dict(tol_bicgstab2=1e-6, max_iter_bicgstab2=200, refine=2, refine_inner_tol=1e-1, refine_max_inner=12,
              refine_max_outer=2, krylov_bc_fix=1, pcg_cap_start=20, graphs=1, pcd_visc_scale=1.0)


def batch(n):
    specs = cases.bubble_ensemble(n, grids=((128, 256),))
    return Batch([(s["grid"], ensemble_params(s, **SOLVER), MIXED) for s in specs], max_cluster=16)


def locked():
    """MiB of page-locked host memory of this process (shared pages of the driver)."""
    with open("/proc/self/status") as f:
        return next(int(line.split()[1]) for line in f if line.startswith("RssShmem")) / 1024


def test_locked_memory_does_not_grow_with_the_cases(gpu):
    with batch(1):
        pass
    a = locked()
    with batch(12):
        assert locked() - a < 4 + 12 * 0.5  # the area, and each case's mirrors


def test_threads_move_arrays_of_different_cases(gpu):
    g = Grid(128, 256, 1.0, 2.0)
    bad = []
    with batch(4) as b:
        views = [b.case(k) for k in range(4)]

        def work(k):
            rng = np.random.default_rng(k)
            for _ in range(40):
                st = {f: rfield(rng, g, kind) for f, kind in (("u_vel", "u"), ("c_field", "cell"), ("zeta", "vert"))}
                views[k].upload_state(st)
                for f, a in st.items():
                    if not np.array_equal(views[k].download(f), a):
                        bad.append((k, f))

        ts = [threading.Thread(target=work, args=(k,)) for k in range(4)]
        for t in ts:
            t.start()
        for t in ts:
            t.join()
    assert not bad
