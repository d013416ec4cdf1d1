"""A pipeline on the box tree: no grid until a kernel mode searches one."""
import ctypes as C

import numpy as np
import pytest

from rvpoint_b200 import datasets as D

pytestmark = pytest.mark.gpu


def live(L):
    d, p = C.c_longlong(0), C.c_longlong(0)
    L.rvp_debug_live_bytes(C.byref(d), C.byref(p))
    return d.value


def same(a, b):
    return a.keys() == b.keys() and all(
        np.array_equal(np.asarray(a[k]), np.asarray(b[k]), equal_nan=True) for k in a)


# a fit on a sparse batch and one on a dense batch: no table of the tree's runs
# overflows, and a mode on the grid afterwards has room for the last batch
def test_fit_after_runs_on_the_tree(gpu_ctx):
    from rvpoint_b200.api import Pipeline
    sparse = D.lidar_batch(n_frames=2, seed=3, min_pts=100, max_pts=200)
    dense = D.lidar_batch(n_frames=2, seed=4, min_pts=30_000, max_pts=40_000)
    pipe = Pipeline(100_000, 2, ctx=gpu_ctx)
    for b in (sparse, dense):
        got = pipe.run_host(b)
        pipe.check()
        pipe.fit_tables()
        pipe.check()
    pipe.set_tuning(0.25, 0, 1)
    pipe.check()
    assert same(pipe.run_host(dense), got)
    pipe.check()
    pipe.close()


@pytest.mark.parametrize("points,frames", [(400_000, 4), (70_000, 120)])
def test_memory_by_mode(gpu_ctx, points, frames):
    from rvpoint_b200.api import Pipeline
    base = live(gpu_ctx.L)
    size = {}
    for mode in (0, 1, 3):
        pipe = Pipeline(points, frames, queries_per_warp=mode, ctx=gpu_ctx)
        size[mode] = live(gpu_ctx.L) - base
        if mode == 0:  # a grid mode afterwards takes what it needs
            pipe.set_tuning(0.25, 0, 1)
            assert live(gpu_ctx.L) - base > size[0]
        pipe.close()
    assert size[0] == size[3] < 0.8 * size[1]


def test_no_memory_for_the_grid(gpu_ctx):
    from rvpoint_b200 import _lib
    from rvpoint_b200.api import Pipeline
    b = D.lidar_batch(n_frames=2, seed=3, min_pts=3000, max_pts=6000)
    pipe = Pipeline(20_000, 2, ctx=gpu_ctx)
    got = pipe.run_host(b)
    for after in (0, 3, 9):
        gpu_ctx.L.rvp_debug_fail_allocation(after)
        try:
            with pytest.raises(_lib.RvpError):
                pipe.set_tuning(0.25, 0, 1)
        finally:
            gpu_ctx.L.rvp_debug_fail_allocation(-1)
        assert same(pipe.run_host(b), got)
    pipe.set_tuning(0.25, 0, 1)
    assert same(pipe.run_host(b), got)
    pipe.close()
