"""Kernels at the sizes where they can go wrong (tile edges, remainders, the
smallest and largest of a range), against the CPU oracle or numpy."""
import numpy as np
import pytest

from rvpoint_b200 import datasets as D

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a, dtype=np.float32).view(np.int32)


# SOR statistics: the float sums are scanned in chunks of 8192 values, runs of
# 16 per thread; a lattice repeats few distances, so many additions are ties
@pytest.mark.parametrize("n", [4, 15, 16, 17, 511, 8191, 8192, 8193, 16385])
@pytest.mark.parametrize("cloud", ["lattice", "room"])
def test_sor_statistics_sum_in_order(gpu_ctx, restatement, n, cloud):
    from rvpoint_b200.api import sor_rvv
    if cloud == "lattice":
        i = np.arange(n)
        c = D.Cloud.from_xyz(np.stack([i % 23, (i // 23) % 29, i // 667], 1) * 0.125)
    else:
        c = D.room_cloud(n=n, seed=n)
    out, mean, keep = sor_rvv(c, 3, 0.5, return_stats=True)
    out2, mean2, keep2 = restatement.sor_exact(c, 3, 0.5)
    assert np.array_equal(bits(mean), bits(mean2))
    assert np.array_equal(keep, keep2) and np.array_equal(bits(out), bits(out2))


# the voxel grid sorts its keys: up to 148 x 4096 of them in one cooperative
# kernel (512 threads, up to eight keys each), more in tiles of 4096
@pytest.mark.parametrize("n", [1, 31, 513, 4097, 75_777, 606_208, 606_209, 2_424_833])
def test_sorted_voxels(gpu_ctx, restatement, n):
    from rvpoint_b200.api import voxel_grid_downsamp_rvv_v2
    rng = np.random.default_rng(n)
    c = D.Cloud.from_xyz(rng.uniform(-40, 40, (n, 3)) * [1.0, 0.5, 0.02])
    out, keys = voxel_grid_downsamp_rvv_v2(c, 0.25, return_keys=True)
    out2, keys2 = restatement.voxel_grid(c, 0.25)
    assert np.array_equal(keys, keys2) and np.array_equal(bits(out), bits(out2))
