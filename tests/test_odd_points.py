"""Points without a position (a NaN or infinite coordinate) and optional outputs."""
import numpy as np
import pytest

from rvpoint_b200 import datasets as D
from test_kernel_edges import bits

pytestmark = pytest.mark.gpu


def odd_cloud(odd, n=3000, at=None):
    """A room with 70 odd points in it (two packets of queries and more)."""
    p = D.room_cloud(n=n, seed=11).aos().astype(np.float32)
    at = np.random.default_rng(2).choice(n, 70, replace=False) if at is None else at
    if odd == "nan":
        p[at] = np.nan
    elif odd == "nan z":
        p[at, 2] = np.nan
    else:
        p[at, 1] = float(odd)
    return D.Cloud.from_xyz(p)


# such a point has no neighbours: its mean is the search radius
@pytest.mark.parametrize("odd", ["nan", "nan z", "inf", "-inf"])
@pytest.mark.parametrize("k", [3, 16, 40])
def test_sor_within_a_radius_of_odd_points(gpu_ctx, restatement, odd, k):
    from rvpoint_b200 import api
    c = odd_cloud(odd)
    h = api.SpatialHash()
    h.setInputCloud(c, 0.2)
    h.build()
    out, mean, keep = api.sor_spatial_hash(c, h, k, 1.0, 0.2, return_stats=True)
    out2, mean2, keep2 = restatement.sor_radius(c, 0.2, k, 1.0, 0.2)
    assert np.array_equal(bits(mean), bits(mean2)) and np.array_equal(keep, keep2)
    assert keep.any() and np.array_equal(bits(out), bits(out2))
