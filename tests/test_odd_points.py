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


# and it is not its own neighbour either, whichever kernel takes the query
@pytest.mark.parametrize("odd", ["nan", "nan z", "inf", "-inf"])
@pytest.mark.parametrize("k", [1, 16, 40])
@pytest.mark.parametrize("run", [False, True])  # spread over the cloud, or one after the other
def test_bounded_neighbours_of_odd_points(gpu_ctx, odd, k, run):
    from rvpoint_b200 import api
    c = odd_cloud(odd, at=np.arange(70) if run else None)
    q = c.aos()
    h = api.SpatialHash()
    h.setInputCloud(c, 0.2)
    h.build()
    for radius in (0.05, 0.5):
        offs, idx, d2 = h.radiusSearchBatch(c.x, c.y, c.z, radius)
        n = np.minimum(np.diff(offs), k)
        cut = np.concatenate([np.arange(a, a + m) for a, m in zip(offs, n)])
        assert (n[~np.isfinite(q).all(1)] == 0).all()
        o3, i3, e3 = h.radiusSearchBatch(c.x, c.y, c.z, radius, max_nn=k)
        assert np.array_equal(np.diff(o3), n)
        assert np.array_equal(i3, idx[cut]) and np.array_equal(bits(e3), bits(d2[cut]))
        i4, e4, n4 = h.knn(c.x, c.y, c.z, k, radius=radius)
        row = np.arange(k)[None] < n[:, None]
        assert np.array_equal(n4, n) and np.array_equal(i4[row], idx[cut])
        assert (i4[~row] == -1).all() and np.isinf(e4[~row]).all()
    i5, _, n5 = h.knn(c.x, c.y, c.z, k)  # without a bound
    if "nan" in odd:
        assert (n5[~np.isfinite(q).all(1)] == 0).all()
    assert (n5[np.isfinite(q).all(1)] == k).all()


# a list that is not wanted has no memory: short lists, longer ones (256 points)
# and those past shared memory (1024), for few queries and for packets of them
# (colliding cells repeat a point once per cell of the window: short radius only)
@pytest.mark.parametrize("radius,primes", [(0.3, None), (2.0, None), (30.0, None), (0.3, (1, 1))])
@pytest.mark.parametrize("nq", [300, 2100])
@pytest.mark.parametrize("mem", [0, 1])
def test_radius_search_without_a_list(gpu_ctx, radius, nq, mem, primes):
    import ctypes as C
    import torch
    from rvpoint_b200 import api
    c = D.room_cloud(n=2100, seed=4)
    h = api.SpatialHash()
    if primes:
        h.setHashPrimes(*primes)
    h.setInputCloud(c, 0.5)
    h.build()
    assert h.hasCollisions() == bool(primes)
    q = [torch.from_numpy(np.array(v[:nq])) for v in (c.x, c.y, c.z)]
    if mem == 1:
        q = [v.cuda() for v in q]
    api._prep(gpu_ctx, mem)
    ptr = lambda t: C.c_void_p(t.data_ptr()) if t is not None else None  # noqa: E731
    for max_nn in (0, 16, 100):
        offs, idx, d2 = h.radiusSearchBatch(*[v if mem else v.numpy() for v in q], radius,
                                            max_nn=max_nn)
        want = [torch.as_tensor(v) for v in (idx, d2)]
        for keep in ((0,), (1,), ()):
            lists = [torch.zeros_like(w) if i in keep else None for i, w in enumerate(want)]
            o = torch.zeros(nq + 1, dtype=torch.int64, device=q[0].device)
            total = C.c_size_t(0)
            st = gpu_ctx.L.rvp_hash_radius_search(
                h.h, *[ptr(v) for v in q], nq, radius, max_nn, mem, ptr(o), ptr(lists[0]),
                ptr(lists[1]), len(want[0]), C.byref(total))
            assert st == 0 and total.value == len(want[0])
            assert torch.equal(o, torch.as_tensor(offs))
            for i in keep:
                assert torch.equal(lists[i].view(torch.int32), want[i].view(torch.int32))


# more queries than one launch numbers (2^30): taken in parts, short and long
# lists (this takes some 75 GB)
@pytest.mark.parametrize("max_nn", [0, 70])
def test_radius_search_of_a_billion_queries(gpu_ctx, max_nn):
    import torch
    from rvpoint_b200 import api
    if torch.cuda.mem_get_info()[0] < 110 << 30:
        pytest.skip("needs 110 GB free")
    most = 1 << 30
    t = np.linspace(0, 1, 2000, dtype=np.float32)
    ctx = api.Context(0)
    h = api.SpatialHash(ctx)
    h.setInputCloud((t, t, t), 0.1)
    h.build()
    near = [0, most - 1, most, most + 4]
    v = torch.tensor([0.1, 0.5, 0.2, 0.45], device="cuda")
    q = torch.full((most + 5,), 1e3, device="cuda")
    q[near] = v
    offs, idx, d2 = h.radiusSearchBatch(q, q, q, 0.5, max_nn=max_nn)
    o2, i2, e2 = h.radiusSearchBatch(v, v, v, 0.5, max_nn=max_nn)
    assert int(o2.diff().max()) > (1024 if max_nn == 0 else 69)
    assert torch.equal(offs[near], o2[:-1]) and int(offs[-1]) == int(o2[-1])
    assert int((offs.diff() != 0).sum()) == len(near)
    assert torch.equal(idx, i2) and torch.equal(d2, e2)
    h.close()
    ctx.close()


# a hash copies its cloud, from another GPU's memory as well
def test_cloud_of_another_gpu(gpu_ctx):
    import torch
    from rvpoint_b200 import api
    if torch.cuda.device_count() < 2:
        pytest.skip("needs two GPUs")
    c = D.room_cloud(n=3000, seed=1)
    found = []
    for dev in ("cuda:0", "cuda:1"):
        h = api.SpatialHash()
        h.setInputCloud(tuple(torch.from_numpy(np.array(a)).to(dev) for a in (c.x, c.y, c.z)), 0.2)
        torch.cuda.synchronize(dev)
        h.build()
        found.append(h.knn(c.x, c.y, c.z, 8))
        h.close()
    assert all(np.array_equal(a, b) for a, b in zip(*found))


# a frame, or a whole cloud, whose largest (or smallest) coordinate is -0: its
# box takes it in
@pytest.mark.parametrize("sign", [-1, 1])
def test_coordinates_of_minus_zero(gpu_ctx, restatement, sign):
    import torch
    from rvpoint_b200 import api
    from rvpoint_b200.learned import DeviceBatch, PlaneScorer
    rng = np.random.default_rng(3)
    sizes = (17, 8, 40, 1, 300)
    n = sum(sizes)
    offs = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    p = (rng.uniform(0.05, 2.0, (n, 3)) * sign).astype(np.float32)
    for a, b in zip(offs, offs[1:]):  # each axis of each frame
        for axis in range(3):
            p[rng.integers(a, b), axis] = -0.0
    assert (p * sign).min() == 0
    b = DeviceBatch.from_host(D.Batch(p[:, 0].copy(), p[:, 1].copy(), p[:, 2].copy(), offs))
    s = PlaneScorer(n, len(sizes), ctx=gpu_ctx)
    cand = torch.arange(n, dtype=torch.int32, device="cuda")
    coffs = torch.from_numpy(offs).cuda()
    every = s.features(b, 1.0).cpu().numpy()
    among = s.features(b, 1.0, cand, coffs, among_candidates=True).cpu().numpy()
    s.close()
    assert np.array_equal(bits(every), bits(among))
    c = D.Cloud.from_xyz(p)
    got = api.euclidean_clusters(c, 0.3)
    want = restatement.euclidean_clusters(c, 0.3)
    assert len(got) == len(want) and all(np.array_equal(g, w) for g, w in zip(got, want))
    h = api.SpatialHash()
    h.setHashPrimes(1, 1)  # (the reference's buckets)
    h.setInputCloud(c, 0.5)
    h.build()
    o, i, _ = h.radiusSearchBatch(c.x, c.y, c.z, 0.3)
    o2, i2, _ = restatement.radius_search(c, 0.5, 0.3, p1=1, p2=1)
    assert np.array_equal(o, o2) and np.array_equal(i, i2)
