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


# SOR statistics from 1025 values on: pairs of segments of 256, 512 at a time;
# one value near 2^20 first takes the float sum away from the true one (0.1 is
# rounded to 0.125), so the binades foreseen for whole runs are not the sum's
@pytest.mark.parametrize("n,far", [(1024, 0), (1025, 0), (30_000, 0), (30_000, 2**20 - 2000),
                                   (131_330, 0)])
def test_sor_statistics_segments(gpu_ctx, n, far):
    from rvpoint_b200.api import sor_rvv
    i = np.arange(n)
    p = np.stack([i % 31, (i // 31) % 37, i // 1147], 1).astype(np.float32) * np.float32(0.1)
    if far:
        p[0] = [-far, 0, 0]
    else:
        p += np.random.default_rng(n).uniform(0, 0.05, p.shape).astype(np.float32)
    c = D.Cloud.from_xyz(p)
    _, mean, _ = sor_rvv(c, 3, 0.5, return_stats=True)
    f = np.float32
    mu = np.add.accumulate(mean)[-1] / f(n)  # in order, in float
    sd = np.sqrt(np.add.accumulate((mean - mu) * (mean - mu))[-1] / f(n))
    # a threshold on a value: one unit less would drop its point
    target = np.sort(mean)[int(0.7 * n)] if not far else np.sort(mean)[-2]
    alpha = f((target - mu) / sd)
    for _ in range(64):
        t = mu + alpha * sd
        if t == target:
            break
        alpha = np.nextafter(alpha, f(np.inf) if t < target else f(-np.inf))
    _, _, keep = sor_rvv(c, 3, float(alpha), return_stats=True)
    assert np.array_equal(keep.astype(bool), mean <= mu + alpha * sd)


# neighbourhoods among the candidates: scenes of up to 1024 and up to 2048
# candidates have a tree each, larger ones are searched by brute force; a point
# that is not finite takes its scene there as well
@pytest.mark.parametrize("sizes", [(3, 17, 33, 1), (1023, 1024, 1025), (2047, 2048, 2049, 40)])
@pytest.mark.parametrize("lattice", [False, True])
def test_candidate_neighbourhoods(gpu_ctx, sizes, lattice):
    import torch
    from rvpoint_b200.learned import DeviceBatch, PlaneScorer
    n = sum(sizes)
    rng = np.random.default_rng(n)
    i = np.arange(n)
    p = (np.stack([i % 13, (i // 13) % 11, i // 143], 1) % 9 * 0.25 if lattice
         else rng.uniform(-5, 5, (n, 3)) * [1, 1, 0.1]).astype(np.float32)
    offs = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    b = DeviceBatch.from_host(D.Batch(p[:, 0].copy(), p[:, 1].copy(), p[:, 2].copy(), offs))
    s = PlaneScorer(n, len(sizes), ctx=gpu_ctx)
    cand = torch.arange(n, dtype=torch.int32, device="cuda")
    coffs = torch.from_numpy(offs).cuda()
    ref = s.features(b, 1.0).cpu().numpy()  # among all points, by the grid
    got = s.features(b, 1.0, cand, coffs, among_candidates=True).cpu().numpy()
    assert np.array_equal(bits(got), bits(ref))
    b.x[0] = float("inf")  # (the other scenes are as before)
    got = s.features(b, 1.0, cand, coffs, among_candidates=True).cpu().numpy()
    assert np.array_equal(bits(got[sizes[0]:]), bits(ref[sizes[0]:]))
    s.close()


# rows of neighbours for the normals in high precision: K = 4, 17, 33 and 64
@pytest.mark.parametrize("n,k", [(5, 3), (33, 16), (64, 32), (1025, 63), (4097, 16)])
def test_precise_rows(gpu_ctx, n, k):
    from rvpoint_b200.api import normal_estimation_precise
    c = D.room_cloud(n=max(n, 50), seed=n).subset(np.arange(n))
    k = min(k, n - 1)
    normals, _, _ = normal_estimation_precise(c, k)
    p = c.aos().astype(np.float64)
    idx, _ = brute_knn(c.aos(), c.aos(), k + 1)
    q = p[idx] - p[idx].mean(1, keepdims=True)
    w, v = np.linalg.eigh(np.einsum("nki,nkj->nij", q, q))
    a = np.abs((normals * v[:, :, 0]).sum(1))
    clear = w[:, 0] < 0.5 * w[:, 1]  # a normal that is well defined
    assert clear.any() and (1 - a[clear] < 1e-5).all()


# the batched pipeline: its trees, with frames that end at a leaf, a node or
# after one point, empty ones among them, and the grid where many tiny frames
# would leave the trees mostly empty (130 frames in a batch of 4000 points)
@pytest.mark.parametrize("sizes,points", [((1023, 0, 1024, 1025, 33, 2049, 1, 0), 8192),
                                          ((40, 31, 1, 0, 65) * 26, 4000)])
def test_pipeline_frames(gpu_ctx, sizes, points):
    import torch
    from rvpoint_b200.api import Pipeline
    rng = np.random.default_rng(len(sizes))
    n = sum(sizes)
    assert (1024 * len(sizes) <= points + 65_536) == (len(sizes) == 8)
    # one point per voxel of 0.1: a frame's voxels are its points
    p = []
    for m in sizes:
        i = rng.choice(64 * 64 * 4, m, replace=False)
        p.append(np.stack([i % 64, i // 64 % 64, i // 4096], 1) * 0.1 + rng.uniform(0.02, 0.08, (m, 3)))
    p = np.concatenate(p).astype(np.float32)
    offs = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    batch = D.Batch(p[:, 0].copy(), p[:, 1].copy(), p[:, 2].copy(), offs)
    got = []
    for mode in (0, 3, 1):  # trees (or the grid), and a warp per query on the grid
        pipe = Pipeline(points, len(sizes), leaf_size=0.1, sor_k=16, normal_k=16,
                        ransac_iters=20, queries_per_warp=mode, ctx=gpu_ctx)
        got.append(pipe.run_host(batch))
        pipe.close()
    for g in got[:2]:
        assert g.keys() == got[2].keys()
        for k in g:
            assert np.array_equal(np.asarray(g[k]), np.asarray(got[2][k]), equal_nan=True), k


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


def brute_knn(p, q, k, r2=np.inf):
    """(indices, d2) rows in (d2, index) order, -1 / inf past the found."""
    d = [p[None, :, a] - q[:, None, a] for a in range(3)]
    d2 = (d[0] * d[0] + d[1] * d[1]) + d[2] * d[2]
    idx = np.full((len(q), k), -1, np.int32)
    dist = np.full((len(q), k), np.inf, np.float32)
    for i in range(len(q)):
        o = np.argsort(d2[i], kind="stable")
        o = o[d2[i][o] <= r2][:k]
        idx[i, :len(o)], dist[i, :len(o)] = o, d2[i][o]
    return idx, dist


# the box tree: leaves of 32 points, 32 children per node; lists of up to 9,
# 17, 25, 33 and 64 distances; equal distances go by index
@pytest.mark.parametrize("n,k", [(1, 1), (2, 5), (31, 9), (32, 17), (33, 10), (65, 64),
                                 (1023, 18), (1024, 33), (1025, 25), (2049, 34), (2500, 1)])
@pytest.mark.parametrize("cloud", ["room", "lattice"])
def test_tree_knn(gpu_ctx, n, k, cloud):
    from rvpoint_b200.api import SpatialHash
    if cloud == "lattice":
        i = np.arange(n)
        c = D.Cloud.from_xyz(np.stack([i % 7, (i // 7) % 5, i // 35], 1) % 6 * 0.25)
    else:
        c = D.room_cloud(n=max(n, 50), seed=n).subset(np.arange(n))
    p = c.aos()
    h = SpatialHash()
    h.setInputCloud(c, 0.5)
    h.build()
    rng = np.random.default_rng(n)
    other = np.concatenate([p[: n // 2] + np.float32(0.01),
                            rng.uniform(-9, 9, (37, 3)).astype(np.float32)])
    for q, r in ((p, 0.0), (other, 0.0), (p[::-1], 0.3), (other, 0.6)):
        q = np.ascontiguousarray(q)
        idx, d2, cnt = h.knn(q[:, 0], q[:, 1], q[:, 2], k, radius=r)
        r2 = np.float32(r) * np.float32(r) if r else np.inf
        idx2, dist2 = brute_knn(p, q, k, r2)
        assert np.array_equal(idx, idx2) and np.array_equal(bits(d2), bits(dist2))
        assert np.array_equal(cnt, (idx2 >= 0).sum(1))


@pytest.mark.parametrize("n", [40, 32_768, 32_769, 70_001])
def test_tree_levels(gpu_ctx, restatement, n):
    """SOR means, and normals of both kinds, through every level of the tree."""
    from rvpoint_b200 import api
    c = D.room_cloud(n=n, seed=n)
    assert np.array_equal(bits(api.sor_rvv(c, 8, 1.0, return_stats=True)[1])[:2000],
                          bits(_means(c.aos(), 8))[:2000])
    nx, ny, nz = api.normal_estimation_sc(c, 9)
    nrm, _, _ = api.normal_estimation_precise(c, 9)
    assert np.allclose(nx * nx + ny * ny + nz * nz, 1.0, atol=1e-5)
    assert np.allclose((nrm ** 2).sum(1), 1.0, atol=1e-5)


def _means(p, k):
    out = np.zeros(len(p), np.float32)
    for i in range(min(len(p), 2000)):
        d = p - p[i]
        d2 = np.sort((d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]) + d[:, 2] * d[:, 2])[1:k + 1]
        s = np.float32(0)
        for v in np.sqrt(d2):
            s = np.float32(s + v)
        out[i] = s / np.float32(k)
    return out


def brute_radius(p, q, r):
    d = [p[None, :, a] - q[:, None, a] for a in range(3)]
    d2 = (d[0] * d[0] + d[1] * d[1]) + d[2] * d[2]
    r2 = np.float32(r) * np.float32(r)
    offs, idx, dist = [0], [], []
    for row in d2:
        o = np.argsort(row, kind="stable")
        o = o[row[o] <= r2]
        idx.append(o)
        dist.append(row[o])
        offs.append(offs[-1] + len(o))
    return np.asarray(offs), np.concatenate(idx).astype(np.int32), np.concatenate(dist)


# radius lists over the tree: lists of up to 32, 64, 512 and 1024 points are
# ordered in different ways, longer ones apart; up to 2048 queries go one per
# warp in their own order
@pytest.mark.parametrize("n,radius", [(1, 1.0), (33, 0.0), (700, 0.4), (2047, 0.8), (2049, 0.8),
                                      (3000, 1.1), (3000, 20.0)])
@pytest.mark.parametrize("cloud", ["room", "lattice"])
def test_tree_radius(gpu_ctx, n, radius, cloud):
    from rvpoint_b200 import api
    if cloud == "lattice":
        i = np.arange(n)
        c = D.Cloud.from_xyz(np.stack([i % 13, (i // 13) % 11, i // 143], 1) % 9 * 0.25)
    else:
        c = D.room_cloud(n=max(n, 50), seed=n).subset(np.arange(n))
    p = c.aos()
    h = api.SpatialHash()
    h.setInputCloud(c, 0.5)
    h.build()
    assert not h.hasCollisions()
    q = np.concatenate([p[: n // 3] + np.float32(0.02), p[::-1]])[: max(1, n - 1)]
    for q in (p, np.ascontiguousarray(q)):
        offs, idx, d2 = h.radiusSearchBatch(q[:, 0], q[:, 1], q[:, 2], radius)
        offs2, idx2, dist2 = brute_radius(p, q, radius)
        assert np.array_equal(offs, offs2) and np.array_equal(idx, idx2)
        assert np.array_equal(bits(d2), bits(dist2))
        cut, idx3, _ = h.radiusSearchBatch(q[:, 0], q[:, 1], q[:, 2], radius, max_nn=70)
        first = np.concatenate([idx2[a:min(a + 70, b)] for a, b in zip(offs2, offs2[1:])])
        assert np.array_equal(np.diff(cut), np.minimum(np.diff(offs2), 70))
        assert np.array_equal(idx3, first)


# list offsets: one block scans up to 49152 counts, 16384 at a time
@pytest.mark.parametrize("n", [16_383, 16_385, 49_152, 49_153])
def test_radius_offsets(gpu_ctx, n):
    from rvpoint_b200 import api
    i = np.arange(n)
    c = D.Cloud.from_xyz(np.stack([i % 37, (i // 37) % 41, i // 1517], 1) * 0.25)
    h = api.SpatialHash()
    h.setInputCloud(c, 0.5)
    h.build()
    q = c.aos()
    q[::3, 2] = 1e3  # nothing near these
    offs, idx, d2 = h.radiusSearchBatch(q[:, 0], q[:, 1], q[:, 2], 0.1)
    assert np.array_equal(np.diff(offs), (i % 3 != 0).astype(np.int64))
    assert np.array_equal(idx, i[i % 3 != 0]) and not d2.any()


@pytest.mark.parametrize("radius", [0.0, 0.03, 0.3, 2.0])  # 0, tens, hundreds, all as neighbours
def test_radius_normals_lists(gpu_ctx, restatement, radius):
    from rvpoint_b200 import api
    c = D.room_cloud(n=1500, seed=3)
    h = api.SpatialHash()
    h.setInputCloud(c, 0.1)
    h.build()
    got = np.stack(api.normal_estimation_rvv(c, h, 10, radius), 1)
    want = np.asarray(restatement.normals_radius(c, 0.1, radius))
    assert np.array_equal((got != 0).any(1), (want != 0).any(1))
    # (the rotations branch on the largest entry: a few differ by more)
    assert (np.abs(got - want).max(1) < 1e-4).mean() > 0.995


# a leaf of points around a dense cloud: its packet would test all the leaves
def test_radius_normals_of_scattered_points(gpu_ctx, restatement):
    from rvpoint_b200 import api
    rng = np.random.default_rng(7)
    near = rng.uniform(-1, 1, (12_000, 3)) * [1, 1, 0.01]
    c = D.Cloud.from_xyz(np.concatenate([near, rng.uniform(-6, 6, (60, 3))])[rng.permutation(12_060)])
    h = api.SpatialHash()
    h.setInputCloud(c, 0.1)
    h.build()
    got = np.stack(api.normal_estimation_rvv(c, h, 10, 0.06), 1)
    want = np.asarray(restatement.normals_radius(c, 0.1, 0.06))
    assert np.array_equal((got != 0).any(1), (want != 0).any(1))
    assert (np.abs(got - want).max(1) < 1e-4).mean() > 0.995


@pytest.mark.parametrize("primes,collide", [((73856093, 19349663), False), ((1, 1), True),
                                            ((-73856093, 19349663), False), ((0, 5), True),
                                            ((1 << 41, 3), True)])  # (3, 0, 0) and (0, 0, 1)
def test_collisions_found(gpu_ctx, restatement, primes, collide):
    from rvpoint_b200 import api
    c = D.room_cloud(n=4000, seed=5)
    h = api.SpatialHash()
    h.setHashPrimes(*primes)
    h.setInputCloud(c, 0.1)
    h.build()
    assert h.hasCollisions() == collide
    offs, idx, _ = h.radiusSearchBatch(c.x, c.y, c.z, 0.1)
    o2, i2, _ = restatement.radius_search(c, 0.1, 0.1, p1=primes[0], p2=primes[1])
    assert np.array_equal(offs, o2) and np.array_equal(idx, i2)


# RANSAC on one cloud: hypotheses are counted in rounds of 64 to 1024, over
# chunks of 2048 points, 64 hypotheses at a time; the stop and the libc state
# are the sequential loop's
@pytest.mark.parametrize("n,iters", [(3, 5), (50, 1), (2047, 63), (2049, 65), (20_000, 2500),
                                     (1_700_000, 300)])
def test_ransac_rounds(gpu_ctx, restatement, n, iters):
    from oracle import oracle as O
    from rvpoint_b200 import api
    c = D.room_cloud(n=max(n, 50), seed=n).subset(np.arange(n))
    stream = O.libc_rand_stream(3 * iters)
    best, model, _, _, ran = restatement.ransac_plane(c, 0.01, iters, stream)
    for kw in ({}, {"rand_stream": stream}):
        got, m = api.ransac_plane_rvv(c, 0.01, iters, **kw)
        assert got == best and np.array_equal(bits(m), bits(np.asarray(model, np.float32)))
    best2, _, _, ran2 = api.ransac_plane_rvv(c, 0.01, iters, return_counts=True)
    assert best2 == best and ran2 == ran


# up to 24576 queries (81920 within a radius) go one per warp, more in packets
@pytest.mark.parametrize("nq,radius", [(24_576, 0.0), (81_920, 0.3)])
@pytest.mark.parametrize("k", [1, 9, 17, 40])
@pytest.mark.parametrize("cloud", ["room", "lattice"])
def test_few_and_many_queries(gpu_ctx, nq, radius, k, cloud):
    from rvpoint_b200.api import SpatialHash
    n = 50_000
    if cloud == "lattice":
        i = np.arange(n)
        c = D.Cloud.from_xyz(np.stack([i % 41, (i // 41) % 43, i // 1763], 1) % 38 * 0.25)
    else:
        c = D.room_cloud(n=n, seed=k)
    p = c.aos()
    h = SpatialHash()
    h.setInputCloud(c, 0.5)
    h.build()
    rng = np.random.default_rng(nq)
    q = np.concatenate([p[rng.permutation(nq) % n][:nq - 500],
                        rng.uniform(-9, 9, (501, 3)).astype(np.float32)])
    few = h.knn(*q[:nq].T, k, radius)
    many = h.knn(*q.T, k, radius)
    for a, b in zip(few, many):
        assert np.array_equal(a.view(np.int32), b[:nq].view(np.int32))
    at = np.concatenate([rng.choice(nq, 100, replace=False), [nq]])
    idx, d2 = brute_knn(p, q[at], k, np.float32(radius) * np.float32(radius) if radius else np.inf)
    assert np.array_equal(many[0][at], idx) and np.array_equal(bits(many[1][at]), bits(d2))
    assert np.array_equal(many[2][at], (idx >= 0).sum(1))


# a call for few queries is one kernel (the queries are neither sorted nor
# compared with the cloud)
def test_few_queries_are_one_launch(gpu_ctx):
    import torch
    from rvpoint_b200.api import SpatialHash
    c = D.room_cloud(n=60_000, seed=1)
    v = [torch.from_numpy(np.array(a)).cuda() for a in (c.x, c.y, c.z)]
    h = SpatialHash()
    h.setInputCloud(v, 0.5)
    h.build()
    for nq, radius in ((1, 0.0), (700, 0.0), (24_576, 0.0), (40_000, 0.3)):
        before = gpu_ctx.launches
        h.knn(*[a[:nq] for a in v], 16, radius)
        assert gpu_ctx.launches - before == 1


# the codes that order the points are as long as the cloud needs: one far or
# infinite point in a cloud of no order, or points dense in a few places, leave
# the leaves small (with 32 bits all of the cloud was one cell: 150 times as long)
@pytest.mark.parametrize("far", [1e6, 1e9, float("inf"), "clusters"])
def test_far_points_do_not_spoil_the_order(gpu_ctx, far):
    import time
    import torch
    from rvpoint_b200.api import SpatialHash
    rng = np.random.default_rng(5)
    p = (rng.uniform(-40, 40, (100_000, 3)) * [1, 1, 0.02]).astype(np.float32)
    times, found = [], []
    for spoilt in (False, True):
        c = p.copy()
        if spoilt:
            if far == "clusters":
                c[:50] = rng.choice([-3e6, 3e6], (50, 3))
            else:
                c[0] = far
        v = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in c.T]
        q = [a[50:] for a in v]
        h = SpatialHash()
        h.setInputCloud(v, 0.5)
        h.build()
        found.append([a.cpu().numpy() for a in h.radiusSearchBatch(*q, 0.3)])
        t = []
        for _ in range(5):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            h.radiusSearchBatch(*q, 0.3)
            torch.cuda.synchronize()
            t.append(time.perf_counter() - t0)
        times.append(min(t))
    near = np.diff(found[0][0])
    lists = [[set(i[a:b][i[a:b] >= 50]) for a, b in zip(o[:500], o[1:501])] for o, i, _ in found]
    assert lists[0] == lists[1] and near.max() > 3
    assert times[1] < 10 * times[0]


# many points in one place (returns that a sensor reports as 0, 0, 0), others
# far around: their packets do not test each other's leaves
def test_points_in_one_place(gpu_ctx, restatement):
    import time
    import torch
    from rvpoint_b200 import api
    rng = np.random.default_rng(3)
    p = rng.normal(0, 1, (150_000, 3))
    p = (p / np.linalg.norm(p, axis=1)[:, None] * rng.uniform(5, 6, (150_000, 1))).astype(np.float32)
    at = rng.permutation(len(p))[:3000]
    times = []
    for same in (False, True):
        if same:
            p[at] = 0
        v = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in p.T]
        h = api.SpatialHash()
        h.setInputCloud(v, 0.5)
        h.build()
        t = []
        for _ in range(6):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            idx, d2, cnt = h.knn(*v, 16, 0.1)
            torch.cuda.synchronize()
            t.append(time.perf_counter() - t0)
        times.append(min(t))
    # (twice as long without the packets' early end and more)
    assert times[1] < 1.9 * times[0]
    first = np.sort(at)[:16]
    assert np.array_equal(idx[at].cpu().numpy(), np.tile(first, (3000, 1)))
    assert not d2[at].any() and bool((cnt[at] == 16).all())
    few = D.Cloud.from_xyz(np.concatenate([p[at[:40]], p[:2500]]))
    _, mean, keep = api.sor_rvv(few, 8, 1.0, return_stats=True)
    _, mean2, keep2 = restatement.sor_exact(few, 8, 1.0)
    assert np.array_equal(bits(mean), bits(mean2)) and np.array_equal(keep, keep2)


# equal distances are ordered where a packet finds them: on a lattice, whose
# every query has some, the second kernel is left with few
@pytest.mark.parametrize("k", [6, 16])
def test_lattice_stays_with_the_packets(gpu_ctx, k):
    from rvpoint_b200.api import Pipeline
    i = np.arange(20_000)
    p = np.stack([i % 27, (i // 27) % 27, i // 729], 1).astype(np.float32) * 0.25 + np.float32(0.125)
    b = D.Batch(p[:, 0].copy(), p[:, 1].copy(), p[:, 2].copy(), np.array([0, len(p)], np.int64))
    got = []
    for mode in (0, 1):
        pipe = Pipeline(len(p), 1, leaf_size=0.25, sor_k=k, normal_k=k, sor_alpha=3.0,
                        queries_per_warp=mode, ctx=gpu_ctx)
        pipe.knn_stats(True)
        got.append(pipe.run_host(b))
        sor = pipe.knn_stats(False)["sor"]
        pipe.close()
        if mode == 0:  # (warp_ring0: the second kernel's)
            assert sor["tile_l0"] + sor["warp_ring0"] == len(p) and sor["warp_ring0"] < len(p) / 4
    for key in got[0]:
        assert np.array_equal(np.asarray(got[0][key]), np.asarray(got[1][key]), equal_nan=True), key


# and in the order of their indices, for many queries (packets) of every list
@pytest.mark.parametrize("k", [2, 7, 9, 10, 16, 17])
def test_packets_order_ties_by_index(gpu_ctx, k):
    from rvpoint_b200.api import SpatialHash
    n = 60_000
    i = np.random.default_rng(k).permutation(n)
    c = D.Cloud.from_xyz(np.stack([i % 41, (i // 41) % 43, i // 1763], 1) * 0.25)
    p = c.aos()
    h = SpatialHash()
    h.setInputCloud(c, 0.5)
    h.build()
    at = np.random.default_rng(0).choice(n, 150, replace=False)
    for q in (p, p + np.float32(0.125)):  # the cloud's own, and the middles of its cells
        for r in (0.0, 0.5):
            idx, d2, cnt = h.knn(*q.T, k, r)
            idx2, dist2 = brute_knn(p, q[at], k, np.float32(r) * np.float32(r) if r else np.inf)
            assert np.array_equal(idx[at], idx2) and np.array_equal(bits(d2[at]), bits(dist2))
            assert np.array_equal(cnt[at], (idx2 >= 0).sum(1))


# radius lists: up to 65536 queries go one per warp in their own order, more in
# packets; lists of a few points, of hundreds and of more than 1024
@pytest.mark.parametrize("max_nn", [0, 70])
@pytest.mark.parametrize("mixed", [False, True])  # other queries, or the cloud itself
def test_few_and_many_radius_queries(gpu_ctx, max_nn, mixed):
    from rvpoint_b200 import api
    nq = 65_536
    rng = np.random.default_rng(1)
    p = rng.uniform(-20, 20, (nq + 1, 3)) * [1, 1, 0.05]
    p[rng.permutation(nq)[:1200]] = rng.normal(0, 0.05, (1200, 3))
    p[rng.permutation(nq)[:400]] = rng.normal(3, 0.05, (400, 3))
    p = p.astype(np.float32)
    h = api.SpatialHash()
    h.setInputCloud((p[:, 0], p[:, 1], p[:, 2]), 0.5)
    h.build()
    q = p + np.float32(0.01) if mixed else p
    few = h.radiusSearchBatch(*q[:nq].T, 0.3, max_nn=max_nn)
    many = h.radiusSearchBatch(*q.T, 0.3, max_nn=max_nn)
    m = int(few[0][-1])
    assert np.array_equal(few[0], many[0][:-1])
    assert np.array_equal(few[1], many[1][:m]) and np.array_equal(bits(few[2]), bits(many[2][:m]))
    if max_nn == 0:
        n = np.diff(many[0])
        assert n.max() > 1024 and ((n > 256) & (n < 1024)).any() and (n < 32).any()
    at = np.concatenate([rng.choice(nq, 60, replace=False), np.argsort(np.diff(few[0]))[-3:], [nq]])
    _, idx, d2 = brute_radius(p, q[at], 0.3)
    o = brute_radius(p, q[at], 0.3)[0]
    cut = max_nn or len(p)
    for i, a in enumerate(at):
        s = slice(many[0][a], many[0][a + 1])
        assert np.array_equal(many[1][s], idx[o[i]:o[i + 1]][:cut])
        assert np.array_equal(bits(many[2][s]), bits(d2[o[i]:o[i + 1]][:cut]))


# radius normals: up to 32768 points go one per warp, more in packets; lists of
# a few points, past a lane's (48), past a short list's (256) and past 1024
def test_few_and_many_radius_normals(gpu_ctx, restatement):
    from rvpoint_b200 import api
    n = 32_768
    rng = np.random.default_rng(4)
    p = rng.uniform(-20, 20, (n + 1, 3)) * [1, 1, 0.01]
    for at, m in (((0, 0, 0), 1300), ((4, 0, 0), 500), ((8, 0, 0), 100)):
        p[rng.permutation(n)[:m]] = rng.normal(0, 0.05, (m, 3)) * [1, 1, 0.1] + at
    p[n] = 300
    p = p.astype(np.float32)
    got = []
    for m in (n, n + 1):
        c = D.Cloud.from_xyz(p[:m])
        h = api.SpatialHash()
        h.setInputCloud(c, 0.3)
        h.build()
        got.append(np.stack(api.normal_estimation_rvv(c, h, 10, 0.3), 1))
    lists = np.diff(h.radiusSearchBatch(*p.T, 0.3)[0])
    for lo, hi in ((3, 48), (49, 256), (257, 1024), (1025, n)):
        assert ((lists >= lo) & (lists <= hi)).any()
    assert np.array_equal(bits(got[0]), bits(got[1][:n])) and not got[1][n].any()
    want = np.asarray(restatement.normals_radius(c, 0.3, 0.3))
    assert np.array_equal((got[1] != 0).any(1), (want != 0).any(1))
    # (the rotations branch on the largest entry: a few differ by more)
    assert (np.abs(got[1] - want).max(1) < 1e-4).mean() > 0.995


# points of some 60 neighbours each: their normals by whole warps, not by one
# lane (less than three times a search for their lists; it was four)
def test_radius_normals_of_longer_lists(gpu_ctx):
    import time
    import torch
    from rvpoint_b200 import api
    x = np.random.default_rng(7).uniform(-50, 50, 150_000).astype(np.float32)
    v = [torch.from_numpy(a).cuda() for a in (x, np.zeros_like(x), np.zeros_like(x))]
    h = api.SpatialHash()
    h.setInputCloud(v, 0.02)
    h.build()

    def best(f):
        t = []
        for _ in range(6):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            f()
            torch.cuda.synchronize()
            t.append(time.perf_counter() - t0)
        return min(t)
    lists = best(lambda: h.radiusSearchBatch(*v, 0.02))
    assert best(lambda: api.normal_estimation_rvv(v, h, 10, 0.02)) < 2.9 * lists


# a search that has stopped launches no further rounds
@pytest.mark.parametrize("iters", [3000, 300_000])
def test_ransac_stops_launching(gpu_ctx, restatement, iters):
    from oracle import oracle as O
    from rvpoint_b200 import api
    rng = np.random.default_rng(1)
    p = np.concatenate([rng.uniform(-5, 5, (18_000, 3)) * [1, 1, 0.001],
                        rng.uniform(-5, 5, (2000, 3))]).astype(np.float32)
    c = D.Cloud.from_xyz(p)
    stream = O.libc_rand_stream(3 * iters)
    best, model, _, _, ran = restatement.ransac_plane(c, 0.05, iters, stream)
    assert ran < 1000
    before = gpu_ctx.launches
    got, m = api.ransac_plane_rvv(c, 0.05, iters)
    assert gpu_ctx.launches - before <= 15  # (all rounds of 300,000: 882)
    assert got == best and np.array_equal(bits(m), bits(np.asarray(model, np.float32)))


# a scene of more candidates than a tree takes has the whole device: one of 6000
# is an eighth of the work of 32 of 3000 (and took three times as long)
def test_large_candidate_scene_uses_the_device(gpu_ctx):
    import time
    import torch
    from rvpoint_b200.learned import DeviceBatch, PlaneScorer
    rng = np.random.default_rng(0)
    times = []
    for scenes, m in ((1, 6000), (32, 3000)):
        n = scenes * m
        p = rng.uniform(-5, 5, (n, 3)).astype(np.float32)
        offs = np.arange(scenes + 1, dtype=np.int64) * m
        b = DeviceBatch.from_host(D.Batch(p[:, 0].copy(), p[:, 1].copy(), p[:, 2].copy(), offs))
        s = PlaneScorer(n, scenes, ctx=gpu_ctx)
        cand = torch.arange(n, dtype=torch.int32, device="cuda")
        coffs = torch.from_numpy(offs).cuda()
        t = []
        for _ in range(4):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            s.features(b, 1.0, cand, coffs, among_candidates=True)
            torch.cuda.synchronize()
            t.append(time.perf_counter() - t0)
        times.append(min(t))
        s.close()
    assert times[0] < times[1]


# neighbours at indices from all over clouds that fill two (32,769 points on),
# three and four levels of nodes (1,048,577 on): SOR's means, and normals in
# high precision against eigenvectors over brute-force neighbours
@pytest.mark.parametrize("n", [32_769, 70_001, 1_100_000])
def test_neighbours_through_all_levels(gpu_ctx, n):
    from rvpoint_b200 import api
    k = 9
    c = D.room_cloud(n=n, seed=n)
    p = c.aos()
    at = np.sort(np.random.default_rng(n).choice(n, 120, replace=False))
    idx, d2 = brute_knn(p, p[at], k + 1)
    want = np.zeros(len(at), np.float32)
    for j in range(1, k + 1):
        want += np.sqrt(d2[:, j])
    mean = api.sor_rvv(c, k, 1.0, return_stats=True)[1]
    assert np.array_equal(bits(mean[at]), bits(want / np.float32(k)))
    nrm, _, _ = api.normal_estimation_precise(c, k)
    q = p.astype(np.float64)[idx]
    q -= q.mean(1, keepdims=True)
    w, v = np.linalg.eigh(np.einsum("nki,nkj->nij", q, q))
    clear = w[:, 0] < 0.5 * w[:, 1]  # a normal that is well defined
    assert clear.mean() > 0.8 and (1 - np.abs((nrm[at] * v[:, :, 0]).sum(1))[clear] < 1e-5).all()


# the reference's own normals, point by point, past one level of nodes
def test_normals_past_one_level(gpu_ctx, restatement):
    from rvpoint_b200 import api
    c = D.room_cloud(n=33_000, seed=8)
    got = np.stack(api.normal_estimation_sc(c, 9), 1)
    want = restatement.normals_knn(c, 9)
    # (the rotations branch on the largest entry: a few differ by more)
    assert (np.abs(got - want).max(1) < 1e-4).mean() > 0.995


# SOR's sums go by chunks of 4096 values, runs of 8, after eight segments of 256
# that were not foreseen: sizes about a chunk's edge behind those, with equal
# distances (ties) and a binade left on the way
@pytest.mark.parametrize("n", [2048, 2049, 6143, 6144, 6145, 6152, 10_239, 10_241, 30_001])
def test_sor_statistics_chunks(gpu_ctx, n):
    from rvpoint_b200.api import sor_rvv
    far = 2**20 - int(0.125 * n / 2)
    i = np.arange(n)
    p = np.stack([i % 31, (i // 31) % 37, i // 1147], 1).astype(np.float32) * np.float32(0.1)
    p[0] = [-far, 0, 0]
    c = D.Cloud.from_xyz(p)
    _, mean, _ = sor_rvv(c, 3, 0.5, return_stats=True)
    f = np.float32
    mu = np.add.accumulate(mean)[-1] / f(n)  # in order, in float
    sd = np.sqrt(np.add.accumulate((mean - mu) * (mean - mu))[-1] / f(n))
    target = np.sort(mean)[-2]
    alpha = f((target - mu) / sd)
    for _ in range(64):
        t = mu + alpha * sd
        if t == target:
            break
        alpha = np.nextafter(alpha, f(np.inf) if t < target else f(-np.inf))
    _, _, keep = sor_rvv(c, 3, float(alpha), return_stats=True)
    assert np.array_equal(keep.astype(bool), mean <= mu + alpha * sd)


# frames of fewer than k + 1 points, where the search keeps means only (the
# normals' lists are longer): a mean is over the points there are
@pytest.mark.parametrize("sor_k,normal_k", [(1, 28), (8, 9), (16, 17), (30, 40)])
def test_frames_of_few_points(gpu_ctx, sor_k, normal_k):
    from rvpoint_b200.api import Pipeline
    rng = np.random.default_rng(sor_k)
    sizes = (1, 2, 0, 5, 9, 16, 17, 30, 33, 70, 1)
    n = sum(sizes)
    i = rng.permutation(40 * 40)[:n]
    p = (np.stack([i % 40, i // 40, i % 3], 1) * 0.1 + rng.uniform(0.02, 0.08, (n, 3))).astype(np.float32)
    offs = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    b = D.Batch(p[:, 0].copy(), p[:, 1].copy(), p[:, 2].copy(), offs)
    got = []
    for mode in (0, 3, 1):
        pipe = Pipeline(n, len(sizes), leaf_size=0.1, sor_k=sor_k, normal_k=normal_k, sor_alpha=2.0,
                        ransac_iters=20, queries_per_warp=mode, ctx=gpu_ctx)
        got.append(pipe.run_host(b))
        pipe.close()
    for g in got[:2]:
        for key in g:
            assert np.array_equal(np.asarray(g[key]), np.asarray(got[2][key]), equal_nan=True), key


# lists past the 8192 pairs that a block sorts in shared memory
@pytest.mark.parametrize("n", [8192, 8193, 9729, 20_000])
@pytest.mark.parametrize("same", [False, True])  # all points in one place
def test_very_long_lists(gpu_ctx, restatement, n, same):
    from rvpoint_b200 import api
    rng = np.random.default_rng(n)
    p = np.zeros((n, 3)) if same else rng.normal(0, 0.1, (n, 3))
    p = p.astype(np.float32)
    h = api.SpatialHash()
    h.setInputCloud((p[:, 0], p[:, 1], p[:, 2]), 0.5)
    h.build()
    q = np.concatenate([p[:20], p[:5] + np.float32(0.3)])
    offs, idx, d2 = h.radiusSearchBatch(*q.T, 1.5)
    o2, i2, e2 = brute_radius(p, q, 1.5)
    assert np.array_equal(offs, o2) and np.diff(offs).max() == n
    assert np.array_equal(idx, i2) and np.array_equal(bits(d2), bits(e2))
    if n < 10_000 and not same:
        c = D.Cloud.from_xyz(p)
        got = np.stack(api.normal_estimation_rvv(c, h, 10, 1.5), 1)
        want = np.asarray(restatement.normals_radius(c, 0.5, 1.5))
        assert (np.abs(got - want).max(1) < 1e-4).mean() > 0.995
