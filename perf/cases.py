"""What a program built on this library has it do, as timed cases.

Each case is one pass through the public entry points of ``rvpoint_b200``
(``api``, ``learned``), with inputs made from a seed on the GPU. The clouds
have the shapes of ``rvpoint_b200.datasets`` (indoor room, spinning LiDAR,
shifted precision room, plane scenes), drawn with torch so that new ones are
quick to make. How many neighbours, voxels or kept points come out depends on
the cloud; such outputs go into buffers that the caller keeps, at their
largest size, with zeros past the end. The kinds of pass:

  radius     SpatialHash: set the cloud, build, radiusSearch for every point
  knn        SpatialHash: set the cloud, build, k nearest for every point
  voxel      voxel_grid_downsamp_rvv_v2
  sor        sor_rvv with its mean distances and mask
  normals    SpatialHash build and normal_estimation_rvv
  precise    normal_estimation_precise
  ransac     ransac_plane_rvv
  batch      Pipeline.run_device over many LiDAR frames held on the GPU
  stream     Pipeline.run_host on frames arriving in host memory
  learned    features, scorer and proposal RANSAC over many plane scenes
  gradients  PlaneScorer.gradients: the scorer's forward and backward pass
"""
import math
import random

import numpy as np
import torch

from rvpoint_b200 import api, datasets, learned

DEV = "cuda"


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # one small object cropped from a scan: the smallest call, all latency
        dict(name="radius_crop", kind="radius", cloud="room", n=2_500, cell=0.03, radius=0.03),
        # a whole 64-beam frame, every point's neighbours within 0.5 m (about
        # 25 M pairs): the largest neighbour lists the workloads ask for
        dict(name="radius_lidar", kind="radius", cloud="lidar", beams=64, azimuths=2048,
             cell=0.5, radius=0.5),
        # the same frame, 16 nearest of every point
        dict(name="knn_lidar", kind="knn", cloud="lidar", beams=64, azimuths=2048, cell=0.5,
             k=16),
        # thinning a mapped room of two million points
        dict(name="voxel_map", kind="voxel", cloud="mapped", n=2_000_000, leaf=0.02),
        # outlier removal of an indoor scan (an odd size: a thinned 100k cloud)
        dict(name="sor_room", kind="sor", cloud="room", n=89_343, k=30),
        # radius normals of an indoor scan, read back by the host
        dict(name="normals_room", kind="normals", cloud="room", n=87_477, cell=0.03,
             radius=0.03),
        # precision normals of a large map far from the origin
        dict(name="precise_map", kind="precise", cloud="mapped", n=2_000_000, k=32),
        # the floor of an indoor scan
        dict(name="ransac_room", kind="ransac", cloud="room", n=100_000, iters=1000,
             thresh=0.01),
        # a recorded drive processed in one batch: 256 uneven frames
        dict(name="batch_256", kind="batch", frames=256, mix=2),
        # a live sensor: one frame in, its results back on the host
        dict(name="stream_1", kind="stream", frames=1, mix=6),
        # plane proposals for many scenes at once
        dict(name="learned_512", kind="learned", scenes=512, n=50_000, iters=1000),
        # a training minibatch of the scorer
        dict(name="gradients_32k", kind="gradients", rows=32_768),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("radius", "knn", "voxel", "sor", "normals", "precise", "ransac", "batch",
                       "stream", "learned", "gradients"))
    lidar = dict(cloud="lidar", beams=rng.choice((16, 32, 64)), azimuths=_log(rng, 300, 2048))
    if kind == "radius":
        if rng.random() < 0.5:
            return dict(kind=kind, cell=0.5, radius=rng.choice((0.2, 0.3, 0.5)), **lidar)
        return dict(kind=kind, cloud="room", n=_log(rng, 1_000, 100_000), cell=0.03,
                    radius=rng.choice((0.02, 0.03, 0.05)))
    if kind == "knn":
        if rng.random() < 0.5:
            return dict(kind=kind, cell=0.5, k=rng.choice((8, 16, 20, 32)), **lidar)
        return dict(kind=kind, cloud="room", n=_log(rng, 2_000, 100_000), cell=0.05,
                    k=rng.choice((8, 16, 30)))
    if kind == "voxel":
        return dict(kind=kind, cloud=rng.choice(("room", "mapped")), n=_log(rng, 2_000, 2_000_000),
                    leaf=rng.choice((0.01, 0.02, 0.05, 0.1)))
    if kind == "sor":
        return dict(kind=kind, cloud="room", n=_log(rng, 2_000, 100_000),
                    k=rng.choice((8, 16, 20, 30)))
    if kind == "normals":
        return dict(kind=kind, cloud="room", n=_log(rng, 2_000, 100_000), cell=0.03,
                    radius=rng.choice((0.03, 0.05)))
    if kind == "precise":
        return dict(kind=kind, cloud="mapped", n=_log(rng, 20_000, 2_000_000),
                    k=rng.choice((10, 16, 32)))
    if kind == "ransac":
        return dict(kind=kind, cloud="room", n=_log(rng, 1_000, 1_000_000),
                    iters=rng.choice((200, 1000, 2000)), thresh=rng.choice((0.01, 0.02, 0.05)))
    if kind == "batch":
        return dict(kind=kind, frames=_log(rng, 4, 256), mix=rng.randrange(1000))
    if kind == "stream":
        return dict(kind=kind, frames=rng.randint(1, 8), mix=rng.randrange(1000))
    if kind == "learned":
        return dict(kind=kind, scenes=_log(rng, 16, 512), n=_log(rng, 5_000, 50_000),
                    iters=rng.choice((500, 1000, 2000)))
    return dict(kind=kind, rows=_log(rng, 2_048, 262_144))


# ---------------------------------------------------------------------------
# clouds (the shapes of rvpoint_b200.datasets, drawn on the GPU)
# ---------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _uni(g, *shape):
    return torch.rand(shape, generator=g, device=DEV, dtype=torch.float64)


def _nrm(g, *shape):
    return torch.randn(shape, generator=g, device=DEV, dtype=torch.float64)


def _xyz(p):
    return tuple(p[:, a].float().contiguous() for a in range(3))


def _room(n, seed):
    """Floor and two walls, a sphere, 2% outliers, 2 mm noise."""
    g = _gen(seed)
    n_plane, n_sphere = round(0.70 * n), round(0.28 * n)
    u = _uni(g, n_plane, 2)
    s = _uni(g, n_plane) * 40.0
    zero = torch.zeros_like(s)
    floor = torch.stack([4 * u[:, 0], 4 * u[:, 1], zero], 1)
    wall_x = torch.stack([zero, 4 * u[:, 0], 3 * u[:, 1]], 1)
    wall_y = torch.stack([4 * u[:, 0], zero, 3 * u[:, 1]], 1)
    p = torch.where((s < 16)[:, None], floor, torch.where((s < 28)[:, None], wall_x, wall_y))
    d = _nrm(g, n_sphere, 3)
    ball = 0.5 * d / d.norm(dim=1, keepdim=True) + torch.tensor([2.0, 2.0, 1.0], device=DEV)
    surf = torch.cat([p, ball])
    surf = surf + 0.002 * _nrm(g, surf.shape[0], 3)
    out = _uni(g, n - n_plane - n_sphere, 3) * torch.tensor([4.0, 4.0, 3.0], device=DEV)
    p = torch.cat([surf, out])
    return _xyz(p[torch.randperm(n, generator=g, device=DEV)])


def _mapped(n, seed):
    """Six room planes and 200 spheres and cylinders, 1 mm noise, shifted by
    (1e4, 1e4, 0)."""
    g = _gen(seed)
    size = torch.tensor([8.0, 6.0, 3.0], device=DEV, dtype=torch.float64)
    n_room = int(0.6 * n)
    # planes z, z, y, y, x, x by area
    area = torch.tensor([48.0, 48.0, 24.0, 24.0, 18.0, 18.0], device=DEV, dtype=torch.float64)
    which = torch.bucketize(_uni(g, n_room) * area.sum(), area.cumsum(0)[:-1], right=True)
    room = _uni(g, n_room, 3) * size
    axis = torch.tensor([2, 2, 1, 1, 0, 0], device=DEV)[which]
    on = torch.arange(3, device=DEV)[None, :] == axis[:, None]
    room = torch.where(on, (which % 2)[:, None] * size[None, :], room)
    m = 200
    r = 0.05 + 0.45 * _uni(g, m)
    c = (r[:, None] + 0.1) + _uni(g, m, 3) * (size[None, :] - 2 * r[:, None] - 0.2)
    cyl = _uni(g, m) < 0.5
    h = 0.2 + 1.8 * _uni(g, m)
    c[:, 2] = torch.where(cyl, 0.05 + _uni(g, m) * (2.9 - h), c[:, 2])
    oa = torch.where(cyl, 2 * math.pi * r * h, 4 * math.pi * r * r)
    n_obj = n - n_room
    o = torch.bucketize(_uni(g, n_obj) * oa.sum(), oa.cumsum(0)[:-1], right=True)
    d = _nrm(g, n_obj, 3)
    ball = c[o] + r[o, None] * d / d.norm(dim=1, keepdim=True)
    th = 2 * math.pi * _uni(g, n_obj)
    side = torch.stack([c[o, 0] + r[o] * th.cos(), c[o, 1] + r[o] * th.sin(),
                        c[o, 2] + h[o] * _uni(g, n_obj)], 1)
    p = torch.cat([room, torch.where(cyl[o][:, None], side, ball)])
    p = p + 0.001 * _nrm(g, n, 3)
    p = p[torch.randperm(n, generator=g, device=DEV)]
    return _xyz(p + torch.tensor([1.0e4, 1.0e4, 0.0], device=DEV))


def _sizes(case):
    """Points of each frame: the whole frame of a single-frame case (80% of
    its rays), else log-uniform from 20k to 131,072 rays, at most 80% of a
    64 x 2048 frame's returns."""
    if "mix" not in case:
        return [case["beams"] * case["azimuths"] * 4 // 5]
    rng = random.Random(case["mix"])
    return [min(104_857, int(math.exp(rng.uniform(math.log(20_000), math.log(131_072)))))
            for _ in range(case["frames"])]


def _lidar(case, seed):
    """Spinning-LiDAR frames back to back: (x, y, z, offsets on the host).
    Ground plane and 40 boxes, 2 cm range noise, 5% dropped returns, then a
    random subset of each frame's returns in scan order."""
    ground, far = -1.7, 120.0
    beams, azimuths = case.get("beams", 64), case.get("azimuths", 2048)
    rays, sizes = beams * azimuths, _sizes(case)
    parts = []
    for f0 in range(0, len(sizes), 16):
        want = torch.tensor(sizes[f0:f0 + 16], device=DEV)
        nf = want.numel()
        g = _gen(int(seed) * 1009 + f0)

        def uni(*shape):
            return torch.rand(shape, generator=g, device=DEV)

        # boxes that keep clear of the sensor: the first 40 of 160 tries
        side = 1.0 + 4.0 * uni(nf, 160, 3)
        rad, th = 60.0 * uni(nf, 160).sqrt(), 2 * math.pi * uni(nf, 160)
        ctr = torch.stack([rad * th.cos(), rad * th.sin()], 2)
        near = rad < 3.0 + 0.75 * side[:, :, :2].norm(dim=2)
        first = torch.sort(near.int(), dim=1, stable=True).indices[:, :40, None]
        side, ctr = side.gather(1, first.expand(-1, -1, 3)), ctr.gather(1, first.expand(-1, -1, 2))
        lo = torch.cat([ctr - side[:, :, :2] / 2, torch.full_like(ctr[:, :, :1], ground)], 2)
        hi = torch.cat([ctr + side[:, :, :2] / 2, ground + side[:, :, 2:]], 2)
        el = torch.linspace(math.radians(-25.0), math.radians(3.0), beams, device=DEV)
        az = (torch.arange(azimuths, device=DEV) + uni(nf, 1)) * (2 * math.pi / azimuths)
        dx = (el.cos()[None, :, None] * az.cos()[:, None, :]).reshape(nf, rays)
        dy = (el.cos()[None, :, None] * az.sin()[:, None, :]).reshape(nf, rays)
        dz = el.sin()[None, :, None].expand(nf, beams, azimuths).reshape(nf, rays)
        d = torch.stack([dx, dy, dz])
        t = torch.where(dz < 0, ground / dz, torch.full_like(dz, math.inf))
        inv = 1.0 / torch.where(d == 0, torch.full_like(d, 1e-30), d)
        for b in range(40):
            a0 = lo[:, b].t()[:, :, None] * inv
            a1 = hi[:, b].t()[:, :, None] * inv
            tn, tf = torch.minimum(a0, a1).amax(0), torch.maximum(a0, a1).amin(0)
            t = torch.where((tn <= tf) & (tn > 0) & (tn < t), tn, t)
        keep = torch.isfinite(t) & (t < far) & (uni(nf, rays) >= 0.05)
        key = uni(nf, rays) + 2.0 * (~keep)
        rank = torch.empty(nf, rays, dtype=torch.int64, device=DEV)
        rank.scatter_(1, torch.sort(key, dim=1, stable=True).indices,
                      torch.arange(rays, device=DEV).expand(nf, rays))
        keep = rank < want[:, None]
        # (a frame with fewer returns keeps dropped rays at the last box or
        # the ground: finite ones)
        t = torch.where(torch.isfinite(t), t, torch.full_like(t, far)).clamp(max=far)
        t = t + 0.02 * torch.randn((nf, rays), generator=g, device=DEV)
        parts.append((d * t)[:, keep])
    p = torch.cat(parts, 1)
    offsets = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    return p[0].contiguous(), p[1].contiguous(), p[2].contiguous(), offsets


def _scenes(scenes, n, seed):
    """Plane scenes: 1-6 planes in a 10 m cube, 30-70% uniform outliers, 5 mm
    noise; (x, y, z) of scenes * n points."""
    g, size = _gen(seed), 10.0
    planes = torch.randint(1, 7, (scenes, 1), generator=g, device=DEV)
    outliers = 0.3 + 0.4 * _uni(g, scenes, 1)
    w = -_uni(g, scenes, 6).log() - _uni(g, scenes, 6).log()  # Gamma(2) shares
    w = torch.where(torch.arange(6, device=DEV) < planes, w, torch.zeros_like(w))
    edge = (w / w.sum(1, keepdim=True)).cumsum(1).contiguous()
    nrm = _nrm(g, scenes, 6, 3)
    nrm = (nrm / nrm.norm(dim=2, keepdim=True)).reshape(-1, 3).float()
    anchor = (size * (0.2 + 0.6 * _uni(g, scenes, 6, 3))).reshape(-1, 3).float()
    which = torch.searchsorted(edge, _uni(g, scenes, n), right=True).clamp(max=5)
    which = torch.minimum(which, planes - 1)
    on = (_uni(g, scenes, n) >= outliers).reshape(-1)
    which = (which + 6 * torch.arange(scenes, device=DEV)[:, None]).reshape(-1)
    p = torch.empty((scenes * n, 3), device=DEV)
    p.copy_(size * torch.rand(p.shape, generator=g, device=DEV))
    todo = torch.nonzero(on)[:, 0]
    for _ in range(12):  # a draw whose foot falls outside the cube is redrawn
        if not todo.numel():
            break
        q = size * torch.rand((todo.numel(), 3), generator=g, device=DEV)
        v = nrm[which[todo]]
        q = q - ((q - anchor[which[todo]]) * v).sum(1, keepdim=True) * v
        ok = ((q >= 0) & (q <= size)).all(1)
        at = todo[ok]
        p[at] = q[ok] + 0.005 * torch.randn((at.numel(), 1), generator=g, device=DEV) * v[ok]
        todo = todo[~ok]
    return p[:, 0].contiguous(), p[:, 1].contiguous(), p[:, 2].contiguous()


def _cloud(case, seed):
    if case["cloud"] == "lidar":
        return _lidar(case, seed)[:3]
    return (_room if case["cloud"] == "room" else _mapped)(case["n"], seed)


def _scorer_params(seed):
    """Weights of the shape training gives: small random ones, and a path
    that prefers flat neighbourhoods (low curvature, high planarity)."""
    rng = np.random.Generator(np.random.PCG64(int(seed)))
    w1, w2 = rng.normal(0, 0.2, (64, 8)), rng.normal(0, 0.08, (64, 64))
    b1, b2, w3 = rng.normal(0, 0.1, 64), rng.normal(0, 0.1, 64), rng.normal(0, 0.1, 64)
    w1[0, 3] -= 1.0
    w1[1, 4] += 1.0
    w2[0, 0] += 1.0
    w2[1, 1] += 1.0
    w3[0] += 1.5
    w3[1] += 1.0
    return np.concatenate([w1.ravel(), b1, w2.ravel(), b2, w3, [-0.5]]).astype(np.float32)


# ---------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------
def prepare(case, seed):
    s = dict(case)
    kind = case["kind"]
    if kind in ("radius", "knn", "voxel", "sor", "normals", "precise", "ransac"):
        s["cloud"] = _cloud(case, seed)
        if kind in ("radius", "knn", "normals"):
            s["hash"] = api.SpatialHash()
        if kind == "radius":
            s["hold"] = [torch.zeros(_pairs_held(case), dtype=t, device=DEV)
                         for t in (torch.int32, torch.float32)]
        if kind in ("voxel", "sor"):
            s["hold"] = torch.zeros((case["n"], 3), device=DEV)
    elif kind in ("batch", "stream"):
        x, y, z, offsets = _lidar(case, seed)
        n, nf = int(offsets[-1]), case["frames"]
        if kind == "batch":
            # the settings the autotuner finds for such batches, and tables
            # fitted on a first run, as a program that runs many of them does
            s["args"] = (x, y, z, torch.from_numpy(offsets).to(DEV), nf, n)
            pipe = api.Pipeline(max_points=n, max_frames=nf)
            pipe.run_device(*s["args"])
            pipe.fit_tables()
            pipe.set_tuning(1.0, 128, 3)
            pipe.set_search_radius_factor(0.7)
            s["pipe"] = pipe
        else:
            s["batch"] = datasets.Batch(x.cpu().numpy(), y.cpu().numpy(), z.cpu().numpy(), offsets)
            s["pipe"] = api.Pipeline(max_points=131_072 * nf, max_frames=nf)
        rows = dict(voxel=(n, 3), sor=(n, 3))
        rows.update({"batch": dict(nx=(n,), ny=(n,), nz=(n,))}.get(kind, dict(normals=(n, 3))))
        make = torch.zeros if kind == "batch" else np.zeros
        opts = dict(device=DEV) if kind == "batch" else dict(dtype=np.float32)
        s["hold"] = {k: make(v, **opts) for k, v in rows.items()}
    elif kind == "learned":
        x, y, z = _scenes(case["scenes"], case["n"], seed)
        offsets = np.arange(case["scenes"] + 1, dtype=np.int64) * case["n"]
        b = learned.DeviceBatch(x, y, z, torch.from_numpy(offsets).to(DEV), offsets)
        scorer = learned.PlaneScorer(b.n, b.n_frames)
        lr = learned.LearnedRansac(scorer, cell=2.0)
        cand, cand_offsets = lr.prepare(b)
        scorer.set_params(_scorer_params(seed))
        feat = learned.proposal_features(scorer, b, cand, cand_offsets, lr.cell, lr.scope)
        scorer.set_norm(feat.mean(0).cpu().numpy(), feat.std(0).clamp_min(1e-6).cpu().numpy())
        s.update(b=b, lr=lr, cand=cand, cand_offsets=cand_offsets)
    else:
        s["feat"], s["labels"] = _rows(case, seed)
        scorer = learned.PlaneScorer(1024, 1)
        scorer.set_params(_scorer_params(seed))
        s["scorer"] = scorer
    return s


def _rows(case, seed):
    """Feature rows of flat and scattered neighbourhoods, normalised, and
    their labels."""
    g = _gen(seed)
    feat = torch.randn((case["rows"], 8), generator=g, device=DEV)
    logit = 2.0 * feat[:, 4] - 2.0 * feat[:, 3] + torch.randn(case["rows"], generator=g, device=DEV)
    return feat, (logit > 1.0).float()


def _pairs(case):
    """About how many neighbour pairs a radius case has."""
    n = _points(case)
    if case["cloud"] == "lidar":
        return int(n + 2.2e-3 * n * n * (case["radius"] / 0.5) ** 2)
    return int(n + 1.2e-4 * n * n * (case["radius"] / 0.03) ** 2)


def _pairs_held(case):
    return 2 * _pairs(case) + 4096


def _points(case):
    return case["n"] if "n" in case else sum(_sizes(case))


def _keep(hold, v):
    """v in the caller's buffer, zeros past its end."""
    hold[:len(v)] = v
    hold[len(v):] = 0
    return hold


class _Device:
    """A device buffer of the pipeline's, as torch reads it."""

    def __init__(self, ptr, shape, dtype):
        self.__cuda_array_interface__ = dict(data=(ptr, False), shape=shape, typestr=dtype,
                                             strides=None, version=3)


def run(s):
    kind = s["kind"]
    if kind == "radius":
        h = s["hash"]
        h.setInputCloud(s["cloud"], s["cell"])
        h.build()
        offsets, idx, d2 = h.radiusSearchBatch(*s["cloud"], s["radius"])
        return offsets, _keep(s["hold"][0], idx), _keep(s["hold"][1], d2)
    if kind == "knn":
        h = s["hash"]
        h.setInputCloud(s["cloud"], s["cell"])
        h.build()
        return h.knn(*s["cloud"], s["k"])
    if kind == "voxel":
        return _keep(s["hold"], api.voxel_grid_downsamp_rvv_v2(s["cloud"], s["leaf"]))
    if kind == "sor":
        out, mean, mask = api.sor_rvv(s["cloud"], s["k"], 1.0, return_stats=True)
        return _keep(s["hold"], out), mean, mask
    if kind == "normals":
        h = s["hash"]
        h.setInputCloud(s["cloud"], s["cell"])
        h.build()
        return api.normal_estimation_rvv(s["cloud"], h, 10, s["radius"])
    if kind == "precise":
        return api.normal_estimation_precise(s["cloud"], s["k"])
    if kind == "ransac":
        return api.ransac_plane_rvv(s["cloud"], s["thresh"], s["iters"])
    if kind == "batch":
        pipe, nf = s["pipe"], s["frames"]
        pipe.run_device(*s["args"])
        vo, so = pipe.frame_offsets()
        o, nv, ns = pipe.outputs(), int(vo[-1]), int(so[-1])

        def view(ptr, shape, dtype="<f4"):
            return torch.as_tensor(_Device(ptr, shape, dtype), device=DEV)

        out = dict(voxel=view(o.voxel_aos, (nv, 3)), sor=view(o.sor_aos, (ns, 3)),
                   nx=view(o.nx, (ns,)), ny=view(o.ny, (ns,)), nz=view(o.nz, (ns,)))
        return dict({k: _keep(s["hold"][k], v) for k, v in out.items()}, voxel_offsets=vo,
                    sor_offsets=so, model=view(o.ransac_model, (nf, 4)).clone(),
                    count=view(o.ransac_count, (nf,), "<i4").clone())
    if kind == "stream":
        out = s["pipe"].run_host(s["batch"])
        return {k: _keep(s["hold"][k], v) if k in s["hold"] else v for k, v in out.items()}
    if kind == "learned":
        lr, b, cand, offs = s["lr"], s["b"], s["cand"], s["cand_offsets"]
        feat = learned.proposal_features(lr.scorer, b, cand, offs, lr.cell, lr.scope)
        logits = lr.scorer.forward(feat)
        models, best, drawn = lr.ransac(b, cand, offs, logits, s["iters"], 0.02)
        return feat, logits, models, best, drawn
    return s["scorer"].gradients(s["feat"], s["labels"])


# ---------------------------------------------------------------------------
# the work of a pass
# ---------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    n = 0 if kind == "gradients" else _points(case)
    if kind == "radius":
        pairs = _pairs(case)
        return dict(bytes=24 * n + 8 * n + 8 * pairs, flops=8 * pairs)
    if kind == "knn":
        return dict(bytes=24 * n + n * (8 * case["k"] + 4), flops=8 * n * case["k"])
    if kind == "voxel":
        return dict(bytes=12 * n + 12 * min(n, 3.0e2 / case["leaf"] ** 2), flops=6 * n)
    if kind == "sor":
        return dict(bytes=12 * n + 17 * n, flops=9 * n * case["k"])
    if kind == "normals":
        m = 1 + 1.0e-4 * n * (case["radius"] / 0.03) ** 2
        return dict(bytes=24 * n, flops=n * (20 * m + 200))
    if kind == "precise":
        return dict(bytes=12 * n + 17 * n, flops=n * (80 * case["k"] + 600))
    if kind == "ransac":
        return dict(bytes=12 * n, flops=9 * n * min(case["iters"], 300))
    if kind in ("batch", "stream"):
        # in, voxels (0.74 n) and kept points (0.67 n) out, normals
        return dict(bytes=12 * n + 8.9 * n + 16 * n, flops=n * (2 * 17 * 20 + 300))
    if kind == "learned":
        rows = case["scenes"] * min(1024, case["n"])
        # features of the candidates, the scorer, and 32 hypotheses of each
        # 512 drawn counted exactly over all points
        rounds = learned.preemptive_rounds(case["iters"], 512)
        return dict(bytes=12 * n * case["scenes"] + 36 * rows,
                    flops=rows * (2 * 4672 + 400) + 9 * 32 * rounds * n * case["scenes"])
    return dict(bytes=36 * case["rows"] + 4 * 4801, flops=6 * 4672 * case["rows"])


# ---------------------------------------------------------------------------
# the same in 64 bits, with plain torch
# ---------------------------------------------------------------------------
def _d2(q, p):
    """Squared distances of every pair, each operation rounded by itself (in
    float32 they decide membership and order)."""
    d = [(p[a][None, :] - q[a][:, None]).square_() for a in range(3)]
    return d[0].add_(d[1]).add_(d[2])


def _fit(v, rows):
    return torch.cat([v, v.new_zeros((rows - v.shape[0],) + tuple(v.shape[1:]))])


def _radius_lists(p, radius):
    """(counts, indices, d2 in float64) of every point's neighbours, in
    (d2, index) order."""
    n = p[0].numel()
    r2 = torch.tensor(radius, dtype=torch.float32, device=DEV).square()
    step = max(64, min(4096, 400_000_000 // max(n, 1)))
    counts, idx, dist = [], [], []
    for a in range(0, n, step):
        d2 = _d2([v[a:a + step] for v in p], p)
        row, col = torch.nonzero(d2 <= r2, as_tuple=True)
        v = d2[row, col]
        o = torch.argsort(v, stable=True)
        o = o[torch.argsort(row[o], stable=True)]
        row, col = row[o], col[o]
        counts.append(torch.bincount(row, minlength=d2.shape[0]))
        idx.append(col)
        dist.append(sum((c[col].double() - c[a:a + step][row].double()).square() for c in p))
    return torch.cat(counts), torch.cat(idx), torch.cat(dist)


def _nearest(p, k):
    """(indices, d2 in float64) of the k nearest of every point, n x k."""
    n = p[0].numel()
    step = max(64, min(4096, 200_000_000 // max(n, 1)))
    q = [v.double() for v in p]
    idx, dist = [], []
    for a in range(0, n, step):
        d2 = _d2([v[a:a + step] for v in q], q)
        v, i = torch.topk(d2, k, dim=1, largest=False, sorted=True)
        idx.append(i)
        dist.append(v)
    return torch.cat(idx), torch.cat(dist)


def _eigh(cov):
    got = [torch.linalg.eigh(c) for c in cov.reshape(-1, 3, 3).split(16_384)]
    return (torch.cat([g[0] for g in got]).reshape(cov.shape[:-1]),
            torch.cat([g[1] for g in got]).reshape(cov.shape))


def _smallest(cov, p):
    """Unit eigenvectors of the smallest eigenvalue, turned to the origin."""
    lam, vec = _eigh(cov)
    return lam, _turned(vec[:, :, 0], p)


def _turned(nrm, p):
    return torch.where(((nrm * -p).sum(1) < 0)[:, None], -nrm, nrm)


def _four_rotations(cov, p):
    """The normal as normal_estimation defines it: four rotations, each on
    the largest off-diagonal entry, that update the two diagonal entries and
    the vectors only; then the vector of the smallest diagonal entry."""
    n = cov.shape[0]
    diag = [cov[:, a, a].clone() for a in range(3)]
    off = {pq: cov[:, pq[0], pq[1]].clone() for pq in ((0, 1), (0, 2), (1, 2))}
    vec = [torch.eye(3, dtype=cov.dtype, device=DEV)[a].expand(n, 3) for a in range(3)]
    for _ in range(4):
        size = torch.stack([off[pq].abs() for pq in off])
        at = torch.where(size[1] > size[0], 1, 0)
        at = torch.where(size[2] > torch.maximum(size[0], size[1]), 2, at)
        for k, (a, b) in enumerate(list(off)):
            m, v = at == k, off[(a, b)]
            phi = 0.5 * torch.atan2(2 * v, diag[a] - diag[b])
            c, s = phi.cos(), phi.sin()
            da = c * c * diag[a] - 2 * s * c * v + s * s * diag[b]
            db = s * s * diag[a] + 2 * s * c * v + c * c * diag[b]
            va = c[:, None] * vec[a] - s[:, None] * vec[b]
            vb = s[:, None] * vec[a] + c[:, None] * vec[b]
            diag[a], diag[b] = torch.where(m, da, diag[a]), torch.where(m, db, diag[b])
            vec[a] = torch.where(m[:, None], va, vec[a])
            vec[b] = torch.where(m[:, None], vb, vec[b])
            off[(a, b)] = torch.where(m, torch.zeros_like(v), v)
    least = torch.stack(diag).argmin(0)
    nrm = torch.stack(vec, 1)[torch.arange(n, device=DEV), least]
    return _turned(nrm, p)


def _forward64(w, x):
    w1, b1, w2, b2, w3, b3 = w
    h = torch.relu(x @ w1.t() + b1)
    h = torch.relu(h @ w2.t() + b2)
    return h @ w3 + b3


def _weights64(seed):
    w = torch.from_numpy(_scorer_params(seed)).to(DEV).bfloat16().double()
    at, out = 0, []
    for shape in ((64, 8), (64,), (64, 64), (64,), (64,), (1,)):
        size = math.prod(shape)
        out.append(w[at:at + size].reshape(shape).clone().requires_grad_())
        at += size
    return out


def _voxels(p, frame, leaf):
    """Centroids in (frame, ix, iy, iz) order."""
    inv = torch.tensor(1.0, device=DEV) / torch.tensor(leaf, dtype=torch.float32, device=DEV)
    cell = [torch.floor(v * inv).long() for v in p]
    key = frame
    for c in cell:
        c = c - c.min()
        key = key * (int(c.max()) + 1) + c
    _, inverse, count = torch.unique(key, return_inverse=True, return_counts=True)
    out = torch.zeros((count.numel(), 3), dtype=torch.float64, device=DEV)
    out.index_add_(0, inverse, torch.stack(p, 1).double())
    return out / count[:, None]


def exact(case, seed):
    kind = case["kind"]
    if kind == "gradients":
        feat, labels = _rows(case, seed)
        w = _weights64(seed)
        loss = torch.nn.functional.binary_cross_entropy_with_logits(
            _forward64(w, feat.double()), labels.double())
        loss.backward()
        return float(loss.detach()), torch.cat([v.grad.reshape(-1) for v in w])
    if kind in ("batch", "stream"):
        x, y, z, offsets = _lidar(case, seed)
        frame = torch.repeat_interleave(torch.arange(case["frames"], device=DEV),
                                        torch.from_numpy(np.diff(offsets)).to(DEV))
        return dict(voxel=_fit(_voxels((x, y, z), frame, 0.1), x.numel()))
    if kind == "learned":
        return _learned64(case, seed)
    p = _cloud(case, seed)
    n = p[0].numel()
    if kind == "voxel":
        frame = torch.zeros(n, dtype=torch.int64, device=DEV)
        return _fit(_voxels(p, frame, case["leaf"]), n)
    if kind == "ransac" or n > 150_000:
        return None
    if kind == "radius":
        counts, idx, d2 = _radius_lists(p, case["radius"])
        offs = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
        offs[1:] = counts.cumsum(0)
        held = _pairs_held(case)
        return offs, _fit(idx.int(), held), _fit(d2, held)
    if kind == "knn":
        return None, _nearest(p, case["k"])[1]
    if kind == "sor":
        d2 = _nearest(p, case["k"] + 1)[1]
        return None, d2[:, 1:].sqrt().mean(1)
    xyz = torch.stack(p, 1).double()
    if kind == "normals":
        counts, idx, _ = _radius_lists(p, case["radius"])
        row = torch.repeat_interleave(torch.arange(n, device=DEV), counts)
        mean = torch.zeros((n, 3), dtype=torch.float64, device=DEV).index_add_(0, row, xyz[idx])
        mean /= counts[:, None]
        d = xyz[idx] - mean[row]
        cov = torch.zeros((n, 3, 3), dtype=torch.float64, device=DEV)
        cov.index_add_(0, row, d[:, :, None] * d[:, None, :])
        nrm = torch.where((counts < 3)[:, None], torch.zeros_like(xyz), _four_rotations(cov, xyz))
        return nrm[:, 0], nrm[:, 1], nrm[:, 2]
    # precise
    d = xyz[_nearest(p, case["k"] + 1)[0]]
    d = d - d.mean(1, keepdim=True)
    lam, nrm = _smallest(d.transpose(1, 2) @ d, xyz)
    return nrm, lam[:, 2] / lam[:, 0], None


def _learned64(case, seed):
    x, y, z = _scenes(case["scenes"], case["n"], seed)
    offsets = np.arange(case["scenes"] + 1, dtype=np.int64) * case["n"]
    cand, _ = learned.candidates(offsets, 1024, 11)
    p = torch.stack([x, y, z], 1).double()[torch.from_numpy(cand.astype(np.int64)).to(DEV)]
    p = p.reshape(case["scenes"], -1, 3)
    out = []
    for part in p.split(32):
        d2 = (part[:, :, None, :] - part[:, None, :, :]).square().sum(3)
        v, i = torch.topk(d2, 17, dim=2, largest=False, sorted=True)
        at = torch.arange(part.shape[0], device=DEV)[:, None, None]
        d = part[at, i] - part[:, :, None, :]
        c = d.mean(2)
        e = d - c[:, :, None, :]
        lam, vec = _eigh(e.transpose(2, 3) @ e)
        nrm, l0 = vec[..., 0], lam[..., 0].clamp_min(0)
        r = v[:, :, 16].sqrt() + 1e-6
        f = [nrm.abs(), (l0 / (l0 + lam[..., 1] + lam[..., 2]))[..., None],
             ((lam[..., 1] - l0) / lam[..., 2])[..., None], r.log()[..., None],
             ((nrm * c).sum(3 - 1).abs() / r)[..., None], (c.norm(dim=2) / r)[..., None]]
        out.append(torch.cat(f, 2).reshape(-1, 8))
    feat = torch.cat(out)
    x = (feat - feat.mean(0)) / feat.std(0).clamp_min(1e-6)
    return feat, _forward64(_weights64(seed), x).detach()
