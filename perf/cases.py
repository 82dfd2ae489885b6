"""Workloads of the nearest-neighbour library, timed through its Python entry points.

Every case is one call, or one short sequence of calls, as a program that uses
the library makes it: searches on a prebuilt kd-tree (from host arrays as with
the reference's Python binding, or on CUDA tensors), a kd-tree built on a fresh
scan and searched once, batches of clouds built and searched together, the
brute-force search and the learned-radius search. Clouds are spinning-lidar
scans of a ground plane with boxes, uniform points, or Gaussian clusters.

A case's keys:
  kind        search | build_search | batch | brute | learned
  memory      device (CUDA tensors), host (numpy arrays), pinned (page-locked
              arrays with the results written into page-locked arrays)
  cloud       lidar | uniform | clusters (batch: Gaussian blobs)
  dtype, dim, points, queries, k, epsilon, radius (0: unbounded),
  radii       per-query radii instead of one
  touch       the object counts the visited points
  queries_are cloud (the cloud itself), moved (the cloud after a small motion)
              or fresh (drawn like the cloud)
"""
from __future__ import annotations

import math

import numpy as np
import torch

import libnabo_gb300 as nabo
from libnabo_gb300.synthetic import log_uniform_sizes

DEVICE = "cuda"


def _search(name, **kw):
    case = dict(name=name, kind="search", memory="device", cloud="lidar", dtype="float32", dim=3, points=83000,
                queries=83000, k=10, epsilon=0.0, radius=0.0, radii=False, touch=False, queries_are="moved")
    case.update(kw)
    return case


def _batch(name, **kw):
    case = dict(name=name, kind="batch", clouds=512, smallest=2000, largest=200000, dtype="float32", dim=3,
                sizes_seed=1236, k_choices="1,5,16", epsilon=0.0, bucket=16, threads=128, split=1, levels=24)
    case.update(kw)
    return case


def listed():
    return [
        # a handful of keypoints looked up in a large map from host arrays:
        # the smallest call, all latency
        _search("keypoints_host", memory="host", points=1149207, queries=16, k=10, radius=1.0),
        # the reference binding's ordinary use: 10 k double points and queries
        # as numpy arrays, k = 5
        _search("small_host_f64", memory="host", cloud="uniform", dtype="float64", points=10000, queries=10000, k=5,
                queries_are="fresh"),
        # scan matching: the closest point of every point of a 64 x 1800-ray
        # scan in the previous scan, within 1 m
        _search("matching_k1", points=83000, queries=83000, k=1, radius=1.0),
        # surface normals: a kd-tree on each new scan, then every point's 10
        # nearest other points
        _search("normals_frame", kind="build_search", points=83000, queries=83000, k=10, queries_are="cloud"),
        # a new 1.15 M point map: build it, then match one scan against it
        _search("map_build", kind="build_search", points=1149207, queries=83000, k=1, radius=1.0),
        # the headline workload: a 64-beam scan of 1.15 M points against the
        # scan before it, k = 10 within 1 m
        _search("scan_k10", points=1149207, queries=1149207, k=10, radius=1.0),
        # the same from and to page-locked host memory
        _search("scan_k10_pinned", memory="pinned", points=1149207, queries=1149207, k=10, radius=1.0),
        # the same with the learned search radius, its network trained on
        # another frame
        _search("scan_k10_learned", kind="learned", points=1149207, queries=1149207, k=10, radius=1.0),
        # density and outlier statistics: many neighbours (an odd number of
        # queries)
        _search("density_k50", points=83000, queries=82999, k=50, queries_are="moved"),
        # descriptor matching: 8-D double clusters, k = 32
        _search("descriptors_f64_k32", cloud="clusters", dtype="float64", dim=8, points=200000, queries=50000, k=32,
                queries_are="fresh"),
        # many uneven clouds built and searched in one captured launch, k of
        # 1, 5 or 16 per cloud, with the autotuner's parameters
        _batch("batch_512"),
        # the brute-force search, 100 k points and queries
        _search("brute_100k_k5", kind="brute", cloud="uniform", points=100000, queries=100000, k=5,
                queries_are="fresh"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(["lookup", "device", "device", "build", "scan", "wide", "descriptors", "batch", "brute",
                         "learned"])
    radius = rng.choice([0.0, 0.5, 1.0])
    if family == "lookup":
        f64 = rng.random() < 0.4
        return _search(None, memory="host", cloud=rng.choice(["lidar", "uniform"]),
                       dtype="float64" if f64 else "float32", points=_log_int(rng, 5000, 1149207),
                       queries=_log_int(rng, 1, 20000), k=rng.choice([1, 3, 5, 8, 10, 16]), queries_are="fresh")
    if family == "device":
        f64 = rng.random() < 0.3
        cloud = rng.choice(["lidar", "uniform"])
        dim = 3 if cloud == "lidar" else rng.choice([2, 3, 3, 4])
        return _search(None, cloud=cloud, dtype="float64" if f64 else "float32", dim=dim,
                       points=_log_int(rng, 10000, 600000), queries=_log_int(rng, 5000, 300000),
                       k=rng.choice([1, 2, 4, 5, 7, 10, 12, 16]), epsilon=rng.choice([0.0, 0.0, 0.1, 0.5]),
                       radius=radius if cloud == "lidar" else 0.0, radii=cloud == "lidar" and rng.random() < 0.3,
                       touch=rng.random() < 0.25, queries_are="fresh")
    if family == "build":
        return _search(None, kind="build_search", cloud=rng.choice(["lidar", "uniform"]),
                       points=_log_int(rng, 10000, 1100000), queries=_log_int(rng, 10000, 200000),
                       k=rng.choice([1, 5, 10, 16]), queries_are="fresh")
    if family == "scan":
        return _search(None, memory=rng.choice(["device", "pinned"]), cloud=rng.choice(["lidar", "uniform"]),
                       points=_log_int(rng, 200000, 1149207), queries=_log_int(rng, 262144, 1149207),
                       k=rng.choice([1, 5, 8, 10, 16]), epsilon=rng.choice([0.0, 0.0, 0.5]), queries_are="fresh")
    if family == "wide":
        return _search(None, points=_log_int(rng, 20000, 300000), queries=_log_int(rng, 10000, 100000),
                       k=rng.choice([33, 50, 64, 100]), queries_are="fresh")
    if family == "descriptors":
        f64 = rng.random() < 0.5
        return _search(None, cloud="clusters", dtype="float64" if f64 else "float32",
                       dim=rng.choice([5, 6, 8, 8, 12, 16]), points=_log_int(rng, 10000, 200000),
                       queries=_log_int(rng, 3000, 30000), k=rng.choice([5, 10, 20, 32]),
                       epsilon=rng.choice([0.0, 0.0, 0.5]), queries_are="fresh")
    if family == "batch":
        return _batch(None, clouds=_log_int(rng, 8, 200), smallest=_log_int(rng, 500, 3000),
                      largest=_log_int(rng, 20000, 150000), sizes_seed=rng.randrange(1 << 20),
                      k_choices=rng.choice(["1,5,16", "10", "1,8", "5,10"]), bucket=rng.choice([8, 16]),
                      split=rng.choice([0, 1, 1]), levels=40)
    if family == "brute":
        dim = rng.choice([2, 3, 3, 4, 8])
        points = _log_int(rng, 5000, 100000)
        return _search(None, kind="brute", cloud="uniform", dim=dim, points=points,
                       queries=min(_log_int(rng, 3000, 100000), int(2e10 / points / dim)),
                       k=rng.choice([1, 5, 10, 16]), queries_are="fresh")
    return _search(None, kind="learned", points=_log_int(rng, 300000, 1100000),
                   queries=_log_int(rng, 262144, 1100000), k=rng.choice([5, 10]), radius=1.0, queries_are="fresh")


# ---------------------------------------------------------------- inputs

def _gen(seed):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(int(seed))
    return g


def _uniform(lo, hi, shape, g):
    return lo + (hi - lo) * torch.rand(shape, generator=g, device=DEVICE, dtype=torch.float64)


def _normal(shape, g):
    return torch.randn(shape, generator=g, device=DEVICE, dtype=torch.float64)


def _lidar(points, scene_seed, noise_seed, beams=64, ground=-1.7, boxes=20, noise=0.02, max_range=120.0):
    """`points` returns, in scan order, of a 64-beam lidar (elevations -25 to
    15 degrees) over a ground plane with 20 boxes of 1-10 m within 60 m."""
    rng = np.random.default_rng(scene_seed)
    lo, hi = np.empty((boxes, 3)), np.empty((boxes, 3))
    for b in range(boxes):
        ext = rng.uniform(1.0, 10.0, 3)
        c = rng.uniform(-60.0, 60.0, 2)
        while np.hypot(*c) <= 3.0 + 0.5 * np.hypot(ext[0], ext[1]):
            c = rng.uniform(-60.0, 60.0, 2)
        lo[b] = [c[0] - ext[0] / 2, c[1] - ext[1] / 2, ground]
        hi[b] = [c[0] + ext[0] / 2, c[1] + ext[1] / 2, ground + ext[2]]
    azimuths = int(math.ceil(points / beams / 0.58))  # at least 0.6 of the beams hit the ground
    elev = torch.deg2rad(torch.linspace(-25.0, 15.0, beams, device=DEVICE, dtype=torch.float64))
    az = torch.arange(azimuths, device=DEVICE, dtype=torch.float64) * (2.0 * math.pi / azimuths)
    dx = (torch.cos(az)[:, None] * torch.cos(elev)[None, :]).reshape(-1)
    dy = (torch.sin(az)[:, None] * torch.cos(elev)[None, :]).reshape(-1)
    dz = torch.sin(elev)[None, :].expand(azimuths, beams).reshape(-1)
    t = torch.where(dz < 0, ground / dz, torch.full_like(dz, math.inf))
    inv = (1.0 / dx, 1.0 / dy, 1.0 / dz)
    for b in range(boxes):
        near = torch.full_like(t, -math.inf)
        far = torch.full_like(t, math.inf)
        for d in range(3):
            t1, t2 = lo[b, d] * inv[d], hi[b, d] * inv[d]
            near = torch.fmax(near, torch.fmin(t1, t2))
            far = torch.fmin(far, torch.fmax(t1, t2))
        t = torch.where((far >= near) & (near > 0) & (near < t), near, t)
    hit = torch.nonzero(t < max_range).reshape(-1)
    hit = hit[torch.linspace(0, hit.numel() - 1, points, device=DEVICE, dtype=torch.float64).round().long()]
    r = t[hit] + noise * _normal((points,), _gen(noise_seed))
    return torch.stack([dx[hit] * r, dy[hit] * r, dz[hit] * r], dim=1)


def _moved(cloud, seed, angle_deg=2.0, shift=0.1):
    """The cloud after a rotation by 2 degrees and a 0.1 m translation."""
    rng = np.random.default_rng(seed + 1000)
    axis = rng.normal(size=3)
    axis /= np.linalg.norm(axis)
    th = math.radians(angle_deg)
    k = np.array([[0, -axis[2], axis[1]], [axis[2], 0, -axis[0]], [-axis[1], axis[0], 0]])
    rot = np.eye(3) + math.sin(th) * k + (1 - math.cos(th)) * (k @ k)
    t = rng.normal(size=3)
    t *= shift / np.linalg.norm(t)
    return cloud @ torch.from_numpy(rot.T.copy()).to(DEVICE) + torch.from_numpy(t).to(DEVICE)


def _clusters(n, dim, mixture_seed, seed, count=32):
    """Isotropic Gaussian clusters with log-uniform sigma in [0.01, 1]."""
    rng = np.random.default_rng(mixture_seed)
    centres = torch.from_numpy(rng.uniform(-5.0, 5.0, (count, dim))).to(DEVICE)
    sigma = torch.from_numpy(np.exp(rng.uniform(math.log(0.01), 0.0, count))).to(DEVICE)
    g = _gen(seed)
    label = torch.randint(count, (n,), generator=g, device=DEVICE)
    return centres[label] + _normal((n, dim), g) * sigma[label][:, None]


def _pick(x, count):
    """`count` rows spread evenly over x, in order."""
    if count == x.shape[0]:
        return x
    return x[torch.linspace(0, x.shape[0] - 1, count, device=DEVICE, dtype=torch.float64).round().long()]


def _inputs(case, seed):
    """(cloud, queries, radii) as CUDA tensors of the case's type."""
    dtype = getattr(torch, case["dtype"])
    n, nq, dim = case["points"], case["queries"], case["dim"]
    if case["cloud"] == "lidar":
        cloud = _lidar(n, seed, seed + 1)
        if case["queries_are"] == "cloud":
            queries = _pick(cloud, nq)
        elif case["queries_are"] == "moved":
            queries = _moved(_pick(cloud, nq), seed)
        else:  # another frame of the scene
            queries = _moved(_lidar(nq, seed, seed + 2), seed)
    elif case["cloud"] == "uniform":
        cloud = _uniform(0.0, 1.0, (n, dim), _gen(seed))
        queries = _pick(cloud, nq) if case["queries_are"] == "cloud" else _uniform(0.0, 1.0, (nq, dim), _gen(seed + 1))
    else:
        cloud = _clusters(n, dim, seed, seed)
        queries = _clusters(nq, dim, seed, seed + 1)
    radii = None
    if case["radii"]:
        radii = _uniform(0.2, 1.5, (nq,), _gen(seed + 3)).to(dtype)
    return cloud.to(dtype), queries.to(dtype), radii


def _batch_plan(case):
    sizes = log_uniform_sizes(case["clouds"], case["smallest"], case["largest"], case["sizes_seed"])
    choices = np.array([int(x) for x in case["k_choices"].split(",")], np.int32)
    ks = np.random.default_rng(case["sizes_seed"] + 1).choice(choices, case["clouds"])
    return sizes, ks


def _batch_inputs(case, seed, blobs=8):
    """Clouds of 8 anisotropic Gaussian blobs each (sigma 0.05-2 per axis), back
    to back, and the same clouds with 0.01 of noise as the queries."""
    sizes, _ = _batch_plan(case)
    dtype = getattr(torch, case["dtype"])
    total, dim = int(sizes.sum()), case["dim"]
    g = _gen(seed)
    count = case["clouds"] * blobs
    centres = _uniform(-10.0, 10.0, (count, dim), g)
    sigma = _uniform(0.05, 2.0, (count, dim), g)
    axes = torch.linalg.qr(_normal((count, dim, dim), g))[0]
    frames = (sigma[:, :, None] * axes.transpose(1, 2)).to(torch.float32)  # row i: sigma_i times axis i
    cloud_id = torch.repeat_interleave(torch.arange(case["clouds"], device=DEVICE), torch.from_numpy(sizes).to(DEVICE))
    label = cloud_id * blobs + torch.randint(blobs, (total,), generator=g, device=DEVICE)
    z = torch.randn((total, dim), generator=g, device=DEVICE)
    clouds = torch.zeros((total, dim), device=DEVICE)
    for i in range(dim):
        clouds += z[:, i:i + 1] * frames[label, i]
    clouds = (clouds + centres.to(torch.float32)[label]).to(dtype)
    queries = clouds + 0.01 * torch.randn((total, dim), generator=g, device=DEVICE).to(dtype)
    return clouds, queries


# ---------------------------------------------------------------- the cases

def _options(case):
    return dict(epsilon=case["epsilon"], maxRadius=case["radius"] if case["radius"] > 0 else np.inf)


def prepare(case, seed):
    if case["kind"] == "batch":
        clouds, queries = _batch_inputs(case, seed)
        sizes, ks = _batch_plan(case)
        batch = nabo.BatchSearch(sizes, dim=case["dim"], dtype=np.dtype(case["dtype"]), bucketSize=case["bucket"],
                                 threadsPerBlock=case["threads"], maxLevels=case["levels"], splitRule=case["split"])
        batch.set_queries(sizes, ks)
        entries = batch.result_entries
        out = (torch.empty(entries, dtype=torch.int32, device=DEVICE),
               torch.empty(entries, dtype=clouds.dtype, device=DEVICE))
        return dict(case=case, batch=batch, clouds=clouds, queries=queries, out=out)
    cloud, queries, radii = _inputs(case, seed)
    state = dict(case=case, queries=queries, radii=radii)
    flags = nabo.TOUCH_STATISTICS if case["touch"] else 0
    if case["kind"] == "build_search":
        state["cloud"] = cloud
        return state
    kind = nabo.SearchType.BRUTE_FORCE_CUDA if case["kind"] == "brute" else nabo.SearchType.KDTREE_CUDA
    search = nabo.NearestNeighbourSearch(cloud, kind, creationOptionFlags=flags)
    state["search"] = search
    if case["kind"] == "learned":
        train = _pick(_moved(_lidar(case["points"], seed, seed + 7), seed), min(100000, case["points"]))
        state["model"] = nabo.RadiusModel(search, train.to(cloud.dtype), case["k"], maxRadius=case["radius"])
    if case["memory"] == "host":
        state["queries"] = queries.cpu().numpy()
        state["radii"] = None if radii is None else radii.cpu().numpy()
    elif case["memory"] == "pinned":
        shape = (case["queries"], case["k"])
        state["queries"] = queries.cpu().pin_memory().numpy()
        state["out"] = (torch.empty(shape, dtype=torch.int32).pin_memory().numpy(),
                        torch.empty(shape, dtype=cloud.dtype).pin_memory().numpy())
    elif case["touch"]:
        state["touched"] = torch.zeros(1, dtype=torch.int64, device=DEVICE)
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        return state["batch"].run(state["clouds"], state["queries"], epsilon=case["epsilon"], out=state["out"])
    opts = _options(case)
    if case["kind"] == "build_search":
        search = nabo.NearestNeighbourSearch(state["cloud"], nabo.SearchType.KDTREE_CUDA)
        idx, d2 = search.knn(state["queries"], case["k"], **opts)
        return dict(indices=idx, dists2=d2, nodes=search.nodeCount, height=search.height, low=search.minBound,
                    high=search.maxBound)
    if case["kind"] == "learned":
        return state["model"].knn(state["queries"], case["k"], **opts)
    search = state["search"]
    if case["memory"] == "pinned":
        return search.knn(state["queries"], case["k"], out=state["out"], **opts)
    if case["memory"] == "device" and case["touch"]:
        state["touched"].zero_()
        idx, d2 = search.knn_device(state["queries"], case["k"], maxRadii=state["radii"], touched=state["touched"],
                                    **opts)
        return idx, d2, state["touched"]
    return search.knn(state["queries"], case["k"], maxRadii=state["radii"], **opts)


def work(case):
    """Each input (points, queries, radii) read once and each result written
    once. Flops: a brute-force search's distances, 3 per coordinate of each
    pair; else those of the neighbours returned."""
    scalar = 4 if case["dtype"] == "float32" else 8
    if case["kind"] == "batch":
        sizes, ks = _batch_plan(case)
        entries = int((sizes * ks).sum())
        return {"bytes": 2 * int(sizes.sum()) * case["dim"] * scalar + entries * (4 + scalar),
                "flops": 3 * case["dim"] * entries}
    n, nq, dim, k = case["points"], case["queries"], case["dim"], case["k"]
    pairs = nq * n if case["kind"] == "brute" else nq * k
    return {"bytes": (n + nq) * dim * scalar + (nq * scalar if case["radii"] else 0) + nq * k * (4 + scalar),
            "flops": 3 * dim * pairs}


def exact(case, seed):
    """Squared distances of the k nearest points in 64 bits, for searches of
    at most 1.1e10 pairs."""
    if case["kind"] == "batch" or case["epsilon"] > 0:
        return None
    n, nq, k = case["points"], case["queries"], case["k"]
    if n * nq > 1.1e10:
        return None
    cloud, queries, radii = _inputs(case, seed)
    eps = float(torch.finfo(cloud.dtype).eps)  # a point at or below it is the query itself
    cloud, queries = cloud.double(), queries.double()
    limit = torch.full((nq,), case["radius"] ** 2 if case["radius"] > 0 else math.inf, dtype=torch.float64,
                       device=DEVICE)
    if radii is not None:
        limit = radii.double() ** 2
    d2 = torch.empty((nq, k), dtype=torch.float64, device=DEVICE)
    rows = max(1, int(5e7 / n))
    for i in range(0, nq, rows):
        q = queries[i:i + rows]
        d = torch.zeros((q.shape[0], n), dtype=torch.float64, device=DEVICE)
        for c in range(case["dim"]):
            d += (q[:, c:c + 1] - cloud[None, :, c]) ** 2
        d[(d <= eps) | (d > limit[i:i + rows, None])] = math.inf
        d2[i:i + rows] = torch.topk(d, k, dim=1, largest=False, sorted=True)[0]
    if case["kind"] == "build_search":
        return dict(indices=None, dists2=d2, nodes=None, height=None, low=None, high=None)
    if case["memory"] in ("host", "pinned"):
        d2 = d2.cpu().numpy()
    return (None, d2, None) if case["memory"] == "device" and case["touch"] and case["kind"] == "search" else (None, d2)
