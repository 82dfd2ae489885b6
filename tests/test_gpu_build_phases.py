"""The device build's phases meet at sizes of their own: segments one block
splits in shared memory (4096 points for small records, down to 512 for the
largest), chunks of positions owned by one block, windows of 32 points. The
tree is the oracle's node for node, leaf order included, on both sides of each
(nabo/kdtree_cpu.cpp:109-225), with ties that make the reference partition
twice and cuts that are clamped to the points' range."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _same_tree(t, o, label):
    for f in ("cut_dim", "right", "bucket_start", "bucket_count", "buckets"):
        assert np.array_equal(t[f], o[f]), f"{label}: {f}"
    inner = o["cut_dim"] >= 0
    assert np.array_equal(t["cut_val"][inner], o["cut_val"][inner]), f"{label}: cuts"


def _cloud(kind, n, dim, dtype, seed):
    rng = np.random.default_rng(seed)
    if kind == "uniform":
        c = rng.random((n, dim))
    elif kind == "grid":  # points on the cuts, many of them equal
        c = rng.integers(0, 9, (n, dim)).astype(float)
    elif kind == "steep":  # clamped cuts, tall trees
        c = np.exp(-rng.exponential(3.0, (n, dim)))
    else:  # half the points equal, the rest on a line
        c = np.where(rng.random((n, 1)) < 0.5, 0.25, np.linspace(-1, 1, n)[:, None] * np.ones((1, dim)))
    return c.astype(dtype)


def _check(cloud, bucket, label):
    import libnabo_gb300 as nb
    tree = nb.NearestNeighbourSearch(cloud, nb.SearchType.KDTREE_CUDA, params=dict(bucketSize=bucket))
    orc = O.OracleTree(cloud, bucket_size=bucket)
    _same_tree(tree.export_tree(), orc.export(), label)
    assert tree.height == orc.height, label


@pytest.mark.parametrize("n", [9, 31, 32, 33, 64, 65, 255, 257, 511, 513, 1023, 1025, 2047, 2049, 4095, 4096, 4097, 5121,
                               155650])
@pytest.mark.parametrize("kind", ["uniform", "grid", "steep", "half"])
def test_sizes_at_phase_edges(n, kind):
    _check(_cloud(kind, n, 3, np.float32, n), 8, f"{kind} {n}")


@pytest.mark.parametrize("dim,dtype", [(1, np.float32), (2, np.float64), (3, np.float64), (4, np.float32),
                                       (5, np.float32), (8, np.float64), (16, np.float32), (16, np.float64)])
@pytest.mark.parametrize("n", [600, 1100, 2100, 20000])
def test_record_sizes(dim, dtype, n):
    for kind in ("uniform", "grid"):
        _check(_cloud(kind, n, dim, dtype, n + dim), 8, f"{kind} {n} D={dim} {np.dtype(dtype).name}")


@pytest.mark.parametrize("bucket", [2, 3, 16, 31, 32, 33, 256, 300, 5000, 30000])
def test_bucket_sizes(bucket):
    for kind in ("uniform", "half"):
        _check(_cloud(kind, 20000, 3, np.float32, bucket), bucket, f"{kind} bucket {bucket}")


def test_records_that_do_not_stay_in_shared_memory():
    # 16-D doubles: more than a block's shared memory per chunk from 1,300 points an SM
    _check(_cloud("uniform", 260000, 16, np.float64, 1), 8, "16-D double")
    _check(_cloud("grid", 260000, 16, np.float64, 2), 8, "16-D double grid")


@pytest.mark.parametrize("graph", [False, True])
def test_batch_across_phases(graph):
    import torch
    import libnabo_gb300 as nb
    sizes = [5, 8, 9, 40, 256, 257, 3000, 4096, 4097, 9000, 2, 30000, 12, 70000, 5000]
    kinds = ["uniform", "grid", "steep", "half"]
    clouds = [_cloud(kinds[i % 4], n, 3, np.float32, 90 + i) for i, n in enumerate(sizes)]
    b = nb.BatchSearch(sizes, dim=3, maxLevels=200)
    b.set_queries([1] * len(sizes), [1] * len(sizes))
    tc = torch.from_numpy(np.concatenate(clouds)).cuda()
    tq = torch.zeros((len(sizes), 3), device="cuda")
    for _ in range(2):
        if graph:
            b.run(tc, tq)
        else:
            b.build(tc)
    torch.cuda.synchronize()
    assert b.status()["ok"], b.status()
    for c, cloud in enumerate(clouds):
        _same_tree(b.export_tree(c), O.OracleTree(cloud).export(), f"cloud {c}")
