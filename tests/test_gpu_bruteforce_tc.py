"""Float brute force with its distance filter on the tensor cores: bit-identical
to the oracle's brute force at the edges of its tiles (128 queries, 128 points,
stages of 128 or 256 points), block rows and seed pass, and where the filter's
error bound matters: ties, duplicates of the query, far and non-finite queries,
offset clouds, ranges it refuses (nabo/brute_force_cpu.cpp:63-103)."""
import numpy as np
import pytest

import helpers as H
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _check(cloud, q, k, flags=0, radius=np.inf, radii=None, label=""):
    import libnabo_gb300 as nb
    bf = nb.NearestNeighbourSearch(cloud, nb.SearchType.BRUTE_FORCE_CUDA)
    gi, gd = bf.knn(q, k, 0.0, flags, radius, maxRadii=radii)
    oi, od, _ = O.bf_knn(cloud, q, k, flags, radius, radii, mode=O.MODE_CANONICAL)
    H.assert_identical(gi, gd, oi, od, label)


@pytest.mark.parametrize("n", [511, 512, 513, 639, 640, 641, 2047, 2048, 2049, 4095, 4225, 20000])
@pytest.mark.parametrize("nq", [1, 127, 128, 129, 700])
def test_tile_edges(n, nq):
    rng = np.random.default_rng(n + nq)
    cloud = rng.random((n, 3)).astype(np.float32)
    q = rng.random((nq, 3)).astype(np.float32)
    _check(cloud, q, 5, label=f"n={n} nq={nq}")


@pytest.mark.parametrize("dim", [1, 2, 3, 4, 5, 8, 13, 16])
@pytest.mark.parametrize("k", [1, 2, 4, 8, 10, 11, 16, 17, 32])
def test_dimensions_and_list_sizes(dim, k):
    rng = np.random.default_rng(dim * 100 + k)
    cloud = (rng.normal(size=(6000, dim)) * 3.0).astype(np.float32)
    q = (rng.normal(size=(300, dim)) * 3.0).astype(np.float32)
    _check(cloud, q, k, label=f"D={dim} k={k}")
    _check(cloud, cloud[:300], k, label=f"D={dim} k={k} own points")


def test_ties_duplicates_and_self_matches():
    rng = np.random.default_rng(1)
    grid = rng.integers(0, 7, (5000, 3)).astype(np.float32)  # many copies of every query
    for flags in (0, 1):
        for k in (1, 5, 20):
            _check(grid, grid[:400], k, flags, label=f"grid k={k} flags={flags}")
    same = np.tile(np.array([[0.5, -2.0, 8.0]], np.float32), (3000, 1))
    same[::7] += rng.random((same[::7].shape[0], 3)).astype(np.float32)
    _check(same, same[:200], 8, label="mostly one point")
    flat = rng.random((4000, 3)).astype(np.float32)
    flat[:, 1] = 3.0
    _check(flat, flat[:200] + np.float32(1e-4), 5, label="flat cloud")


def test_radii():
    rng = np.random.default_rng(2)
    cloud = rng.random((9000, 3)).astype(np.float32)
    q = rng.random((500, 3)).astype(np.float32)
    for r in (0.0, 0.01, 0.05):
        _check(cloud, q, 10, radius=r, label=f"r={r}")
    radii = rng.random(500).astype(np.float32) * np.float32(0.1)
    radii[::9] = np.nan
    radii[1::9] = np.inf
    _check(cloud, q, 10, radii=radii, label="radii")


@pytest.mark.parametrize("offset,scale", [(0.0, 1e-12), (0.0, 1e12), (1e3, 1e-3), (3e4, 1.0), (-7e6, 10.0), (0.0, 1e16),
                                          (0.0, 1e25)])
def test_ranges(offset, scale):
    rng = np.random.default_rng(3)
    cloud = (offset + scale * rng.random((5000, 3))).astype(np.float32)
    q = (offset + scale * rng.random((300, 3))).astype(np.float32)
    q[:20] += np.float32(scale * 3e3)  # beyond the filter's query range
    q[20:40] *= np.float32(30.0)
    _check(cloud, q, 7, label=f"offset {offset} scale {scale}")


def test_non_finite_and_huge_queries():
    rng = np.random.default_rng(4)
    cloud = rng.random((5000, 3)).astype(np.float32)
    q = rng.random((256, 3)).astype(np.float32)
    q[0] = np.nan
    q[1, 1] = np.inf
    q[2, 2] = -np.inf
    q[3] = 1e30
    q[4] = -3e19
    q[5] = 1e18
    _check(cloud, q, 5, label="non-finite queries")
