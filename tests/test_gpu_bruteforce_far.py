"""Float brute force on clouds whose points are not all of one range: a few far points, heavy tails, two scales. The
tensor-core filter takes its coordinates from a sample and its slack from each stage of points, and tests far points
exactly: results are the oracle's (nabo/brute_force_cpu.cpp:63-103), and far points cost what they are, not the filter."""
import numpy as np
import pytest

import helpers as H
from oracle import oracle as O

import libnabo_gb300 as nb
from libnabo_gb300 import synthetic as S

pytestmark = pytest.mark.gpu


def _check(cloud, q, k, flags=0, label=""):
    gi, gd = nb.NearestNeighbourSearch(cloud, nb.SearchType.BRUTE_FORCE_CUDA).knn(q, k, 0.0, flags)
    oi, od, _ = O.bf_knn(cloud, q, k, flags, np.inf, None, mode=O.MODE_CANONICAL)
    H.assert_identical(gi, gd, oi, od, label)


@pytest.mark.parametrize("k", [1, 5, 16, 32])
@pytest.mark.parametrize("dim", [2, 3, 8, 16])
def test_far_points(dim, k):
    rng = np.random.default_rng(dim * 40 + k)
    for n in (512, 4097, 9000):
        base = rng.random((n, dim)).astype(np.float32)
        for far in (8.0, 40.0, 130.0, 1e4, 1e9):  # about the largest norm the filter holds, and beyond
            cloud = base.copy()
            i = rng.choice(n, 5, replace=False)
            cloud[i[0], 0] = far
            cloud[i[1]] = -far
            cloud[i[2:], dim - 1] = far * (1 + rng.random(3)).astype(np.float32)
            q = np.concatenate([rng.random((150, dim)), cloud[i], cloud[i] + rng.normal(size=(5, dim)),
                                rng.normal(size=(20, dim)) * far]).astype(np.float32)
            for flags in (0, 1):
                _check(cloud, q, k, flags, f"D={dim} k={k} n={n} far={far}")


@pytest.mark.parametrize("kind", ["lognormal", "cauchy", "two scales", "one point and some", "far half", "seeds"])
def test_heavy_tails(kind):
    rng = np.random.default_rng(7)
    n = 20000
    if kind == "lognormal":
        cloud = np.exp(rng.normal(0, 3, (n, 3)))
    elif kind == "cauchy":
        cloud = rng.standard_cauchy((n, 3))
    elif kind == "two scales":  # 1 % of the points a million times farther out
        cloud = rng.random((n, 3)) * np.where(rng.random((n, 1)) < 0.01, 1e6, 1.0)
    elif kind == "one point and some":  # the sample's reach is zero
        cloud = np.where(np.arange(n)[:, None] % 1500 == 7, rng.random((n, 3)) * 50, np.array([[3.0, -1.0, 2.0]]))
    elif kind == "far half":
        cloud = rng.random((n, 3)) + np.where(np.arange(n)[:, None] < n // 2, 0.0, 3e5)
    else:  # every stage of the seed pass holds far points, and nothing else near
        cloud = rng.random((n, 3))
        cloud[(np.arange(n) // 256) % 8 == 0] *= 1e5
    cloud = cloud.astype(np.float32)
    q = np.concatenate([cloud[rng.choice(n, 300)], cloud[rng.choice(n, 300)] * np.float32(1.001)])
    for k in (1, 5, 20):
        for flags in (0, 1):
            _check(cloud, q, k, flags, f"{kind} k={k}")


def _times(pairs, k):
    """Median event times of (cloud, queries) searches, taken in turn."""
    torch = pytest.importorskip("torch")
    work = [(nb.NearestNeighbourSearch(c, nb.SearchType.BRUTE_FORCE_CUDA), torch.from_numpy(q).cuda()) for c, q in pairs]
    times = [[] for _ in work]
    for _ in range(11):
        for (s, q), t in zip(work, times):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            s.knn_device(q, k)
            b.record()
            torch.cuda.synchronize()
            t.append(a.elapsed_time(b))
    return [float(np.median(t)) for t in times]


def test_a_far_return_does_not_cost_the_filter():
    """Without its filter the far cloud took 4.5 times as long as the scan itself."""
    scan = S.lidar_scan(n_azimuth=1800)
    far = scan.copy()
    far[len(far) // 3] = (1e4, 0.0, 0.0)
    near_ms, far_ms = _times([(scan, scan), (far, scan)], 5)
    assert far_ms < 2.0 * near_ms


def test_idle_slots_of_an_offset_cloud_cost_nothing():
    """1000 queries leave a part of the last block idle; taken for queries at the origin, far beyond the cloud, its slots
    made the search 1.8 times as long."""
    cloud = np.random.default_rng(1).random((100_000, 3)).astype(np.float32)
    shifted = cloud + np.float32(3e5)
    at_origin, offset = _times([(cloud, cloud[:1000]), (shifted, shifted[:1000])], 5)
    assert offset < 1.4 * at_origin
