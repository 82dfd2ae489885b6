"""Double kd-tree searches decide near sides and far children on float bounds
and compute the exact box distances only where a child may be visited: results
and TOUCH_STATISTICS counts stay bit-identical to the oracle's canonical
traversal where the bounds are weakest -- queries on the cuts, coordinates
whose squares underflow or exceed the float range, far queries, NaN and
infinite queries, leaves of more than 32 points (nabo/kdtree_cpu.cpp:367-447)."""
import numpy as np
import pytest

import helpers as H
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _check(cloud, q, k, eps=0.0, bucket=8, radius=np.inf):
    import libnabo_gb300 as nb
    tree = nb.NearestNeighbourSearch(cloud, nb.SearchType.KDTREE_CUDA, creationOptionFlags=nb.TOUCH_STATISTICS,
                                     params=dict(bucketSize=bucket))
    orc = O.OracleTree(cloud, bucket_size=bucket, creation_flags=O.TOUCH_STATISTICS)
    for flags in (0, nb.ALLOW_SELF_MATCH):
        gi, gd = tree.knn(q, k, eps, flags, radius)
        oi, od, ot = orc.knn(q, k, eps, flags, radius, mode=O.MODE_CANONICAL)
        H.assert_identical(gi, gd, oi, od, f"k={k} eps={eps} bucket={bucket} flags={flags}")
        assert tree.touched == ot


@pytest.mark.parametrize("dim", [1, 2, 3, 4, 7, 8, 16])
@pytest.mark.parametrize("k", [1, 5, 16])
def test_grid_points_queried_on_the_cuts(dim, k):
    rng = np.random.default_rng(dim)
    cloud = rng.integers(0, 6, (3000, dim)).astype(np.float64)
    q = rng.integers(0, 12, (700, dim)) / 2.0
    for eps in (0.0, 0.5):
        _check(cloud, q, k, eps)


@pytest.mark.parametrize("scale", [1e-160, 1e-40, 1e-21, 1e-6, 1e19, 1e30, 1e60])
def test_scales_around_the_float_range(scale):
    rng = np.random.default_rng(5)
    cloud = (rng.random((3000, 3)) - 0.3) * scale
    q = (rng.random((500, 3)) - 0.3) * scale
    q[:100] = cloud[:100] * (1.0 + 1e-12)
    for eps in (0.0, 0.1):
        _check(cloud, q, 5, eps)


@pytest.mark.parametrize("bucket", [2, 31, 32, 33, 70])
@pytest.mark.parametrize("k", [8, 32])
def test_leaf_sizes(bucket, k):
    rng = np.random.default_rng(bucket)
    cloud = rng.normal(size=(4000, 3))
    _check(cloud, rng.normal(size=(600, 3)), k, 0.0, bucket)
    _check(cloud, rng.normal(size=(600, 3)), k, 0.5, bucket, radius=0.2)


def test_offset_cloud_far_and_non_finite_queries():
    rng = np.random.default_rng(9)
    cloud = 1e7 + rng.random((5000, 3)) * 1e-2  # differences far below the bounds' error
    q = 1e7 + rng.random((400, 3)) * 1e-2
    q[::7] += 1e9
    q[1::40] = np.inf
    q[2::40, 1] = -np.inf
    q[3::40] = np.nan
    q[4::40, 2] = np.nan
    for k in (1, 10):
        _check(cloud, q, k)
        _check(cloud, q, k, 2.0)
