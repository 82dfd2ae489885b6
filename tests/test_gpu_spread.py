"""Searches too small to fill the GPU run fewer queries per warp: results and
TOUCH_STATISTICS counts stay the oracle's at the sizes where the number of
queries per warp changes."""
import numpy as np
import pytest

import helpers as H
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nq", [1, 2, 33, 151, 2432, 2433, 4865, 40000, 77825])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_queries_spread_over_warps(nq, dtype):
    import libnabo_gb300 as nb
    rng = np.random.default_rng(nq)
    cloud = rng.random((3000, 3)).astype(dtype)
    q = rng.random((nq, 3)).astype(dtype)
    tree = nb.NearestNeighbourSearch(cloud, nb.SearchType.KDTREE_CUDA, creationOptionFlags=nb.TOUCH_STATISTICS)
    gi, gd = tree.knn(q, 5)
    oi, od, ot = O.OracleTree(cloud, creation_flags=O.TOUCH_STATISTICS).knn(q, 5, mode=O.MODE_CANONICAL)
    H.assert_identical(gi, gd, oi, od, f"nq={nq}")
    assert tree.touched == ot
