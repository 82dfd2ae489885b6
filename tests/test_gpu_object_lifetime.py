"""Destroying a search object: it waits for searches still running on other streams, and leaves a stream capture that
another thread has open alone (a library thread may be capturing its own graph, and so may a user's)."""
import threading

import numpy as np
import pytest

torch = pytest.importorskip("torch")

import libnabo_gb300 as nb
from libnabo_gb300 import synthetic as S

pytestmark = pytest.mark.gpu

KINDS = [nb.SearchType.KDTREE_CUDA, nb.SearchType.BRUTE_FORCE_CUDA]


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("kind", KINDS)
def test_destroy_during_another_threads_capture(kind, dtype):
    cloud = S.uniform(3000, 3, seed=11).astype(dtype)
    objects = [nb.NearestNeighbourSearch(cloud, kind)]
    x = torch.zeros(64, device="cuda")
    y = torch.zeros_like(x)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode="thread_local"):
        y.copy_(x + 1)
        t = threading.Thread(target=objects.clear)
        t.start()
        t.join()
    x.fill_(2)
    graph.replay()
    torch.cuda.synchronize()
    assert bool((y == 3).all())


@pytest.mark.parametrize("kind", KINDS)
def test_destroy_waits_for_running_searches(kind):
    cloud, query = S.uniform(100_000, 3, seed=12), S.uniform(50_000, 3, seed=13)
    tq = torch.from_numpy(query).cuda()
    s = nb.NearestNeighbourSearch(cloud, kind)
    want = s.knn_device(tq, 10)
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        for _ in range(4):
            got = s.knn_device(tq, 10)
    del s
    other = nb.NearestNeighbourSearch(S.uniform(100_000, 3, seed=14), kind)  # takes the freed memory
    torch.cuda.synchronize()
    assert torch.equal(want[0], got[0]) and torch.equal(want[1], got[1])
    del other
