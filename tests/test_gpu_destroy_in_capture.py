"""Destroying a search object while a stream capture is open, in the mode that torch.cuda.graph takes by default: in
another thread's capture or the destroying thread's own, the graph stays valid and the object's memory goes back."""
import ctypes
import gc
import threading

import numpy as np
import pytest

torch = pytest.importorskip("torch")

import libnabo_gb300 as nb
from libnabo_gb300 import _native
from libnabo_gb300 import synthetic as S

pytestmark = pytest.mark.gpu


def _capture_while(action, mode):
    x = torch.zeros(64, device="cuda")
    y = torch.zeros_like(x)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode=mode):
        y.copy_(x + 1)
        action()
        y.add_(1)
    x.fill_(2)
    graph.replay()
    torch.cuda.synchronize()
    assert bool((y == 4).all())


def _elsewhere(f):
    def action():
        t = threading.Thread(target=f)
        t.start()
        t.join()
    return action


def _destroy(s, codes):
    codes.append(_native.lib.nabo_cuda_destroy(s._h))
    s._h = ctypes.c_void_p()


@pytest.mark.parametrize("mode", ["global", "thread_local", "relaxed"])
@pytest.mark.parametrize("own", [False, True], ids=["another_thread", "own_thread"])
@pytest.mark.parametrize("kind", [nb.SearchType.KDTREE_CUDA, nb.SearchType.BRUTE_FORCE_CUDA])
def test_graph_stays_valid(kind, own, mode):
    cloud = S.uniform(3000, 3, seed=11)
    s = nb.NearestNeighbourSearch(cloud, kind)
    s.knn(cloud[:100], 5)  # (with the staging a host call keeps)
    codes = []
    action = lambda: _destroy(s, codes)
    _capture_while(action if own else _elsewhere(action), mode)
    assert codes == [0]


def test_memory_goes_back():
    cloud = torch.rand((8_000_000, 3), device="cuda")  # 256 MB of records and nodes
    nb.NearestNeighbourSearch(cloud)
    gc.collect()
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    for _ in range(16):
        s = nb.NearestNeighbourSearch(cloud)
        codes = []
        _capture_while(_elsewhere(lambda: _destroy(s, codes)), "global")
        assert codes == [0]
    # 16 lost objects would be 4 GB; the pool keeps 2 GiB at most
    assert before - torch.cuda.mem_get_info()[0] < (5 << 29)
