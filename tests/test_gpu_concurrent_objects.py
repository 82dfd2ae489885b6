"""Host threads that build trees, or search different objects, at the same time: what one call asks of the device (the
shared memory its kernels may take, which is a setting of the kernel and not of the call) does not fail another's, and
every tree is the oracle's."""
import threading

import numpy as np
import pytest

import helpers as H
from oracle import oracle as O

import libnabo_gb300 as nb

pytestmark = pytest.mark.gpu


def _run(workers):
    errors = []

    def guarded(f):
        try:
            f()
        except Exception as e:  # noqa: BLE001 -- reported below
            errors.append(e)

    threads = [threading.Thread(target=guarded, args=(f,)) for f in workers]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


@pytest.mark.parametrize("split_rule", [0, 1], ids=["reference", "median"])
def test_builds_of_different_sizes_and_buckets(split_rule):
    rng = np.random.default_rng(31)
    setups = [(10_000, 8, 60), (83_000, 16, 40), (83_000, 32, 40), (1_000_000, 8, 12)]
    clouds = [rng.random((n, 3)).astype(np.float32) for n, _, _ in setups]
    trees = [None] * len(setups)

    def worker(i):
        _, bucket, repeats = setups[i]
        for _ in range(repeats):
            trees[i] = nb.NearestNeighbourSearch(clouds[i], params=dict(bucketSize=bucket, splitRule=split_rule))

    _run([lambda i=i: worker(i) for i in range(len(setups))])
    for i, (n, bucket, _) in enumerate(setups):
        t = trees[i].export_tree()
        if split_rule == 0:
            o = O.OracleTree(clouds[i], bucket_size=bucket).export()
            for f in ("cut_dim", "right", "bucket_start", "bucket_count", "buckets"):
                assert np.array_equal(t[f], o[f]), (n, f)
        else:
            alone = nb.NearestNeighbourSearch(clouds[i], params=dict(bucketSize=bucket, splitRule=1)).export_tree()
            assert np.array_equal(t["buckets"], alone["buckets"]) and np.array_equal(t["right"], alone["right"]), n


def test_long_lists_in_trees_of_different_heights():
    """k above 32: the stacks are in shared memory, sized by the tree's height."""
    rng = np.random.default_rng(32)
    clouds = [rng.random((20_000, 16)), np.exp(-rng.exponential(3.0, (20_000, 16))), rng.random((3_000, 16))]
    query = rng.random((300, 16))
    objects = [nb.NearestNeighbourSearch(c) for c in clouds]
    assert len({s.height for s in objects}) > 1
    want = [O.OracleTree(c).knn(query, 50, mode=O.MODE_CANONICAL)[:2] for c in clouds]
    got = [None] * len(clouds)

    def worker(i):
        for _ in range(60):
            got[i] = objects[i].knn(query, 50)

    _run([lambda i=i: worker(i) for i in range(len(clouds))])
    for i, (oi, od) in enumerate(want):
        H.assert_identical(got[i][0], got[i][1], oi, od, f"object {i}")
