"""The bucket pass at the edges of its row blocks, column blocks and mark
windows, with empty, part-filled and full sets, against the oracle's pass over
the same bucket."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import assert_sets_equal
from sigmod23ann_b200 import KnngContext, workloads

pytestmark = pytest.mark.gpu


def _oracle_bucket_sets(oracle_lib, pts, k, reps):
    """Sets after `reps` passes over the whole set as one bucket in id order."""
    o = oracle_lib.Oracle(pts, k=k, rng_mode=1, seed=1)
    for r in range(reps):
        o.rep(1, 5000, r)
    return o.sets()


# Rows of a block: 16 below 9,472 points, 32 above; columns 64; marks for 1,024
# columns at a time.
@pytest.mark.parametrize("n", [2, 3, 15, 16, 17, 63, 64, 65, 130, 1023, 1025, 2100])
@pytest.mark.parametrize("d,k", [(64, 10), (100, 100), (128, 128)])
def test_one_bucket(knng_lib, oracle_lib, n, d, k):
    pts = workloads.gaussian_mixture(n=n, d=d, clusters=4, sigma=0.2, seed=n)
    if n > 100:
        pts[50:60] = pts[40:50]  # equal distances: the update's tie order
    o = _oracle_bucket_sets(oracle_lib, pts, k, 1)
    with KnngContext(0) as c:
        c.load_points(pts)
        c.reset_sets(k)
        for _ in range(2):  # the second pass meets every member again
            c.begin_rep()
            c.process_leaves([0], [n])
            assert_sets_equal(c.sets(), o, f"n {n} d {d} k {k}")
        # The same sets handed over, and met again.
        c.set_sets(o)
        c.process_leaves([0], [n])
        assert_sets_equal(c.sets(), o, "handed over")


def test_many_buckets_in_blocks_of_32_rows(knng_lib, oracle_lib):
    n, d, k = 12_000, 100, 100
    pts = workloads.gaussian_mixture(n=n, d=d, clusters=8, sigma=0.2, seed=3)
    rng = np.random.default_rng(4)
    order = rng.permutation(n).astype(np.uint32)
    edges = np.unique(np.concatenate([[0, 1, 3, 35, 99, 131, n], rng.integers(200, n, 30)])).astype(np.uint32)
    with KnngContext(0) as c:
        c.load_points(pts)
        c.reset_sets(k)
        c.set_indices(order)
        keep = np.diff(edges) <= 4096
        c.process_leaves(edges[:-1][keep], edges[1:][keep])
        got = c.sets()
    for s, e in zip(edges[:-1][keep], edges[1:][keep]):
        ids = order[s:e]
        if len(ids) < 2:
            assert (got["size"][ids] == 0).all()
            continue
        o = _oracle_bucket_sets(oracle_lib, np.ascontiguousarray(pts[ids]), k, 1)
        size = o["size"]
        assert np.array_equal(got["size"][ids], size)
        assert np.array_equal(got["dist"][ids].view(np.uint32), o["dist"].view(np.uint32)), (s, e)
        filled = np.arange(k)[None] < size[:, None]
        assert np.array_equal(got["id"][ids][filled], ids[o["id"]][filled])


@pytest.mark.parametrize("n", [2, 33, 129, 130, 131, 160, 256, 257, 300, 1000])
@pytest.mark.parametrize("d", [64, 100, 128])
def test_precision_form_keeps_the_128_best(knng_lib, n, d):
    """Points with small integer coordinates: the BF16 estimates are the exact
    distances, with many ties, so the kept candidates of a bucket are the 128
    smallest by (distance, position) and lists of 128 hold just them."""
    from sigmod23ann_b200 import default_params

    rng = np.random.default_rng(n + d)
    pts = np.zeros((n, d), np.float32)
    pts[:, :6] = rng.integers(-2, 3, (n, 6))
    dist = ((pts[:, None].astype(np.int64) - pts[None].astype(np.int64)) ** 2).sum(-1)
    key = dist * n + np.arange(n)[None]
    np.fill_diagonal(key, np.iinfo(np.int64).max)
    best = np.sort(key, axis=1)[:, :min(128, n - 1)]
    want = np.ones((n, 128), np.uint32)
    want[:, :best.shape[1]] = best % n  # ascending by (distance, id)
    with KnngContext(0) as c:
        got = c.build(pts, default_params(k=128, reps=1, refine=0, max_leaf=1025, max_leaf_odd=0, precision=1))
    assert np.array_equal(got, want)
