"""The bucket pass at the edges of its row blocks, column blocks and mark
windows, with empty, part-filled and full sets, against the oracle's pass over
the same bucket."""
from __future__ import annotations

import os

import numpy as np
import pytest

from helpers import assert_sets_equal
from sigmod23ann_b200 import KnngContext, KnngError, default_params, workloads

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


# Column blocks of 128, and the mark window of 1,024 to the point; with blocks of
# 16 rows here, and of 32 (other points in the set, in no bucket) below.
@pytest.mark.parametrize("n", [127, 128, 129, 255, 256, 257, 1024, 1152, 1153, 2048])
@pytest.mark.parametrize("d,k", [(64, 10), (100, 100), (128, 128)])
def test_column_block_edges(knng_lib, oracle_lib, n, d, k):
    pts = workloads.gaussian_mixture(n=n, d=d, clusters=4, sigma=0.2, seed=n + 1)
    pts[50:60] = pts[40:50]  # equal distances: the update's tie order
    o = _oracle_bucket_sets(oracle_lib, pts, k, 1)
    rest = workloads.gaussian_mixture(n=9600, d=d, clusters=4, sigma=0.2, seed=n)
    for held in (pts, np.concatenate([pts, rest])):
        with KnngContext(0) as c:
            c.load_points(held)
            c.reset_sets(k)
            for _ in range(2):  # the second pass meets every member again
                c.begin_rep()
                c.process_leaves([0], [n])
                got = {key: v[:n] for key, v in c.sets().items()}
                assert_sets_equal(got, o, f"n {n} d {d} k {k} of {len(held)}")


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


def _smallest_budget(call, high):
    """The smallest budget, to 256 bytes, that `call` runs with on a fresh context."""
    low = 1 << 20
    while high - low > 256:
        mid = (low + high) // 2
        try:
            with KnngContext(0, mid) as c:
                call(c)
            high = mid
        except KnngError as e:
            assert e.status == 4
            low = mid
    return high


@pytest.mark.parametrize("n,d,k,leaf", [(9000, 100, 20, 300), (12_001, 64, 10, 90)])
def test_the_pass_needs_no_memory_of_its_own(knng_lib, n, d, k, leaf):
    """Buckets given by the caller run with the budget that points, order, sets
    and the bucket bounds take up, without room for a list of row blocks, and to
    the same sets (blocks of 16 and of 32 rows, empty buckets and single points
    among them)."""
    pts = workloads.gaussian_mixture(n=n, d=d, clusters=8, sigma=0.2, seed=n)
    cuts = [0, 0, 1, 2, 5, 100, *range(100 + leaf, n, leaf), n]
    starts, ends = np.array(cuts[:-1], np.uint32), np.array(cuts[1:], np.uint32)
    got = {}

    def call(c):
        c.load_points(pts)
        c.reset_sets(k)
        for _ in range(2):
            c.process_leaves(starts, ends)
        got["sets"] = c.sets()

    with KnngContext(0) as c:
        call(c)
    want = got["sets"]
    held = n * (4 * d + 8 + 8 * k + 12) + 2 * (4 * len(starts) + 16)
    assert _smallest_budget(call, 64 << 20) <= held + 256
    with KnngContext(0, held) as c:
        call(c)
    assert_sets_equal(got["sets"], want, "without a list")
    # A list that fitted gives way to what is allocated after it.
    with KnngContext(0, held + 2 * (n // 16 + len(starts) + 8) * 4) as c:
        call(c)
        assert_sets_equal(got["sets"], want, "with a list")
    room = held + 4 * n * k + 64
    with KnngContext(0, room) as c:
        call(c)
        ids = c.finalize()
    with KnngContext(0) as c:
        call(c)
        assert np.array_equal(c.finalize(), ids)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("offsets", [None, [0, 1, 2, 4, 7, 4000, 6001]])
def test_items_fit_behind_the_leaves(knng_lib, precision, offsets):
    """Repetitions with the smallest buckets (two points and one; point sets of one
    point too), where leaves and row blocks fill their arrays: the lists of the
    form that keeps its own."""
    n = 6001
    pts = workloads.gaussian_mixture(n=n, d=64, clusters=8, sigma=0.2, seed=5)
    lists = []
    for loop in ("graph", "device", "host"):
        os.environ["KNNG_REP_LOOP"] = loop
        try:
            with KnngContext(0) as c:
                p = default_params(k=7, reps=2, refine=0, max_leaf=3, max_leaf_odd=2, lloyd_iters=1, precision=precision)
                if offsets is None:
                    lists.append(c.build(pts, p))
                else:
                    lists.append(np.concatenate(c.build_batch([pts[a:b] for a, b in zip(offsets, offsets[1:])], p)))
        finally:
            os.environ.pop("KNNG_REP_LOOP", None)
    assert np.array_equal(lists[0], lists[2])
    assert np.array_equal(lists[1], lists[2])


@pytest.mark.parametrize("n", [2, 33, 129, 130, 131, 160, 256, 257, 300, 1000])
@pytest.mark.parametrize("d", [64, 100, 128])
def test_precision_form_keeps_the_128_best(knng_lib, n, d):
    """Points with small integer coordinates: the BF16 estimates are the exact
    distances, with many ties, so the kept candidates of a bucket are the 128
    smallest by (distance, position) and lists of 128 hold just them."""
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
