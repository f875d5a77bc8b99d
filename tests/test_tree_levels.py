"""A tree level's kernels at their edges: the farthest pair of a seed list, the
scan of the partition's items, and the planes made from two centres."""
from __future__ import annotations

import numpy as np
import pytest

from sigmod23ann_b200 import KnngContext, workloads

pytestmark = pytest.mark.gpu

F = np.float32


def _farthest(rows: np.ndarray):
    """First (i, j) in order with the largest squared distance above 0; the
    values are small whole numbers, so that every order of adding is exact."""
    best, pair = 0.0, None
    for i in range(len(rows)):
        for j in range(i + 1, len(rows)):
            dd = float(((rows[i] - rows[j]).astype(np.float64) ** 2).sum())
            if dd > best:
                best, pair = dd, (i, j)
    return pair


@pytest.mark.parametrize("d", [64, 100, 128])
def test_farthest_pair_of_short_and_tied_lists(knng_lib, d):
    """Lists around a CTA's 256 pairs (23 entries make 253, 24 make 276); two
    values a dimension make many ties, equal rows no pair at all."""
    rng = np.random.default_rng(d)
    pts = np.zeros((400, d), F)
    pts[:200, :3] = rng.integers(0, 2, (200, 3))
    pts[200:300] = rng.integers(-9, 10, (100, d))
    lists = [rng.integers(0, 300, m) for m in (1, 2, 3, 22, 23, 24, 33, 64, 65, 90)]
    lists += [rng.integers(0, 200, m) for m in (2, 24, 64)] + [np.arange(300, 340), np.arange(399, 400)]
    off = np.cumsum([0] + [len(x) for x in lists]).astype(np.uint64)
    with KnngContext(0) as ctx:
        ctx.load_points(pts)
        ctx.reset_sets(10)
        ctx.begin_rep()
        first, second, ok = ctx.farthest_pair(off, np.concatenate(lists))
    for a, x in enumerate(lists):
        want = _farthest(pts[x])
        assert bool(ok[a]) == (want is not None), (a, len(x))
        if want is not None:
            assert (int(first[a]), int(second[a])) == want, (a, len(x))


def test_partition_of_many_items(knng_lib):
    """More items than the scan has threads, an uneven share to each: 2,500
    nodes of 1 to 40 points and two of several items."""
    rng = np.random.default_rng(3)
    sizes = rng.integers(1, 41, 2500)
    sizes[[0, 1200]] = 5000, 2049
    ends = np.cumsum(sizes)
    starts = ends - sizes
    pts = np.zeros((int(ends[-1]), 64), F)
    pts[:, 7] = rng.integers(-4, 5, len(pts))
    coefs = np.zeros((2500, 64), F)
    coefs[:, 7] = 1
    at = np.where(np.arange(2500) % 3 == 0, F(-0.5), F(0.5))
    with KnngContext(0) as ctx:
        ctx.load_points(pts)
        ctx.reset_sets(10)
        ctx.begin_rep()
        mids = ctx.split_nodes(starts, ends, coefs, at)
        idx = ctx.indices()
    side = pts[:, 7] > np.repeat(at, sizes)
    got = np.zeros(len(pts), bool)  # True where a position holds a point of the node's first part
    for s, e, mid in zip(starts, ends, mids):
        assert np.array_equal(np.sort(idx[s:e]), np.arange(s, e))
        got[idx[s:mid]] = True
    first_is_true = got[side].all() and not got[~side].any()
    first_is_false = got[~side].all() and not got[side].any()
    assert first_is_true or first_is_false


@pytest.mark.parametrize("d", [64, 128])
def test_repetition_in_other_dimensions(oracle_lib, knng_lib, d):
    """Planes made inside the side test, with and without a tail of dims (100
    dims have one): positions and buckets equal the oracle's."""
    pts = workloads.gaussian_mixture(n=9_000, d=d, clusters=24, sigma=0.15, seed=d)
    o = oracle_lib.Oracle(pts, k=20, rng_mode=1, seed=31)
    o.rep(2, 300, 0)
    with KnngContext(0) as ctx:
        ctx.load_points(pts)
        ctx.reset_sets(20)
        ctx.run_rep(300, 2, 3000, 31, 0)
        np.testing.assert_array_equal(ctx.indices(), o.indices())
        s, e = ctx.leaves()
        t = o.trace()
        order = np.argsort(t["leaf_start"])
        np.testing.assert_array_equal(s, t["leaf_start"][order])
        np.testing.assert_array_equal(e, t["leaf_end"][order])


@pytest.mark.parametrize("n,nd,leaf", [(65, 1, 33), (1024, 7, 31), (1057, 32, 64), (2081, 30, 1025), (3300, 3, 2)])
def test_kd_sums_at_batch_and_chunk_edges(oracle_lib, knng_lib, n, nd, leaf):
    """Nodes of every size from the bucket bound up: batches of 32 rows and
    chunks of 1,024 that end early, one rotated dimension and all 32."""
    pts = workloads.gaussian_mixture(n=n, d=100, clusters=8, sigma=0.3, seed=n)
    o = oracle_lib.Oracle(pts, k=10)
    o.kd_rep(leaf, nd, 99, 0)
    with KnngContext(0) as ctx:
        ctx.load_points(pts)
        ctx.reset_sets(10)
        ctx.run_rep_kd(leaf, nd, 99, 0)
        np.testing.assert_array_equal(ctx.indices(), o.indices())


def test_list_lengths_in_turn_on_one_context(knng_lib):
    """The captured repetition is kept by the arrays it was captured with: lists of
    several lengths in turn, the sets' arrays allocated anew each time and other
    memory taken between, give the lists of fresh contexts."""
    from sigmod23ann_b200 import default_params

    pts = workloads.gaussian_mixture(n=7000, d=64, clusters=8, sigma=0.2, seed=41)

    def params(k: int):
        return default_params(k=k, reps=2, refine=1, max_leaf=257, max_leaf_odd=0, lloyd_iters=1, seed=2)

    want = {}
    for k in (100, 10, 77, 99):
        with KnngContext(0) as c:
            want[k] = c.build(pts, params(k), want_dists=True)
    with KnngContext(0) as c:
        for k in (100, 10, 100, 77, 99, 10, 100, 99, 77, 100):
            ids, dists = c.build(pts, params(k), want_dists=True)
            assert np.array_equal(ids, want[k][0]), k
            assert np.array_equal(dists.view(np.uint32), want[k][1].view(np.uint32)), k
