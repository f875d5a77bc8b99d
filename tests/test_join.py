"""The join and its replay against the one-warp-per-point pass: list lengths
around the tile's column steps, every dimension, unfilled lists, ranges of
points when the budget is small, and sets handed over with distances that are
not those of the points."""
from __future__ import annotations

import os

import numpy as np
import pytest

from helpers import assert_sets_equal
from sigmod23ann_b200 import KnngContext, Stats, default_params, workloads

pytestmark = pytest.mark.gpu


def _sets_after_reps(pts, k, leaf, reps=2):
    with KnngContext(0) as c:
        c.load_points(pts)
        c.reset_sets(k)
        for r in range(reps):
            c.run_rep(leaf, 1, 3000, seed=5, rep_index=r)
        return c.sets()


def _pass_from(pts, k, sets, budget=0, pointwise=False, passes=1):
    if pointwise:
        os.environ["KNNG_REFINE"] = "pointwise"
    try:
        with KnngContext(0, budget) as c:
            c.load_points(pts)
            c.reset_sets(k)
            c.set_sets(sets)
            st = Stats()
            changed = [c.refine(st) for _ in range(passes)]
            return c.sets(), changed, st
    finally:
        os.environ.pop("KNNG_REFINE", None)


@pytest.mark.parametrize("n,d,k,leaf", [(700, 64, 1, 90), (3001, 64, 10, 65), (2999, 100, 16, 129), (2500, 128, 17, 129),
                                        (3000, 100, 32, 257), (2777, 128, 64, 200), (2500, 64, 65, 257),
                                        (2100, 128, 100, 90), (3000, 100, 127, 300), (2500, 128, 128, 300), (129, 100, 100, 400)])
def test_pass_equals_pointwise(knng_lib, n, d, k, leaf):
    pts = workloads.gaussian_mixture(n=n, d=d, clusters=8, sigma=0.2, seed=n + d)
    # With the sets a build holds (its own distances) and handed over.
    with KnngContext(0) as c:
        c.load_points(pts)
        c.reset_sets(k)
        for r in range(2):
            c.run_rep(leaf, 1, 3000, seed=5, rep_index=r)
        before = c.sets()
        changed = [c.refine(), c.refine()]
        own = c.sets()
    want, want_changed, _ = _pass_from(pts, k, before, pointwise=True, passes=2)
    assert_sets_equal(own, want, "own sets")
    assert changed == want_changed
    given, given_changed, _ = _pass_from(pts, k, before, passes=2)
    assert_sets_equal(given, want, "handed over")
    assert given_changed == want_changed


def test_small_budgets_take_ranges_of_points(knng_lib):
    """With room for some of the points' bits only, the pass goes range by
    range; with room for none, point by point.  The sets are the same."""
    n, d, k = 40_000, 64, 50
    pts = workloads.gaussian_mixture(n=n, d=d, clusters=16, sigma=0.2, seed=8)
    before = _sets_after_reps(pts, k, 129)
    want, want_changed, _ = _pass_from(pts, k, before)
    held = n * (4 * d + 8 + 8 * k + 12)  # points, order, sets
    lists = n * k * 8                    # snapshot and its distances
    seen = set()
    for extra in (64 << 20, 40 << 20, 20 << 20):
        got, changed, st = _pass_from(pts, k, before, budget=held + lists + extra)
        assert_sets_equal(got, want, f"extra {extra}")
        assert changed == want_changed
        seen.add(int(st.refine_join_launches))
    assert max(seen) > 1, seen


@pytest.mark.parametrize("n,d,k,passes", [(20_000, 64, 10, 2), (12_000, 100, 60, 1), (12_000, 100, 60, 2)])
def test_finished_lists_fit_whatever_the_passes_took(knng_lib, n, d, k, passes):
    """From the budget on that a whole build has always needed (its buffers, a
    pass's snapshots and per-edge lists, the finished lists), every budget does:
    a pass that takes its points in ranges takes what there is, and gives way to
    the lists.  The lists are the same."""
    pts = workloads.gaussian_mixture(n=n, d=d, clusters=16, sigma=0.2, seed=n + k)
    p = default_params(k=k, reps=1, refine=passes, max_leaf=257, max_leaf_odd=0, lloyd_iters=1, seed=5)
    with KnngContext(0) as c:
        want = c.build(pts, p, want_dists=True)
    need = n * (4 * d + 8 + 8 * k + 12)  # points, order, sets
    need += n * 64 + (4 << 20)           # a repetition's buffers, small scratch
    need += n * (8 * k + 16) + n * k * 4  # snapshots and their marks, per-edge lists
    need += n * k * 8                    # the finished lists
    for share in range(0, 24):
        with KnngContext(0, need + n * k * share) as c:
            ids, dists = c.build(pts, p, want_dists=True)
        assert np.array_equal(ids, want[0]) and np.array_equal(dists, want[1]), share


@pytest.mark.parametrize("n,d,k,passes", [(20_000, 64, 10, 2), (12_000, 100, 60, 1), (12_000, 100, 60, 2)])
def test_a_context_builds_again_under_any_budget(knng_lib, n, d, k, passes):
    """The same builds three times on one context: what the earlier ones hold (the
    finished lists, a pass's lists of other ranges) is in no later one's way."""
    pts = workloads.gaussian_mixture(n=n, d=d, clusters=16, sigma=0.2, seed=n + k)
    p = default_params(k=k, reps=1, refine=passes, max_leaf=257, max_leaf_odd=0, lloyd_iters=1, seed=5)
    with KnngContext(0) as c:
        want = c.build(pts, p, want_dists=True)
    least = n * (4 * d + 8 + 8 * k + 12)  # points, order, sets
    least += n * 64 + (4 << 20)           # a repetition's buffers, small scratch
    least += n * 4 * k                    # a pass's snapshot
    least += n * k * 8                    # the finished lists
    joins = set()
    for share in range(0, 40):
        with KnngContext(0, least + n * k * share) as c:
            for _ in range(3):
                st = Stats()
                ids, dists = c.build(pts, p, want_dists=True, stats=st)
                assert np.array_equal(ids, want[0]) and np.array_equal(dists, want[1]), share
                joins.add(int(st.refine_join_launches))
    assert max(joins) > passes, joins  # ranges among them


@pytest.mark.parametrize("n,d,k", [(12_000, 64, 50), (9_000, 100, 100)])
def test_no_room_for_a_64th_goes_point_by_point(knng_lib, n, d, k):
    """A budget with room for less than a 64th of the points' join beside its
    reserve: the pass goes point by point, to the same sets, and reports no join,
    also where the pass before it on that context had one."""
    pts = workloads.gaussian_mixture(n=n, d=d, clusters=16, sigma=0.2, seed=8)
    before = _sets_after_reps(pts, k, 129)
    want, want_changed, _ = _pass_from(pts, k, before, pointwise=True)
    held = n * (4 * d + 8 + 8 * k + 12)           # points, order, sets
    lists = n * k * 8 + n * 24                    # snapshot, its distances; counts and offsets
    edges = n * k * 20                            # a full range
    for part, joins in ((100, 0), (2, None)):     # of the edges, beside an eighth in reserve
        got, changed, st = _pass_from(pts, k, before, budget=(held + lists + edges // part) * 8 // 7)
        assert_sets_equal(got, want, f"1/{part} of the edges")
        assert changed == want_changed
        assert st.refine_join_launches > 1 if joins is None else st.refine_join_launches == 0
    # A pass with room, then one without: the finished lists are held by then.
    want, want_changed, _ = _pass_from(pts, k, before, pointwise=True, passes=2)
    with KnngContext(0, (held + lists + edges // 10) * 8 // 7) as c:
        c.load_points(pts)
        c.reset_sets(k)
        c.set_sets(before)
        first, second = Stats(), Stats()
        changed = [c.refine(first)]
        c.finalize(want_dists=True)
        changed.append(c.refine(second))
        assert_sets_equal(c.sets(), want, "with and without room")
    assert changed == want_changed
    assert first.refine_join_launches > 1
    assert second.refine_join_launches == 0
    assert second.refine_pairs == 0 and second.refine_exact == 0 and second.ms_refine_join == 0


@pytest.mark.parametrize("n,d,k", [(12_001, 64, 50), (9_000, 128, 100), (10_000, 100, 17)])
def test_ranges_with_the_previous_lists(knng_lib, monkeypatch, n, d, k):
    """Three passes in several ranges each, with room for the previous pass's lists:
    later passes leave out the pairs those offered (edges marked as old in reverse
    lists that start past the first point).  The sets and changes are those of the
    per-point passes; with the marks switched off more pairs pass the filter."""
    pts = workloads.gaussian_mixture(n=n, d=d, clusters=16, sigma=0.2, seed=14)
    before = _sets_after_reps(pts, k, 129, reps=1)
    want, want_changed, _ = _pass_from(pts, k, before, pointwise=True, passes=3)
    need = n * (4 * d + 8 + 8 * k + 12) + n * k * 8 + n * 24  # points, order, sets; snapshot, distances, offsets
    need += n * (4 * k + 16)                                  # the previous lists and the marks
    need = (need + n * k * 20 * 2 // 5) * 8 // 7              # two fifths of the edges, an eighth in reserve
    got, changed, st = _pass_from(pts, k, before, budget=need, passes=3)
    assert_sets_equal(got, want, "in ranges")
    assert changed == want_changed
    assert st.refine_join_launches > 2 * 3
    monkeypatch.setenv("KNNG_REFINE_SKIP", "0")
    all_got, all_changed, all_st = _pass_from(pts, k, before, budget=need, passes=3)
    assert_sets_equal(all_got, want, "every pair offered")
    assert all_changed == want_changed
    assert st.refine_filter_pass < 0.9 * all_st.refine_filter_pass


def test_distances_of_given_sets_do_not_steer_the_filter(knng_lib):
    """Sets handed over may hold any distances (here a thousandth of the real
    ones, with the real bounds): the filter's norms come from the points."""
    pts = workloads.gaussian_mixture(n=4000, d=100, clusters=8, sigma=0.2, seed=9)
    before = _sets_after_reps(pts, 100, 300)
    before["dist"] = before["dist"] * np.float32(1e-3)
    want, want_changed, _ = _pass_from(pts, 100, before, pointwise=True)
    got, changed, _ = _pass_from(pts, 100, before)
    assert_sets_equal(got, want, "scaled distances")
    assert changed == want_changed


@pytest.mark.parametrize("cap", [1, 31, 64, 257, 700, 1500, 4000, None])
def test_candidates_around_the_cta_cap(knng_lib, monkeypatch, cap):
    """Part-filled lists (buckets under 43 points), so that every point has
    thousands of candidates: the caps of the CTA's replay are passed while its
    eight warps add candidates side by side, at counts below, amid and (None)
    near what the points have."""
    pts = workloads.gaussian_mixture(n=2600, d=64, clusters=8, sigma=0.2, seed=12)
    before = _sets_after_reps(pts, 128, 43, reps=3)
    want, want_changed, _ = _pass_from(pts, 128, before, pointwise=True)
    monkeypatch.setenv("KNNG_REFINE_SLOTS", "0")
    if cap is not None:
        monkeypatch.setenv("KNNG_REFINE_POOL", str(cap))
    got, changed, st = _pass_from(pts, 128, before)
    assert_sets_equal(got, want, f"cap {cap}")
    assert changed == want_changed
    assert st.refine_overflow > 0
    if cap is not None and cap <= 64:
        assert st.refine_lost > 0
