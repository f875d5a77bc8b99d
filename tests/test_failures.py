"""Failure detection without a GPU fault: every wait a kernel makes on its own
bulk copies or tensor-core operations has a poll limit.  A diagnostic entry
point shortens the limit to 0 so that the waits run out on purpose; the kernel
then records the failure, drains what it has in flight and returns, the call
reports KNNG_ERR_CUDA, and the same context runs the next call normally."""
from __future__ import annotations

import numpy as np
import pytest

from sigmod23ann_b200 import KnngContext, KnngError, Stats, default_params, workloads
from sigmod23ann_b200.api import debug_set_wait_limit

pytestmark = pytest.mark.gpu

DEFAULT_LIMIT = 1 << 26


def _same_sets(a: dict, b: dict) -> bool:
    return all(np.array_equal(np.asarray(a[k]).view(np.uint32), np.asarray(b[k]).view(np.uint32)) for k in a)


def test_split_wait_runs_out_and_context_recovers(knng_lib):
    """The Lloyd sums' bulk-copy waits (tree construction) give up at once."""
    pts = workloads.gaussian_mixture(n=6000, d=100, clusters=8, sigma=0.2, seed=31)
    params = default_params(reps=2, refine=1, max_leaf=257, max_leaf_odd=0, lloyd_iters=2, seed=3)
    with KnngContext(0) as ref:
        want = ref.build(pts, params)
    with KnngContext(0) as ctx:
        try:
            debug_set_wait_limit(ctx, 0)
            with pytest.raises(KnngError) as e:
                ctx.build(pts, params)
            assert e.value.status == 2 and "gave up" in str(e.value)
        finally:
            debug_set_wait_limit(ctx, DEFAULT_LIMIT)
        assert np.array_equal(ctx.build(pts, params), want)


def test_join_wait_runs_out_and_context_recovers(knng_lib):
    """The neighbour-of-neighbour join's copy / MMA waits give up at once; the
    sets are left as they were, and the pass then runs normally."""
    pts = workloads.gaussian_mixture(n=6000, d=100, clusters=8, sigma=0.2, seed=32)
    with KnngContext(0) as ref:
        ref.load_points(pts)
        ref.reset_sets(100)
        for r in range(2):
            ref.run_rep(257, 2, 3000, seed=4, rep_index=r)
        ref.refine()
        want = ref.sets()
    with KnngContext(0) as ctx:
        ctx.load_points(pts)
        ctx.reset_sets(100)
        for r in range(2):
            ctx.run_rep(257, 2, 3000, seed=4, rep_index=r)
        before = ctx.sets()
        try:
            debug_set_wait_limit(ctx, 0)
            with pytest.raises(KnngError) as e:
                ctx.refine()
            assert e.value.status == 2 and "gave up" in str(e.value)
        finally:
            debug_set_wait_limit(ctx, DEFAULT_LIMIT)
        assert _same_sets(before, ctx.sets())
        ctx.refine()
        assert _same_sets(want, ctx.sets())


@pytest.mark.parametrize("limit", [1, 2, 3, 5, 8, 20, 100])
def test_short_limits_fail_or_give_the_result(knng_lib, limit):
    """Limits that some waits of a warp's lanes meet and others may not: the
    build reports the failure or returns the right lists, never anything
    between, and the context runs on."""
    pts = workloads.gaussian_mixture(n=9000, d=128, clusters=8, sigma=0.2, seed=33)
    params = default_params(reps=2, refine=0, max_leaf=129, max_leaf_odd=0, lloyd_iters=2, seed=3)
    with KnngContext(0) as ref:
        want = ref.build(pts, params)
    with KnngContext(0) as ctx:
        try:
            debug_set_wait_limit(ctx, limit)
            try:
                assert np.array_equal(ctx.build(pts, params), want)
            except KnngError as e:
                assert e.status == 2 and "gave up" in str(e)
        finally:
            debug_set_wait_limit(ctx, DEFAULT_LIMIT)
        assert np.array_equal(ctx.build(pts, params), want)


@pytest.mark.parametrize("fails_in", [0, 1, 2, 4])
def test_a_pass_in_ranges_is_whole_or_not_started(knng_lib, monkeypatch, fails_in):
    """A budget with room for part of the points' join: the pass goes in ranges.
    The first range's join gives up: the call fails and no set has changed.  A
    later one's: the pass ends with the sets it ends with otherwise."""
    n, d, k = 12_000, 64, 50
    pts = workloads.gaussian_mixture(n=n, d=d, clusters=16, sigma=0.2, seed=34)

    def context():
        # Points, order, sets; snapshot and its distances; counts and offsets; room
        # for the edges (20 bytes each) of some of the points beside the reserve.
        base = n * (4 * d + 8 + 8 * k + 12) + n * k * 8 + n * 24 + n * k * 20 // 6
        return KnngContext(0, base * 8 // 7 + (1 << 20))

    with KnngContext(0) as a:
        a.load_points(pts)
        a.reset_sets(k)
        for r in range(2):
            a.run_rep(129, 1, 3000, seed=5, rep_index=r)
        before = a.sets()
    wants = []
    with context() as a:
        a.load_points(pts)
        a.reset_sets(k)
        a.set_sets(before)
        for _ in range(2):
            st = Stats()
            wants.append((a.refine(st), a.sets()))
            assert st.refine_join_launches >= 5 and st.refine_lost == 0
    monkeypatch.setenv("KNNG_JOIN_FAILS_IN", str(fails_in))
    with context() as a:
        a.load_points(pts)
        a.reset_sets(k)
        a.set_sets(before)
        if fails_in == 0:
            with pytest.raises(KnngError) as e:
                a.refine()
            assert e.value.status == 2 and "gave up" in str(e.value)
            assert _same_sets(before, a.sets())
        else:
            for changed, want in wants:
                st = Stats()
                assert a.refine(st) == changed
                assert _same_sets(want, a.sets())
                assert st.refine_join_launches == fails_in + 1 and st.refine_lost > 0


def test_a_repetition_that_found_no_room_leaves_nothing_half_made(knng_lib):
    """A budget that holds the points and sets but not a repetition's buffers: each
    try is refused anew, on the same context, and one that fits then runs."""
    n, d = 20_000, 64
    pts = workloads.gaussian_mixture(n=n, d=d, clusters=8, sigma=0.2, seed=35)
    few = default_params(k=10, reps=2, refine=0, max_leaf=129, max_leaf_odd=0, lloyd_iters=1, seed=3)
    many = default_params(k=64, reps=2, refine=0, max_leaf=129, max_leaf_odd=0, lloyd_iters=1, seed=3)
    with KnngContext(0) as ref:
        want = ref.build(pts, few)
    for room in (0, 100 << 10, 300 << 10, 500 << 10):
        with KnngContext(0, n * (4 * d + 8 + 8 * 64 + 12) + room) as ctx:
            for _ in range(3):
                with pytest.raises(KnngError) as e:
                    ctx.build(pts, many)
                assert e.value.status == 4
            ctx.load_points(pts)
            ctx.reset_sets(64)
            for _ in range(2):
                with pytest.raises(KnngError) as e:
                    ctx.run_rep(129, 1, 3000, seed=3, rep_index=0)
                assert e.value.status == 4
            assert np.array_equal(ctx.build(pts, few), want)


def test_sets_that_found_no_room_are_not_there(knng_lib):
    """A budget that holds some of the sets' arrays: the call is refused, stage calls
    then answer that there are no sets, and shorter lists that fit run."""
    n, d = 6_000, 64
    pts = workloads.gaussian_mixture(n=n, d=d, clusters=8, sigma=0.2, seed=36)
    with KnngContext(0) as ref:
        ref.load_points(pts)
        ref.reset_sets(10)
        ref.run_rep(129, 1, 3000, seed=3, rep_index=0)
        want = ref.sets()
    # The distances fit, then the ids, the sizes, the slots too; never the bounds.
    for part in (4 * 128, 8 * 128, 8 * 128 + 4, 8 * 128 + 8):
        with KnngContext(0, n * (4 * d + 8 + part) + n * 2) as ctx:
            ctx.load_points(pts)
            for _ in range(2):
                with pytest.raises(KnngError) as e:
                    ctx.reset_sets(128)
                assert e.value.status == 4
                for call in (lambda: ctx.run_rep(129, 1, 3000, seed=3, rep_index=0), ctx.refine,
                             lambda: ctx.process_leaves([0], [n])):
                    with pytest.raises(KnngError) as e:
                        call()
                    assert e.value.status in (1, 5)
                ctx.load_points(pts)  # brings back no sets, and is not refused for them
            ctx.reset_sets(10)
            ctx.run_rep(129, 1, 3000, seed=3, rep_index=0)
            assert _same_sets(want, ctx.sets())
