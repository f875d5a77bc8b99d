"""A set's entries sorted in registers, four a lane, for the refinement's lists
and the result: capacities around the lanes' runs and the words of the marks,
full and partly filled sets."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import assert_sets_equal
from sigmod23ann_b200 import KnngContext, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 3, 4, 31, 33, 64, 97, 100, 127, 128])
@pytest.mark.parametrize("leaf", [30, 200])
def test_lists_and_results_equal_the_oracle(oracle_lib, knng_lib, k, leaf):
    """Buckets below 30 points leave sets of more entries partly filled (their
    empty slots repeat an id); the second pass also marks the entries that the
    first one's lists had."""
    pts = workloads.gaussian_mixture(n=700, d=64, clusters=6, sigma=0.2, seed=k)
    o = oracle_lib.Oracle(pts, k=k, rng_mode=1, seed=5)
    o.rep(1, leaf, 0)
    with KnngContext(0) as ctx:
        ctx.load_points(pts)
        ctx.reset_sets(k)
        ctx.run_rep(leaf, 1, 3000, 5, 0)
        for i in range(2):
            assert ctx.refine() == o.refine(), i
            assert_sets_equal(ctx.sets(), o.sets(), f"k {k} pass {i}")
        ids, dist = ctx.finalize(want_dists=True)
    want_ids, want = o.finalize()
    np.testing.assert_array_equal(ids, want_ids)
    np.testing.assert_array_equal(dist.view(np.uint32), want.view(np.uint32))
