"""The per-side double sums of one Lloyd iteration at the edges of the sums
kernel's tiles and groups, against sums made one point at a time."""
from __future__ import annotations

import numpy as np
import pytest

from sigmod23ann_b200 import KnngContext

pytestmark = pytest.mark.gpu

F = np.float32


def _points(n: int, d: int, trues: int, seed: int) -> tuple[np.ndarray, np.ndarray]:
    """n points whose side is the sign of dim 1; magnitudes from subnormal to
    2^20, signed zeros among them."""
    rng = np.random.default_rng(seed)
    pts = (rng.standard_normal((n, d)) * np.exp2(rng.integers(-20, 20, (n, d)))).astype(F)
    pts[rng.random((n, d)) < 0.1] = F(-0.0)
    pts[rng.random((n, d)) < 0.1] = F(1e-42)
    side = np.zeros(n, bool)
    side[rng.permutation(n)[:trues]] = True
    pts[:, 1] = np.where(side, F(1e9), F(-1e9))
    return pts, side


def _centre(rows: np.ndarray) -> np.ndarray:
    """Mean of the rows: doubles added in order, then rounded to float."""
    acc = np.zeros(rows.shape[1], np.float64)
    for r in rows:
        acc = acc + r.astype(np.float64)
    return (acc / len(rows)).astype(F)


def _lloyd(ctx: KnngContext, pts: np.ndarray, first: np.ndarray, second: np.ndarray):
    n = len(pts)
    ctx.load_points(pts)
    coefs, _, ok = ctx.lloyd([0], [n], [0, 0], np.zeros(0, np.uint32), first[None], second[None], 1)
    return coefs[0], int(ok[0])


@pytest.mark.parametrize("d", [64, 100, 128])
def test_sums_at_tile_edges(knng_lib, d):
    first, second = np.zeros(d, F), np.zeros(d, F)
    first[1], second[1] = F(1e9), F(-1e9)
    with KnngContext(0) as ctx:
        for n, trues in ((2, 1), (9, 8), (63, 17), (64, 32), (65, 64), (66, 1), (127, 8), (128, 120), (129, 63),
                         (256, 128), (321, 160), (700, 23)):
            pts, side = _points(n, d, trues, seed=n)
            c1, c2 = _centre(pts[side]), _centre(pts[~side])
            want = c1 - F(0.5) * (c1 + c2)
            got, ok = _lloyd(ctx, pts, first, second)
            assert ok == 1
            assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), (d, n, trues)


def test_sums_with_infinities_and_nan(knng_lib):
    """A value that is not finite makes its dimension's centre infinite or NaN
    (its coefficient is then NaN) and leaves the others alone."""
    d, n = 100, 200
    pts, side = _points(n, d, 90, seed=5)
    first, second = np.zeros(d, F), np.zeros(d, F)
    first[1], second[1] = F(1e9), F(-1e9)
    first[7], second[7] = F(1), F(-1)  # +inf there keeps a point on the true side
    pts[np.flatnonzero(side)[3], 7] = F(np.inf)
    want = _centre(pts[side]) - F(0.5) * (_centre(pts[side]) + _centre(pts[~side]))
    with KnngContext(0) as ctx:
        got, ok = _lloyd(ctx, pts, first, second)
    assert ok == 1
    assert np.isnan(want[7]) and np.isnan(got[7])
    keep = np.arange(d) != 7
    assert np.array_equal(got[keep].view(np.uint32), want[keep].view(np.uint32))


def test_one_sided_set_is_reported(knng_lib):
    d, n = 100, 130
    pts, _ = _points(n, d, n, seed=6)
    first, second = np.zeros(d, F), np.zeros(d, F)
    first[1], second[1] = F(1e9), F(-1e9)
    with KnngContext(0) as ctx:
        _, ok = _lloyd(ctx, pts, first, second)
    assert ok == 0
