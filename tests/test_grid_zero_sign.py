"""The grid's corner where the points' least coordinates are zeros of both signs: the
reference keeps the first least value in the points' order, so the corner of a grid
without padding has that zero's sign (CPU: cmg_plc_grid)."""
import numpy as np
import pytest


def _first_least(points):
    lo = points[0].copy()
    for p in points[1:]:
        lo = np.where(p < lo, p, lo)
    return lo


@pytest.mark.parametrize("n", [2, 7, 8, 9, 15, 16, 17, 31, 100])
def test_corner_keeps_the_first_zero(cm, n):
    rng = np.random.default_rng(n)
    for _ in range(40):
        P = np.ones((n, 3))
        # some coordinates zero, of either sign; one cube edge per axis, so that the extents
        # are whole cells and the corner is the least point itself
        P[rng.random((n, 3)) < 0.6] = 0.0
        P = np.where((rng.random((n, 3)) < 0.5) & (P == 0.0), -0.0, P)
        P[0] = 1.0
        P[n - 1] = np.where(P[n - 1] == 1.0, -0.0, P[n - 1])
        corner, spacing, dims = cm.plc_grid(cm.PLC.from_arrays(P, [[0, 0, n - 1]]), 4, 0)
        assert spacing == 0.25 and dims == (4, 4, 4)
        want = _first_least(P)
        assert np.array_equal(corner, want) and np.array_equal(np.signbit(corner), np.signbit(want))
