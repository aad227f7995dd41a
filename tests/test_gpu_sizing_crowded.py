"""Sizing queries that crowd into one or a few cells: the counting sort's places, several
lanes of a warp to a cell, against the oracle."""
import numpy as np
import pytest

from cybermeshgenerator_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 255, 257, 5000])
@pytest.mark.parametrize("spots", [1, 2, 3, 40])
def test_crowded_queries(cm, orc, n, spots):
    P, T = W.kuhn_tet_mesh(6, 0.3, seed=6)
    rng = np.random.default_rng(n + spots)
    S = rng.uniform(0.05, 1.0, len(P))
    at = rng.uniform(-0.2, 1.2, size=(spots, 3))
    Q = at[rng.integers(0, spots, size=n)] + rng.choice([0.0, 1e-9], size=(n, 1)) * rng.normal(size=(n, 3))
    Q[rng.random(n) < 0.1] = 9.0  # outside the domain
    got, which = cm.SizingField(P, T, S, 0.5).eval(Q, which=True)
    want, wwhich = orc.sizing(P, T, S, 0.5, Q)
    assert np.array_equal(got.view(np.uint64), np.asarray(want).view(np.uint64))
    assert np.array_equal(which.astype(np.int64), wwhich)
