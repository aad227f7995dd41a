"""The sizing evaluation's cell-wise walk and its FP32 node search against the oracle:
query counts around a warp, several cells in a warp, lists longer than one step, queries
at the same distance from several nodes (left to the FP64 search), the global list beside
cells, and fields at offsets and scales where FP32 says little or nothing."""
import numpy as np
import pytest

from cybermeshgenerator_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,jitter,nq,scale,at", [
    (1, 0.0, 1, 1.0, 0.0), (1, 0.0, 3000, 1.0, 0.0), (56, 0.2, 3, 1.0, 0.0), (2, 0.3, 31, 1.0, 0.0), (3, 0.0, 33, 1.0, -5.0), (4, 0.3, 257, 1.0, 0.0),
    (9, 0.0, 5000, 1.0, 0.0), (9, 0.4, 5000, 1.0, 1e6), (7, 0.3, 3000, 1e-30, 0.0), (7, 0.3, 3000, 1e30, 1e30),
    (5, 0.2, 3000, 1e45, 0.0), (5, 0.2, 3000, 1e-45, 0.0), (6, 0.3, 4000, 1.0, 1e12)])
def test_field_equals_oracle(cm, orc, n, jitter, nq, scale, at):
    rng = np.random.default_rng(17 * n + nq)
    P, T = W.kuhn_tet_mesh(n, jitter, seed=n)
    Q = W.sizing_queries(P, T, nq, seed=nq)
    # outside, over cell centres and nodes (equal distances), and inside a hole of tets
    k = max(1, nq // 8)
    sym = (rng.integers(0, 2 * n + 1, size=(k, 3)) * 0.5) / n
    sym[:, rng.integers(0, 3)] = rng.choice([-0.25, 1.25], size=k)
    Q = np.vstack([Q, sym, sym + rng.normal(size=sym.shape) * 1e-9])
    T = T[rng.random(len(T)) < 0.9] if n > 2 else T
    P, Q = P * scale + at, Q * scale + at
    # long cell lists: many thin copies over the same nodes, out of order
    if n == 4:
        T = np.vstack([T[rng.permutation(len(T))]] * 9).astype(np.int32)
    S = rng.uniform(0.05, 1.0, len(P))
    f = cm.SizingField(P, T, S, 0.5)
    got, which = f.eval(Q, which=True)
    want, wwhich = orc.sizing(P, T, S, 0.5, Q)
    assert np.array_equal(got.view(np.uint64), np.asarray(want).view(np.uint64))
    assert np.array_equal(which.astype(np.int64), wwhich)
