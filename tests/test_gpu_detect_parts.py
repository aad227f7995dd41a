"""Self-intersections that leave more pairs to the exact tests than are listed at once: a stack
of coplanar, overlapping triangles (no certificate decides a coplanar pair, and coplanar
pairs do not cross) with some that go through it. The search takes its cells in parts; the
pairs among a sample of the triangles equal the oracle's for the sample."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3000, 50000])
def test_coplanar_stack(cm, orc, n):
    rng = np.random.default_rng(n)
    flat = np.round(rng.uniform(0, 1, (n, 1, 2)) * 64) / 256 + np.round(rng.uniform(-1, 1, (n, 3, 2)) * 64) / 64
    tri = np.concatenate([flat, np.full((n, 3, 1), 0.25)], axis=2)
    through = rng.uniform(-0.3, 0.6, (40, 3, 3))
    tri = np.concatenate([tri, through])[rng.permutation(n + 40)]
    pts, tris = tri.reshape(-1, 3), np.arange(3 * len(tri), dtype=np.int32).reshape(-1, 3)
    got = cm.self_intersections(cm.PLC.from_arrays(pts, tris))[:, :2].astype(np.int64)
    assert np.array_equal(got, got[np.lexsort((got[:, 1], got[:, 0]))]) and (got[:, 0] < got[:, 1]).all()
    crossing = np.ptp(tri[:, :, 2], axis=1) > 0
    assert (crossing[got[:, 0]] | crossing[got[:, 1]]).all() and len(got) > 40 * n // 100
    ids = np.sort(np.concatenate([np.flatnonzero(crossing), rng.choice(np.flatnonzero(~crossing), 1500, replace=False)]))
    want = orc.self_intersections(pts, tris[ids])
    inside = np.isin(got, ids).all(1)
    assert np.array_equal(got[inside], ids[want])
