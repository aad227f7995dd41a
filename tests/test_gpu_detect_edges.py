"""The FP32 middle phase of the self-intersection search against the oracle's all-pairs
restatement: loose triangles from sparse to everything-crosses-everything (both of the
search's lists run over), lattice corners (coplanar and touching pairs), flat and sliver
triangles, one triangle over all cells, and coordinates at extreme scales and offsets."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _soup(kind, n, size, rng):
    v = rng.uniform(0, 1, (n, 1, 3)) + size * rng.normal(size=(n, 3, 3))
    if kind == "lattice":
        v = np.round(v * 12) / 12
    elif kind == "flat":
        v[..., 2] *= 1e-9
        v[: n // 4, 2] = 0.5 * (v[: n // 4, 0] + v[: n // 4, 1])
    elif kind == "large":
        v[0] = [[-3, -2, 0.4], [4, -1, 0.5], [0, 5, 0.6]]
    return v


CASES = [("loose", 2, 0.5, 1.0, 0.0), ("loose", 3000, 0.01, 1.0, 0.0), ("loose", 1200, 0.2, 1.0, -4.0),
         ("loose", 1500, 2.0, 1.0, 0.0), ("lattice", 1500, 0.06, 1.0, 0.0), ("lattice", 700, 0.3, 0.25, 1.0),
         ("flat", 800, 0.05, 1.0, 0.0), ("large", 2000, 0.01, 1.0, 0.0), ("loose", 1000, 0.05, 1e-3, 1e7),
         ("loose", 1000, 0.05, 1e-85, 0.0), ("loose", 1000, 0.05, 1e-60, 0.0), ("loose", 1000, 0.05, 1e60, 0.0)]


@pytest.mark.parametrize("kind,n,size,scale,at", CASES)
def test_pairs_equal_oracle(cm, orc, kind, n, size, scale, at):
    rng = np.random.default_rng(n)
    pts = (_soup(kind, n, size, rng) * scale + at).reshape(-1, 3)
    tris = np.arange(3 * n, dtype=np.int32).reshape(-1, 3)
    if kind == "lattice":   # shared corners too
        pts, inv = np.unique(pts, axis=0, return_inverse=True)
        tris = inv.reshape(-1, 3).astype(np.int32)
    got = cm.self_intersections(cm.PLC.from_arrays(pts, tris))
    want = orc.self_intersections(pts, tris)
    # the search reports pairs whose boxes meet (coplanar decisions of the orientation test
    # can name others, among degenerate and touching triangles)
    lo, hi = pts[tris].min(1), pts[tris].max(1)
    a, b = want[:, 0], want[:, 1]
    want = want[((lo[a] <= hi[b]) & (lo[b] <= hi[a])).all(1)]
    assert np.array_equal(got[:, :2].astype(np.int64), want)
