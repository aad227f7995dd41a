"""Self-intersections against every pair of the oracle's all-pairs answer, none taken out
beforehand. In general position the two are equal. Among triangles with coplanar and touching
parts, or flat to the rounding of a determinant, the orientation test that the oracle applies
to all pairs also names some whose boxes are apart (such triangles share no point); the
search, which looks at pairs with boxes that meet, leaves exactly these out."""
import numpy as np
import pytest

from test_gpu_detect_edges import CASES, _soup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,n,size,scale,at", CASES)
def test_every_pair(cm, orc, kind, n, size, scale, at):
    rng = np.random.default_rng(n)
    pts = (_soup(kind, n, size, rng) * scale + at).reshape(-1, 3)
    tris = np.arange(3 * n, dtype=np.int32).reshape(-1, 3)
    if kind == "lattice":
        pts, inv = np.unique(pts, axis=0, return_inverse=True)
        tris = inv.reshape(-1, 3).astype(np.int32)
    got = cm.self_intersections(cm.PLC.from_arrays(pts, tris))[:, :2].astype(np.int64)
    want = orc.self_intersections(pts, tris)
    if kind in ("loose", "large"):
        assert np.array_equal(got, want)
        return
    found = set(map(tuple, got.tolist()))
    every = set(map(tuple, want.tolist()))
    assert found <= every and len(found) == len(got)
    for a, b in every - found:
        A, B = pts[tris[a]], pts[tris[b]]
        assert (A.max(0) < B.min(0)).any() or (B.max(0) < A.min(0)).any()
    assert len(every - found) == {1500: 470, 700: 12, 800: 8}[n]
