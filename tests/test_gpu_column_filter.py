"""The column test's FP32 certificate against the oracle's occupancy, bit for bit: loose
triangles of all sizes, lattice vertices (ties by construction), flat and sliver triangles,
vertices far outside the grid, grids far from the origin and at extreme scales, rows that
end inside a CTA's 32 columns, and buckets of many chunks of one column."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _soup(kind, n, dims, rng):
    """n triangles in cell units over a grid of dims cells with its corner at 0."""
    d = np.asarray(dims, float)
    c = rng.uniform(-1, 1.0, (n, 1, 3)) * 0.05 * d + rng.uniform(0, 1, (n, 1, 3)) * d
    size = 10.0 ** rng.uniform(-1.5, 0.7, (n, 1, 1))
    v = c + size * rng.normal(size=(n, 3, 3))
    if kind == "lattice":
        v = np.round(2 * v) / 2
    elif kind == "sliver":
        v[:, 2] = v[:, 0] + (v[:, 1] - v[:, 0]) * rng.uniform(0, 1, (n, 1)) + 1e-6 * rng.normal(size=(n, 3))
        v[: n // 3, :, 2] = v[: n // 3, :1, 2]           # horizontal
        v[n // 3: n // 2, 2, :2] = v[n // 3: n // 2, 0, :2]  # vertical
    elif kind == "far":
        v[::7, 1] *= 1e9
        v[::5, 2] = d / 2 + 300 * (v[::5, 2] - d / 2)
    return v.reshape(-1, 3)


CASES = [("loose", 400, (33, 17, 20), 1.0, 0.0), ("loose", 3000, (64, 5, 300), 0.037, 11.0),
         ("loose", 20000, (129, 40, 31), 1.0, -3.0), ("lattice", 2500, (40, 31, 24), 0.25, 0.5),
         ("lattice", 60, (32, 32, 32), 1.0, 0.0), ("sliver", 1500, (31, 32, 33), 3.0, 7.0),
         ("far", 300, (45, 12, 16), 1.0, 0.0), ("loose", 900, (1, 1, 70), 1.0, 2.0),
         ("loose", 5000, (2, 1, 3), 1.0, 0.0), ("loose", 600, (32, 9, 16), 1.0, 1e9),
         ("loose", 600, (20, 9, 16), 1e-12, 1e-12), ("loose", 600, (20, 9, 16), 1e25, 1e24),
         ("loose", 600, (20, 9, 16), 1e-30, 0.0), ("loose", 600, (20, 9, 16), 1e-9, 1.0)]


@pytest.mark.parametrize("mode", ["compat", "exact"])
@pytest.mark.parametrize("kind,n,dims,h,at", CASES)
def test_occupancy_equals_oracle(cm, orc, kind, n, dims, h, at, mode):
    import oracle as O
    rng = np.random.default_rng(n + dims[0])
    pts = np.ascontiguousarray(_soup(kind, n, dims, rng) * h + at)
    tris = np.arange(3 * n, dtype=np.int32).reshape(-1, 3)
    corner = np.full(3, at)
    if kind != "lattice":
        corner = corner + h * np.array([0.1, -0.3, 0.2])
    got = cm.voxelize_ex(cm.PLC.from_arrays(pts, tris), grid=(corner, h, dims), outputs=cm.OUT_OCCUPANCY,
                         predicates=cm.PRED_COMPAT if mode == "compat" else cm.PRED_EXACT).occupancy
    want, _ = orc.occupancy(pts, tris, orc.grid(corner, h, dims), O.COMPAT if mode == "compat" else O.EXACT)
    assert np.array_equal(got, want)
