"""Distances of meshes whose squares leave FP32's normal range (coordinates from 1e-18 down to
where FP64's leave its own), and of tiny triangles in an ordinary mesh: FP64 equals the
oracle's minimum over all triangles bit for bit, mixed stays within its stated bound."""
import numpy as np
import pytest

from cybermeshgenerator_gb300 import workloads as W

pytestmark = pytest.mark.gpu

MESHES = {"ico": lambda: W.jittered_icosphere(2, 0.05, seed=1), "box": lambda: W.brick(1, 0.7, 0.3),
          "both": lambda: W.merge(W.brick(1, 1, 1), W.icosphere(1))}


def _check(cm, orc, p, t, **grid):
    plc = cm.PLC.from_arrays(p, t)
    exact = cm.voxelize_ex(plc, outputs=4 | 8, precision=cm.PREC_FP64, **grid)
    g = orc.grid(exact.corner, exact.spacing, exact.dims)
    d2, tri, reg = orc.sdf_brute(p, t, g)
    assert np.array_equal(np.abs(exact.sdf64).view(np.uint64), np.sqrt(d2).view(np.uint64))
    assert np.array_equal(exact.nearest_triangle, tri) and np.array_equal(exact.nearest_region, reg)
    mixed = cm.voxelize_ex(plc, outputs=4 | cm.OUT_ERROR_BOUND, precision=cm.PREC_MIXED, **grid)
    assert np.all(np.abs(np.abs(mixed.sdf64) - np.sqrt(d2)) <= mixed.error_bound.astype(np.float64))


@pytest.mark.parametrize("mesh", sorted(MESHES))
@pytest.mark.parametrize("power", [-150, -70, -44, -38, -32, -27, -26, -25, -24, -23, -22, -21, -20, -19, -18, -16, 18])
def test_scaled_mesh(cm, orc, mesh, power):
    p, t = MESHES[mesh]()
    _check(cm, orc, np.asarray(p, float) * 10.0 ** power, t, resolution=21, pad=1)


@pytest.mark.parametrize("size", [1e-6, 1e-12, 1e-18, 1e-19, 1e-20, 1e-22, 1e-30])
def test_tiny_triangles_in_an_ordinary_mesh(cm, orc, size):
    """Small bodies on a grid's cell centres, where no rounding hides their edges."""
    rng = np.random.default_rng(3)
    q, u = W.icosphere(0)
    bodies = [(size * (1 + k) * np.asarray(q) + at, u) for k, at in
              enumerate([np.zeros(3), np.array([0.25, 0, 0]), np.array([0, 0, 0.25])])]
    p, t = W.merge((rng.normal(size=(30, 3)) + 3.0, np.arange(30).reshape(-1, 3)), *bodies)
    _check(cm, orc, p, t.astype(np.int32), grid=((-0.625, -0.625, -0.625), 0.25, (7, 6, 5)))
