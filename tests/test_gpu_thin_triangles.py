"""Triangles for which the reference's distance is no number (repeated corners: 0 / 0) or not the
distance (collinear corners, slivers of 1e-15): it skips the first kind and takes the second
as computed. FP64 distances, nearest triangles and regions equal the oracle's minimum over
all triangles, also where such a triangle lies nearest and alone; mixed precision stays within
its bound, beyond the band too. Single calls, batches, graph replays, and calls with and
without such triangles in turn."""
import numpy as np
import pytest

from cybermeshgenerator_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _soup(seed):
    """Lattice triangles, many of them repeated or collinear, and slivers; scaled and turned."""
    rng = np.random.default_rng(seed)
    n = int(rng.integers(3, 300))
    p = np.round(rng.uniform(-1, 1, (n, 3, 3)) * 8) / 8
    k = rng.integers(0, 6, n)
    p[k == 0, 1] = p[k == 0, 0]
    p[k == 1, 2] = p[k == 1, 1]
    p[k == 2, 2] = p[k == 2, 0]
    p[k == 3, 2] = p[k == 3, 0] + (p[k == 3, 1] - p[k == 3, 0]) * rng.choice([0.5, 0.25, 2.0, -1.0])
    p[k == 4, 2] += (p[k == 4, 1] - p[k == 4, 0]) * 0.25 - p[k == 4, 2] + p[k == 4, 0] + 1e-15 * rng.normal(size=(int((k == 4).sum()), 3))
    p = p.reshape(-1, 3)
    if seed % 2:
        p = p @ np.linalg.qr(rng.normal(size=(3, 3)))[0]
    return p * 10.0 ** rng.choice([0, -5, 4]), np.arange(3 * n, dtype=np.int32).reshape(-1, 3)


def _truth(orc, p, t, r):
    d2, tri, reg = orc.sdf_brute(p, t, orc.grid(r.corner, r.spacing, r.dims))
    return np.sqrt(d2), tri, reg


def _check_exact(r, truth):
    d, tri, reg = truth
    assert np.array_equal(np.abs(r.sdf64).view(np.uint64), d.view(np.uint64))
    assert np.array_equal(r.nearest_triangle, tri) and np.array_equal(r.nearest_region, reg)


def _check_mixed(r, truth):
    assert np.all(np.abs(np.abs(r.sdf64) - truth[0]) <= r.error_bound.astype(np.float64))


@pytest.mark.parametrize("seed", range(60))
def test_soups(cm, orc, seed):
    p, t = _soup(seed)
    plc = cm.PLC.from_arrays(p, t)
    kw = dict(resolution=3 + seed % 23, pad=seed % 4)
    r = cm.voxelize_ex(plc, outputs=4 | 8, **kw)
    truth = _truth(orc, p, t, r)
    _check_exact(r, truth)
    for band in (0.0, 1.0):
        _check_mixed(cm.voxelize_ex(plc, outputs=4 | 16, precision=1, band=band, **kw), truth)


@pytest.mark.parametrize("corners", [[[0.8, 0, 0], [0.8, 0, 0], [0.8, 0.3, 0]], [[0.8, 0, 0], [0.8, 0.3, 0], [0.8, 0.3, 0]],
                                     [[0.8, 0, 0], [0.8, 0.3, 0], [0.8, 0, 0]], [[0.8, 0, 0]] * 3,
                                     [[0.8, 0, 0], [0.8, 0.3, 0], [0.8, 0.15, 0]], [[0.8, 0, 0], [0.8, 0.3, 0], [0.8, 0.1, 1e-16]]])
@pytest.mark.parametrize("cells", [8, 40])
def test_one_beside_a_sphere(cm, orc, corners, cells):
    q, u = W.icosphere(2)
    p, t = W.merge((0.4 * np.asarray(q), u), (np.array(corners, float), np.array([[0, 1, 2]], np.int32)))
    t = t.astype(np.int32)
    plc, ball = cm.PLC.from_arrays(p, t), cm.PLC.from_arrays(0.4 * np.asarray(q), u)
    grid = dict(grid=((-0.5, -0.5, -0.5), 1.6 / cells, (cells, cells, cells)))
    clean = cm.voxelize_ex(ball, outputs=4, **grid).sdf64.copy()
    truth = None
    for _ in range(2):  # with and without it in turn
        r = cm.voxelize_ex(plc, outputs=4 | 8, **grid)
        truth = truth or _truth(orc, p, t, r)
        _check_exact(r, truth)
        assert np.array_equal(cm.voxelize_ex(ball, outputs=4, **grid).sdf64.view(np.uint64), clean.view(np.uint64))
        _check_mixed(cm.voxelize_ex(plc, outputs=4 | 16, precision=1, **grid), truth)
    b = cm.Batch([plc, ball], [16, 16], [1, 1], outputs=4 | 8, **grid)  # (a batch numbers its triangles through)
    for graph in (False, True, True):
        b.run(graph=graph).sync()
        _check_exact(b.result(0), truth)
        assert np.array_equal(b.result(1).sdf64.view(np.uint64), clean.view(np.uint64))
    m = cm.Batch([ball, plc], [16, 16], [1, 1], outputs=4 | 16, precision=1, **grid)
    _check_mixed(m.run().sync().result(1), truth)
