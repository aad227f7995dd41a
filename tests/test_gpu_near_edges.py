"""The warp-per-sub-brick distance kernel (csrc/sdf_near.cu) where its parts have edges:
grids that end inside a sub-brick or hold a single cell, z-slabs, triangle counts around
a warp's 32 and a step's 128 list entries, a vertex of high valence (more near-ties than
are kept at once), triangles of very different sizes, repeated and degenerate ones. FP64
equals the plain kernel (every candidate in FP64) bit for bit; mixed stays within its
stated bound, its band equals FP64."""
import numpy as np
import pytest

from cybermeshgenerator_gb300 import workloads as W

pytestmark = pytest.mark.gpu

OUTS = 1 | 2 | 4 | 8


def _cone(n):
    """A closed double cone: two apexes of valence n."""
    a = 2 * np.pi * np.arange(n) / n
    ring = np.stack([np.cos(a), np.sin(a), 0.3 * np.ones(n)], 1)
    p = np.concatenate([ring, [[0.1, 0.0, 1.0], [0.0, 0.1, -0.6]]])
    i, j = np.arange(n), (np.arange(n) + 1) % n
    return p, np.concatenate([np.stack([i, j, np.full(n, n)], 1), np.stack([j, i, np.full(n, n + 1)], 1)]).astype(np.int32)


def _mixed_sizes():
    """One large triangle under a cloud of small spheres, repeats and degenerate triangles."""
    p, t = W.merge(W.icosphere(2), (np.array([[-9, -9, -1.5], [9, -9, -1.5], [0, 12, -1.4]], float),
                                    np.array([[0, 1, 2]], np.int32)))
    q, u = W.icosphere(1)
    p, t = W.merge((p, t), (0.05 * q + [1.4, 0, 0], u), (0.02 * q + [0, 1.5, 0.3], u))
    t = np.concatenate([t, t[:7], [[0, 1, 1], [2, 2, 2]], np.array([[0, 1, 2]])])
    return p, t.astype(np.int32)


def _soup(n):
    rng = np.random.default_rng(n)
    p = rng.normal(size=(n, 1, 3)) + 0.2 * rng.normal(size=(n, 3, 3))
    return p.reshape(-1, 3), np.arange(3 * n, dtype=np.int32).reshape(-1, 3)


MESHES = {"cone40": lambda: _cone(40), "cone600": lambda: _cone(600), "sizes": _mixed_sizes,
          **{f"soup{n}": (lambda n=n: _soup(n)) for n in (1, 31, 32, 33, 127, 128, 129, 160, 500)}}


def _bits(a):
    return np.ascontiguousarray(a).view(np.uint8)


@pytest.mark.parametrize("dims", [(1, 1, 1), (3, 4, 5), (17, 15, 2), (33, 18, 21)])
@pytest.mark.parametrize("mesh", sorted(MESHES))
def test_edges(cm, mesh, dims):
    p, t = MESHES[mesh]()
    h = 2.6 / max(dims)
    kw = dict(grid=((-1.31, -1.27, -1.22), h, dims), outputs=OUTS)
    plc = cm.PLC.from_arrays(p, t)
    plain = cm.voxelize_ex(plc, precision=cm.PREC_FP64_PLAIN, **kw)
    exact = cm.voxelize_ex(plc, precision=cm.PREC_FP64, **kw)
    names = ("occupancy", "sdf32", "sdf64", "nearest_triangle", "nearest_region")
    for n in names:
        assert np.array_equal(_bits(getattr(exact, n)), _bits(getattr(plain, n))), n
    if dims[2] > 2:  # a slab that starts and ends inside sub-bricks
        z0, z1 = 1, dims[2] - 1
        cut = slice(z0 * dims[0] * dims[1], z1 * dims[0] * dims[1])
        slab = cm.voxelize_ex(plc, precision=cm.PREC_FP64, layers=(z0, z1), **kw)
        for n in names:
            assert np.array_equal(_bits(getattr(slab, n)), _bits(getattr(plain, n)[cut])), n
    for band in (0.0, 1.0, 1e9):
        m = cm.voxelize_ex(plc, precision=cm.PREC_MIXED, band=band,
                           **{**kw, "outputs": OUTS | cm.OUT_ERROR_BOUND})
        assert np.array_equal(m.occupancy, plain.occupancy)
        assert np.all(np.abs(m.sdf64 - plain.sdf64) <= m.error_bound.astype(np.float64))
        fine = m.error_bound == 0
        assert fine.sum() == m.stats["band_cells"] and (band < 1e9 or fine.all())
        assert np.array_equal(_bits(m.sdf64[fine]), _bits(plain.sdf64[fine]))
        assert np.array_equal(m.nearest_triangle[fine], plain.nearest_triangle[fine])
