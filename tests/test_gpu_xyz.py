"""voxelize()'s device-side array order against voxelize_ex's cells, at grids around the
32-cell tiles of the transposition, and calls whose lists outgrow what earlier calls left
in the device's workspace (they are sized and run again)."""
import numpy as np
import pytest

from cybermeshgenerator_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("resolution,pad,box", [(1, 0, (1, 1, 1)), (5, 1, (3, 1, 0.2)), (31, 0, (1, 0.99, 0.5)),
                                                (32, 0, (0.4, 1, 1)), (33, 2, (1, 0.03, 1)), (65, 1, (0.3, 0.8, 1))])
def test_order_of_voxelize(cm, resolution, pad, box):
    plc = cm.PLC.from_arrays(*W.brick(*box))
    for mode, field in (("occupancy", "occupancy"), ("sdf", "sdf32")):
        got = cm.voxelize(plc, resolution, mode, pad)
        ex = cm.voxelize_ex(plc, resolution=resolution, pad=pad, outputs=1 | 2)
        want = getattr(ex, field).reshape(ex.dims[::-1]).transpose(2, 1, 0)
        assert got.grid.shape == want.shape and got.grid.dtype == want.dtype
        assert got.grid.flags.c_contiguous and got.grid.flags.writeable
        assert np.array_equal(got.grid.view(np.uint8), np.ascontiguousarray(want).view(np.uint8))


def test_growing_and_shrinking_calls(cm):
    """The same meshes before and after larger ones give the same bits."""
    plcs = [cm.PLC.from_arrays(*W.jittered_icosphere(s, 0.02, seed=s)) for s in (0, 2, 4, 1, 5, 3)]
    first = [cm.voxelize(p, 20 + 9 * i, "sdf", 1).grid for i, p in enumerate(plcs)]
    occ = [cm.voxelize(p, 90 - 9 * i, "occupancy", 1).grid for i, p in enumerate(plcs)]
    for i, p in reversed(list(enumerate(plcs))):
        assert np.array_equal(cm.voxelize(p, 20 + 9 * i, "sdf", 1).grid, first[i])
        assert np.array_equal(cm.voxelize(p, 90 - 9 * i, "occupancy", 1).grid, occ[i])
    # an occupancy grid larger than any before it, in the first call that needs it
    p = cm.PLC.from_arrays(*W.brick(1, 0.7, 0.4))
    got = cm.voxelize(p, 420, "occupancy", 1).grid
    ex = cm.voxelize_ex(p, resolution=420, pad=1, outputs=1)
    assert np.array_equal(got, ex.occupancy.reshape(ex.dims[::-1]).transpose(2, 1, 0))
