"""Results of voxelize() that a caller keeps: small ones own their memory, large ones hold
page-locked blocks up to a limit for all of them together and are copies beyond it, and none
changes when later calls run."""
import ctypes
import gc
import threading

import numpy as np
import pytest

from cybermeshgenerator_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _in_place(grid):
    return grid.base is not None and not grid.flags.owndata


@pytest.fixture()
def limit(cm, monkeypatch):
    gc.collect()  # grids of earlier tests count too

    def set_(n):
        monkeypatch.setattr(cm, "_KEEP_BYTES", n, raising=False)
    return set_


def test_small_grids_are_the_callers_own(cm):
    plc = cm.PLC.from_arrays(*W.jittered_icosphere(1, 0.02, seed=1))
    held = [cm.voxelize(plc, 4 + k % 10, mode, 1).grid for k in range(64) for mode in ("sdf", "occupancy")]
    for g in held:
        assert g.nbytes <= 16 << 10 and g.flags.owndata and g.base is None


def test_a_block_is_no_larger_than_twice_its_grid_and_64_KiB(cm):
    """Small grids after large ones, kept: what they lock by the library's own count."""
    from cybermeshgenerator_gb300 import _lib
    L = _lib.load()
    gc.collect()
    big = cm.PLC.from_arrays(*W.jittered_icosphere(2, 0.02, seed=5))
    for r in (40, 90, 60, 30):
        cm.voxelize(big, r, "sdf", 1)  # idle blocks of many sizes
    err = ctypes.create_string_buffer(256)
    held, room = [], 0
    for r in range(12, 40):
        out = ctypes.c_void_p()
        assert L.cmg_plc_voxelize_xyz(big._handle, r, 1, 1, ctypes.byref(out), err, 256) == 0
        dims = [ctypes.c_int() for _ in range(3)]
        L.cmg_voxels_dims(out.value, *(ctypes.byref(d) for d in dims))
        room += 2 * 4 * int(np.prod([d.value for d in dims])) + (64 << 10)
        assert L.cmg_voxels_keep(out.value, room) == 1, r
        held.append(out.value)
    for h in held:
        L.cmg_voxels_destroy(h)


def test_kept_grids_hold_a_bounded_amount(cm, limit):
    plc = cm.PLC.from_arrays(*W.jittered_icosphere(3, 0.02, seed=2))
    size = cm.voxelize(plc, 70, "sdf", 1).grid.nbytes
    want = cm.voxelize(plc, 70, "sdf", 1).grid.tobytes()
    limit(8 * size)
    held = [cm.voxelize(plc, 70, "sdf", 1).grid for _ in range(24)]
    n = sum(_in_place(g) for g in held)
    # a block holds its grid and may be as large again and 64 KiB more
    assert 8 * size // (2 * size + (64 << 10)) <= n <= 8
    for g in held:
        assert g.tobytes() == want and g.flags.c_contiguous and g.flags.writeable
    held[0][...] = 0
    assert all(g.tobytes() == want for g in held[1:])
    g = None
    del held
    gc.collect()
    assert _in_place(cm.voxelize(plc, 70, "sdf", 1).grid)  # their blocks went back
    limit(0)
    got = cm.voxelize(plc, 70, "sdf", 1).grid
    assert got.flags.owndata and got.tobytes() == want


def test_keeping_by_threads(cm, limit):
    plc = cm.PLC.from_arrays(*W.jittered_icosphere(2, 0.02, seed=3))
    want = {r: cm.voxelize(plc, r, "sdf", 1).grid.tobytes() for r in (60, 64, 68)}
    limit(10 << 20)
    bad = []

    def work(k):
        held = []
        for i in range(40):
            r = (60, 64, 68)[(i + k) % 3]
            held.append((r, cm.voxelize(plc, r, "sdf", 1).grid))
            if i % 7 == k:
                held = held[len(held) // 2:]
        bad.extend(r for r, g in held if g.tobytes() != want[r])

    ts = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad
    gc.collect()
    assert _in_place(cm.voxelize(plc, 64, "sdf", 1).grid)


def test_keep_counts_a_handle_once(cm):
    from cybermeshgenerator_gb300 import _lib
    L = _lib.load()
    gc.collect()
    plc = cm.PLC.from_arrays(*W.jittered_icosphere(1, 0.02, seed=4))
    err = ctypes.create_string_buffer(256)
    h = []
    for _ in range(2):
        out = ctypes.c_void_p()
        assert L.cmg_plc_voxelize(plc._handle, 40, 1, 1, ctypes.byref(out), err, 256) == 0
        h.append(out.value)
    assert L.cmg_voxels_keep(None, 1 << 40) == 0
    assert L.cmg_voxels_keep(h[0], 0) == 0
    assert L.cmg_voxels_keep(h[0], 1 << 40) == 1 and L.cmg_voxels_keep(h[0], 0) == 1
    assert L.cmg_voxels_keep(h[1], 0) == 0
    L.cmg_voxels_destroy(h[0])
    assert L.cmg_voxels_keep(h[1], 64 << 20) == 1  # (one grid's block)
    L.cmg_voxels_destroy(h[1])
