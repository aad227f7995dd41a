"""Facets that a PLC has no memory for: the call answers CMG_ERR_INTERNAL and leaves the PLC
as it was (its triangles, and those added later). CPU; the memory is withheld by an
address-space limit in a process of its own."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

PROG = r"""
import ctypes, os, resource, sys
import numpy as np
import cybermeshgenerator_gb300 as cm
from cybermeshgenerator_gb300 import _lib
L = _lib.load()
first, extra = int(sys.argv[1]), int(sys.argv[2])
page = os.sysconf("SC_PAGE_SIZE")
used = lambda: int(open("/proc/self/statm").read().split()[0]) * page

def add(plc, t):
    return L.cmg_plc_add_triangles(plc._handle, t.ctypes.data_as(_lib.c_int_p), len(t), 0)

big = np.tile(np.array([[0, 1, 2]], np.int32), (extra, 1))
small = np.array([[0, 1, 2], [2, 1, 3]], np.int32)
plc = cm.PLC().add_points(np.eye(4, 3))
if first:
    assert add(plc, small) == 0
add(cm.PLC(), big[:500000])  # whatever the first large allocation sets up
# room for the 12 bytes of indices per triangle, not for the 8 of offsets after them
resource.setrlimit(resource.RLIMIT_AS, (used() + 12 * extra + 4 * extra, resource.RLIM_INFINITY))
st = add(plc, big)
resource.setrlimit(resource.RLIMIT_AS, (resource.RLIM_INFINITY, resource.RLIM_INFINITY))
assert st == 6, st
want = small[: 2 * first]
assert np.array_equal(plc.triangles, want.reshape(-1, 3)), len(plc.triangles)
plc.add_facet([0, 1, 3])
assert np.array_equal(plc.triangles, np.vstack([want.reshape(-1, 3), [[0, 1, 3]]]))
plc.add_facet([0, 1, 2, 3])
assert len(plc.triangles) == len(want) + 3
"""


@pytest.mark.parametrize("first", [0, 1])
def test_facets_without_memory_leave_the_plc(cm, first):
    r = subprocess.run([sys.executable, "-c", PROG, str(first), str(16 << 20)], cwd=ROOT, text=True,
                       capture_output=True, timeout=300, env={**os.environ, "CUDA_VISIBLE_DEVICES": ""})
    assert r.returncode == 0, r.stderr
