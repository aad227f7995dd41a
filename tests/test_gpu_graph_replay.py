"""Graph replays of a batch whose points moved, through the C++ engine
(tests/cpp/test_graph_replay.cpp)."""
import os
import subprocess

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu


def test_replays_after_the_points_moved(cm, tmp_path):
    from cybermeshgenerator_gb300 import build
    lib = build.build()
    exe = str(tmp_path / "test_graph_replay")
    cuda = os.path.join(build._cuda_home(build._nvcc()), "include")
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-I", build.CSRC, "-I", cuda,
                        os.path.join(ROOT, "tests", "cpp", "test_graph_replay.cpp"), lib,
                        "-Wl,-rpath," + os.path.dirname(lib), "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
