"""The one-pass boundary fill against the edge by edge one, compiled as host
code: random tables of the built-in conditions on grids from three cells up,
bit for bit, whatever the order of the points."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="nvcc not present")
def test_composed_fill_equals_edge_by_edge(tmp_path):
    exe = str(tmp_path / "bc_compose")
    r = subprocess.run(["nvcc", "-std=c++17", "-I", os.path.join(ROOT, "include"),
                        "-I", os.path.join(ROOT, "sams_b200", "csrc"),
                        os.path.join(ROOT, "tests", "cpp", "bc_compose.cu"), "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and '"bad": 0' in r.stdout, r.stdout + r.stderr
