"""The tilings of the fused kernels (lare_march.cuh), compiled as host code:
every own point of each phase falls to exactly one thread over grids from one
cell to several hundred, thin, square and long."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="nvcc not present")
def test_tilings_cover_every_point_once(tmp_path):
    exe = str(tmp_path / "march_tiles")
    r = subprocess.run(["nvcc", "-std=c++17", "-I", os.path.join(ROOT, "include"),
                        "-I", os.path.join(ROOT, "sams_b200", "csrc"),
                        os.path.join(ROOT, "tests", "cpp", "march_tiles.cu"), "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and '"bad": 0' in r.stdout, r.stdout + r.stderr
