"""The ops' division (FastDiv, lare_device.cuh), compiled as host code: on the
straight path, with the IEEE bits, over the scales it states."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="nvcc not present")
def test_division_takes_its_whole_range_of_scales(tmp_path):
    exe = str(tmp_path / "div_scales")
    r = subprocess.run(["nvcc", "-O2", "-std=c++17", "-Xcompiler", "-ffp-contract=off",
                        "-I", os.path.join(ROOT, "include"), "-I", os.path.join(ROOT, "sams_b200", "csrc"),
                        os.path.join(ROOT, "tests", "cpp", "div_scales.cu"), "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and '"bad": 0' in r.stdout, r.stdout + r.stderr
