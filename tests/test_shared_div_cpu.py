"""Division without branches (lare_div.cuh), compiled as host code:
the bits of the IEEE reciprocal and quotient wherever its conditions hold."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="nvcc not present")
def test_shared_division_is_ieee(tmp_path):
    exe = str(tmp_path / "shared_div")
    r = subprocess.run(["nvcc", "-O2", "-std=c++17", "-Xcompiler", "-ffp-contract=off",
                        "-I", os.path.join(ROOT, "sams_b200", "csrc"),
                        os.path.join(ROOT, "tests", "cpp", "shared_div.cu"), "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and '"bad": 0' in r.stdout, r.stdout + r.stderr
