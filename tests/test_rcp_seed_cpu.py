"""The reciprocal under the branch-free division (lare_div.cuh), compiled as
host code: correctly rounded from every seed within its stated bound."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="nvcc not present")
def test_reciprocal_from_any_seed_in_bound(tmp_path):
    exe = str(tmp_path / "rcp_seed")
    r = subprocess.run(["nvcc", "-O2", "-std=c++17", "-Xcompiler", "-ffp-contract=off",
                        "-I", os.path.join(ROOT, "sams_b200", "csrc"),
                        os.path.join(ROOT, "tests", "cpp", "rcp_seed.cu"), "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and '"bad": 0' in r.stdout, r.stdout + r.stderr
