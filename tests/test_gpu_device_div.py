"""The branch-free division on the device itself (its host form starts from
another seed): 32 million operands against the IEEE operations."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_device_division_is_ieee(tmp_path):
    from sams_b200 import build
    exe = str(tmp_path / "device_div")
    r = subprocess.run([build.nvcc(), *build.NVCC_FLAGS, "-I", os.path.join(ROOT, "include"), "-I", os.path.join(ROOT, "sams_b200", "csrc"),
                        os.path.join(ROOT, "tests", "cpp", "device_div.cu"), "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and '"bad": 0' in r.stdout, r.stdout + r.stderr
