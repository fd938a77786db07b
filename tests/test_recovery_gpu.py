"""The building blocks of the primitive recovery on the device (recovery_check.cu, built here with
nvcc): quotient and square root against the IEEE operations, solves with divisors of any size."""
import os
import shutil
import subprocess

import pytest

from gvh import build as gbuild

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(shutil.which("nvcc") is None, reason="nvcc not found")]

HERE = os.path.dirname(os.path.abspath(__file__))


def test_quotient_and_root(tmp_path):
    exe = tmp_path / "recovery_check"
    arch = [f for f in gbuild.NVCC_FLAGS if f in ("-gencode", "-std=c++17") or f.startswith("arch=")]
    subprocess.run(["nvcc", *arch, "-I", gbuild.CSRC, "-o", str(exe), os.path.join(HERE, "recovery_check.cu")],
                   check=True, timeout=600)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
