"""Which stage kernel a lattice takes (stage_parts, measured figures beside it): the borders of the
rule for an ideal fluid, with shear, and with shear and bulk (tests/stage_parts_check.cu, built with
nvcc and run on the CPU)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "gpu-vh_b200", "csrc")


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="nvcc not found")
def test_stage_parts(tmp_path):
    exe = tmp_path / "stage_parts_check"
    subprocess.run(["nvcc", "-std=c++17", "-I", CSRC, "-o", str(exe), os.path.join(HERE, "stage_parts_check.cu")],
                   check=True, timeout=600)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
