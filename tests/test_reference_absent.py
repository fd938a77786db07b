"""Tests that run the reference's own build skip where it is not built, and only then: any other
missing file still fails."""
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))

CHILD = """
import oracle

LAT = dict(nx=2, ny=2, nz=2, dx=0.1, dy=0.1, dz=0.1, dt=0.01, etabar=0.2, theta=2.0, conformal=True, shear=True,
           bulk=False)

def test_needs_the_reference(monkeypatch, tmp_path):
    monkeypatch.setattr(oracle, "REF_DIR", str(tmp_path))
    oracle.RefLattice(**LAT)

def test_needs_another_file(tmp_path):
    open(tmp_path / "absent")
"""


def test_missing_reference_build_skips(tmp_path):
    (tmp_path / "test_child.py").write_text(CHILD)
    r = subprocess.run([sys.executable, "-m", "pytest", "-q", "-p", "conftest", "-p", "no:cacheprovider", "--rootdir",
                        str(tmp_path), "-rsf", str(tmp_path / "test_child.py")], cwd=tmp_path, capture_output=True,
                       text=True, timeout=300, env=dict(os.environ, PYTHONPATH=HERE))
    assert "1 failed, 1 skipped" in r.stdout, r.stdout
    assert "reference build libref_fp64_conf_shear.so not built" in r.stdout
