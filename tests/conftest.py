import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for p in (ROOT, os.path.join(ROOT, "gpu-vh_b200")):
    if p not in sys.path:
        sys.path.insert(0, p)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (B200); runs the CUDA path")


def _has_gpu():
    try:
        import torch
        return torch.cuda.is_available()
    except Exception:
        return False


def pytest_collection_modifyitems(config, items):
    if _has_gpu():
        return
    skip = pytest.mark.skip(reason="no CUDA device")
    for it in items:
        if "gpu" in it.keywords:
            it.add_marker(skip)


@pytest.hookimpl(wrapper=True)
def pytest_pyfunc_call(pyfuncitem):
    """A test that needs a build of the reference's own sources (oracle/_ref, made where the
    reference tree is present) skips where that build is absent."""
    import oracle

    try:
        return (yield)
    except FileNotFoundError as err:
        path = str(err.args[0])
        if not path.startswith(oracle.REF_DIR + os.sep):
            raise
        pytest.skip(f"reference build {os.path.basename(path)} not built (oracle/build_ref.py needs the reference tree)")
