"""The mixed path's bulk pressure keeps its bits: one QCD step of a small lattice, alone and in a
batch, against values stored from the build before the recoveries were paired
(tests/golden/mixed_bulk_pressure.npz). The two differ from one another in one rounding of
zeta/s (bulk_zeta_over_s), and 1e-8 of Pi is what a solve that wanders can turn into another event."""
import os

import numpy as np
import pytest

import gvh
from helpers import rich_state

pytestmark = pytest.mark.gpu

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "mixed_bulk_pressure.npz")
SHAPE = (12, 9, 5)


def pressures():
    L = gvh.Lattice(*SHAPE, 0.3, 0.3, 0.3, 0.01, 0.16, precision="mixed", tau0=0.5)
    prim = rich_state(L, seed=5, spacing=0.5)
    L.set_primitive(prim)
    L.step(0.5, 0.01)
    B = gvh.Batch(8 << 20, precision="mixed")
    event = B.add_event(*SHAPE, 0.3, 0.3, 0.3, 0.01, 0.16, prim, tau0=0.5)
    B.step(1)
    return {"alone": L.interior(L.get_state()["Pi"]), "batch": L.interior(B.get_state(event)["Pi"])}


def test_mixed_bulk_pressure_keeps_its_bits():
    want = np.load(GOLDEN)
    for name, got in pressures().items():
        np.testing.assert_array_equal(got, want[name], err_msg=name)
