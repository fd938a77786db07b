"""Settings at the ends of what the entry points accept."""
import numpy as np
import pytest

import gvh
import oracle
from helpers import rel_err, rich_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(9, 8, 7), (44, 43, 42)], ids=["small", "wave"])
@pytest.mark.parametrize("conformal", [False, True], ids=["qcd", "conformal"])
def test_infinite_shear_viscosity(conformal, shape):
    """eta/s = infinity switches the relaxation of pi off (T / eta/s = 0); the rest of the step stays
    as it is. Tolerances as the parity tests'."""
    nx, ny, nz = shape
    kw = dict(nx=nx, ny=ny, nz=nz, dx=0.3, dy=0.3, dz=0.3, dt=0.01, etabar=np.inf, theta=2.0, conformal=conformal,
              shear=True, bulk=not conformal)
    G, O = gvh.Lattice(**kw), oracle.OracleLattice(**kw)
    prim = rich_state(G, seed=21)
    G.set_primitive(prim)
    O.set_primitive(prim)
    for n in range(2):
        G.step(0.5 + 0.01 * n, 0.01)
        O.step(0.5 + 0.01 * n, 0.01)
    assert G.status() == 0
    sg, so = G.get_state(), O.get_state()
    for k in G.field_names:
        assert np.isfinite(so[k]).all()
        assert rel_err(G.interior(sg[k]), O.interior(so[k])) <= (1e-12 if conformal else 1e-9), k
