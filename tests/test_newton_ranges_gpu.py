"""Primitive recovery over the whole range of energies: the fast solves of the stage kernels
cover guesses and iterates in [1/16, 2^14) fm^-4, dilute guesses (e <= 0.1) take the closed form,
the rest the general iteration. A line of cells whose energy grows by 15% a cell from 2e-3 to
1e6 fm^-4 crosses every border within a stencil; each cell is compared with the oracle at its own
scale."""
import numpy as np
import pytest

import gvh
import oracle
from helpers import f32

pytestmark = pytest.mark.gpu

# per cell, relative: the solver's bar of the parity tests (QCD), rounding (conformal)
TOL = {False: 1e-9, True: 1e-12}


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("flow", [0.0, 0.4, -2.0])
@pytest.mark.parametrize("conformal", [False, True], ids=["qcd", "conformal"])
def test_recovery_from_dilute_to_dense(conformal, flow, axis):
    n = [2, 2, 2]
    n[axis] = 144
    kw = dict(nx=n[0], ny=n[1], nz=n[2], dx=1.0, dy=1.0, dz=1.0, dt=0.002, etabar=0.2, theta=1.8,
              conformal=conformal, shear=True, bulk=not conformal)
    G, O = gvh.Lattice(**kw), oracle.OracleLattice(**kw)
    shape = (G.ncz, G.ncy, G.ncx)
    at = np.arange(shape[2 - axis]) - 2
    e = f32(2e-3 * 1.15 ** at)
    e = np.broadcast_to(e.reshape([-1 if m == 2 - axis else 1 for m in range(3)]), shape)
    u = [np.zeros(shape) for _ in range(3)]
    u[axis] = np.full(shape, float(np.float32(flow)))
    ut = np.sqrt(1 + u[0] ** 2 + u[1] ** 2 + 0.6 ** 2 * u[2] ** 2)
    prim = {k: np.ascontiguousarray(v).reshape(-1) for k, v in dict(e=e, ut=ut, ux=u[0], uy=u[1], un=u[2]).items()}
    G.set_primitive(prim)
    O.set_primitive(prim)
    G.step(0.6, kw["dt"])
    O.step(0.6, kw["dt"])
    sg, so = G.get_state(), O.get_state()
    for k in ("e", "p", "ttt", "ut"):
        a, b = G.interior(sg[k]), O.interior(so[k])
        assert np.isfinite(a).all()
        assert np.max(np.abs(a - b) / np.abs(b)) <= TOL[conformal], k
