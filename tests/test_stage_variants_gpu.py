"""Every stage kernel (eight warps per 32 cells, four, two and one threads per cell) through what
only some lattices reach: the borders of the primitive recovery's fast forms, the bounds-checked
build with a partial last block, and the allocation-free step."""
import ctypes
import hashlib
import os
import subprocess
import sys

import numpy as np
import pytest

import gvh
import oracle
from gvh import build as gbuild
from helpers import f32, rel_err, rich_state
from test_zz_no_alloc import bound, stack

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)

RAMP = {8: (144, 2, 2), 4: (144, 100, 1), 2: (144, 16, 13), 1: (144, 24, 20)}
PHYSICS = {"qcd_bulk": dict(shear=True, bulk=True), "qcd_shear": dict(shear=True, bulk=False),
           "qcd_ideal": dict(shear=False, bulk=False)}


def ramp(L, flow):
    """e grows by 15% a cell along x from 2e-3 to 1e6 fm^-4 (across 1/16, 0.1 and 2^14); uniform in y, eta."""
    shape = (L.ncz, L.ncy, L.ncx)
    e = np.broadcast_to(f32(2e-3 * 1.15 ** (np.arange(L.ncx) - 2)), shape)
    ux = np.full(shape, float(np.float32(flow)))
    z = np.zeros(shape)
    return {k: np.ascontiguousarray(v).reshape(-1)
            for k, v in dict(e=e, ut=np.sqrt(1 + ux ** 2), ux=ux, uy=z, un=z).items()}


def after_ramp(cls, shape, physics, flow, **more):
    kw = dict(nx=shape[0], ny=shape[1], nz=shape[2], dx=1.0, dy=1.0, dz=1.0, dt=0.002, etabar=0.2, theta=1.8,
              conformal=False, **PHYSICS[physics], **more)
    L = cls(**kw)
    L.set_primitive(ramp(L, flow))
    L.step(0.6, 0.002)
    return L, {k: L.interior(v) for k, v in L.get_state().items()}


@pytest.mark.parametrize("flow", [0.0, 0.4, -2.0])
@pytest.mark.parametrize("physics", list(PHYSICS))
def test_recovery_borders_on_every_kernel(physics, flow):
    """FP64: each cell against the oracle at its own scale (test_newton_ranges_gpu.py's bar), and no
    kernel raises a status bit that another does not. Mixed: nothing varies along y and eta, so every
    kernel must give the same line, bit for bit."""
    _, line = after_ramp(oracle.OracleLattice, RAMP[8], physics, flow)
    status, mixed = {}, {}
    for parts, shape in RAMP.items():
        L, got = after_ramp(gvh.Lattice, shape, physics, flow)
        status[parts] = L.status()
        for k in ("e", "p", "ttt", "ut"):
            want = line[k][0, 0]
            assert np.isfinite(got[k]).all(), (parts, k)
            assert np.max(np.abs(got[k] - want) / np.abs(want)) <= 1e-9, (parts, k)
        M, got = after_ramp(gvh.Lattice, shape, physics, flow, precision="mixed")
        status[parts, "mixed"] = M.status()
        mixed[parts] = got
    assert len(set(status.values())) == 1 and not status[8] & gvh.GVH_STATUS_NAN, status
    for parts, got in mixed.items():
        for k, v in got.items():
            np.testing.assert_array_equal(v, np.broadcast_to(mixed[8][k][:1, :1], v.shape), err_msg=f"{parts} {k}")


# one lattice per kernel, the last block partial (32, 32, 64 and 128 cells a block)
RAGGED = {8: (21, 19, 17), 4: (33, 33, 17), 2: (37, 40, 21), 1: (61, 47, 29)}

CHILD = r"""
import sys
sys.path[:0] = [sys.argv[1], sys.argv[1] + "/gpu-vh_b200", sys.argv[1] + "/tests"]
import test_stage_variants_gpu as t
t.digests()
"""


def digests():
    for parts, shape in RAGGED.items():
        for physics in PHYSICS.values():
            L = gvh.Lattice(*shape, 0.3, 0.3, 0.3, 0.01, 0.16, **physics)
            L.set_primitive(rich_state(L, seed=4, spacing=0.2))
            for n in range(2):
                L.step(0.5 + 0.01 * n, 0.01)
            st = L.get_state()
            print(parts, L.status(), hashlib.sha256(b"".join(st[k].tobytes() for k in L.field_names)).hexdigest())
    B = gvh.Batch(64 << 20)
    L = gvh.Lattice(*RAGGED[4], 0.3, 0.3, 0.3, 0.01, 0.16)
    event = B.add_event(*RAGGED[4], 0.3, 0.3, 0.3, 0.01, 0.16, rich_state(L, seed=4, spacing=0.2), tau0=0.5)
    B.step(2)
    st = B.get_state(event)
    print("batch", B.info(event).status, hashlib.sha256(b"".join(st[k].tobytes() for k in L.field_names)).hexdigest())


def test_bounds_checked_build_on_every_kernel():
    """No index leaves the arrays, and the states are those of the plain build."""
    if not os.path.exists(gbuild.BOUNDS_LIB):
        pytest.skip("libgvh_bounds.so not built (__graft_entry__.build builds it)")
    out = []
    for lib in (gbuild.BOUNDS_LIB, gbuild.LIB):
        r = subprocess.run([sys.executable, "-c", CHILD, ROOT], env=dict(os.environ, GVH_LIBRARY=lib),
                           capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stderr[-2000:]
        out.append(r.stdout.split("\n"))
    assert all(line.split()[1] == "0" for line in out[0] if line)
    assert out[0] == out[1] and len(out[0]) > 13


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("parts", list(RAGGED))
def test_allocation_free_step_on_every_kernel(parts, precision):
    """Against a batch, whose kernel takes one thread per cell: rounding through the QCD solver in FP64
    (the parity tests' bar), single-precision contraction in mixed (test_zz_no_alloc.py's)."""
    import torch

    shape = RAGGED[parts]
    L = gvh.Lattice(*shape, 0.3, 0.3, 0.3, 0.01, 0.16, precision=precision)
    prim = rich_state(L, seed=8, spacing=0.2)
    L.set_primitive(prim)
    s = L.get_state()
    t = [torch.tensor(stack(L, s, n), device="cuda") for n in
         (L.qnames, ["e"], ["p"], ["utp", "uxp", "uyp", "unp"], ["ut", "ux", "uy", "un"])]
    nxt = torch.empty_like(t[4])
    torch.cuda.synchronize()
    rc = bound().gvh_rk2_step_noalloc(ctypes.byref(L.lattice), ctypes.byref(L.hydro), ctypes.byref(L.options), 0.5, 0.01,
                                      0.0, *[x.data_ptr() for x in t], nxt.data_ptr(), None, None)
    assert rc == 0, bound().gvh_noalloc_last_error()
    torch.cuda.synchronize()
    B = gvh.Batch(64 << 20, precision=precision)
    event = B.add_event(*shape, 0.3, 0.3, 0.3, 0.01, 0.16, prim, tau0=0.5)
    B.step(1)
    want = B.get_state(event)
    for x, names in zip([t[0], t[1], t[2], nxt], (L.qnames, ["e"], ["p"], ["ut", "ux", "uy", "un"])):
        for a, k in zip(x.cpu().numpy().reshape(len(names), -1), names):
            assert rel_err(a, L.interior(want[k]).reshape(-1)) <= (1e-9 if precision == "fp64" else 1e-6), k
