"""How the stage kernels are launched: steps queued back to back, whose kernels overlap their
edges, and steps captured into a CUDA graph, must give what steps with a wait between them give,
bit for bit."""
import ctypes

import numpy as np
import pytest

import gvh
from helpers import rel_err, rich_state
from test_zz_no_alloc import bound, stack

pytestmark = pytest.mark.gpu

# below and above one wave of the one-thread-per-cell kernel
SHAPES = {"small": (13, 9, 6), "wave": (61, 47, 29)}


def run(shape, precision, how, steps=6):
    import torch

    nx, ny, nz = SHAPES[shape]
    L = gvh.Lattice(nx, ny, nz, 0.3, 0.3, 0.3, 0.01, 0.16, precision=precision)
    s = torch.cuda.Stream()
    L.set_stream(s.cuda_stream)
    L.set_primitive(rich_state(L, seed=7))
    if how == "captured":
        # three steps bring the handle's buffers back to where they were, so a graph of three
        # can be replayed
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            for n in range(3):
                L.step(0.5, 0.01)
        for _ in range(steps // 3):
            g.replay()
        torch.cuda.synchronize()
    else:
        for n in range(steps):
            L.step(0.5, 0.01)
            if how == "waited":
                L.synchronize()
    assert L.status() == 0
    return L.get_state()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("shape", list(SHAPES))
def test_overlapped_and_captured_steps_equal_separate_steps(shape, precision):
    want = run(shape, precision, "waited")
    for how in ("queued", "captured"):
        got = run(shape, precision, how)
        for k, v in want.items():
            np.testing.assert_array_equal(got[k], v, err_msg=f"{how} {k}")


def test_captured_allocation_free_step():
    """The allocation-free step clears its status word in the stream before the kernels; captured,
    that node precedes the first kernel."""
    import torch

    lib = bound()
    kw = dict(nx=12, ny=10, nz=7, dx=0.3, dy=0.3, dz=0.3, dt=0.01, etabar=0.16, theta=2.0, conformal=False)
    G = gvh.Lattice(**kw)
    G.set_primitive(rich_state(G, seed=31))
    s0 = G.get_state()
    dev = torch.device("cuda", torch.cuda.current_device())
    state = [torch.tensor(stack(G, s0, names), device=dev) for names in
             (G.qnames, ["e"], ["p"], ["utp", "uxp", "uyp", "unp"], ["ut", "ux", "uy", "un"])]
    nxt = torch.empty_like(state[4])

    def step(stream):
        assert lib.gvh_rk2_step_noalloc(ctypes.byref(G.lattice), ctypes.byref(G.hydro), ctypes.byref(G.options), 0.5,
                                        0.01, 0.0, *[t.data_ptr() for t in state], nxt.data_ptr(), None, stream) == 0

    keep = [t.clone() for t in state]
    step(torch.cuda.current_stream().cuda_stream)  # the first call sets the device up
    torch.cuda.synchronize()
    want = [t.clone() for t in state] + [nxt.clone()]
    for t, k in zip(state, keep):
        t.copy_(k)
    nxt.zero_()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    s = torch.cuda.Stream()
    with torch.cuda.graph(g, stream=s):
        step(s.cuda_stream)
    g.replay()
    torch.cuda.synchronize()
    for a, b in zip(state + [nxt], want):
        assert torch.equal(a, b)


# The kernels a lattice smaller than one wave takes (eight warps per 32 cells, four or two threads
# per cell, one thread per cell), on both sides of each rule's line for 148 SMs: 9,472, 18,944,
# 37,888 and 56,832 cells; with a partial last block, one-cell axes, and sizes of a few cells.
PART_SHAPES = [(1, 1, 1), (3, 1, 1), (1, 5, 7), (37, 32, 8), (37, 32, 9), (37, 32, 16), (37, 32, 17), (37, 64, 16),
               (37, 64, 17), (37, 96, 16), (37, 96, 17), (97, 97, 1), (101, 101, 1)]


@pytest.mark.parametrize("physics", ["qcd_bulk", "conformal_shear", "qcd_ideal"])
@pytest.mark.parametrize("shape", PART_SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_small_lattice_kernels_match_the_oracle(shape, physics):
    """One step against the oracle on both sides of every line of the rule. Tolerance as the
    parity tests': 1e-12 of the field's maximum, 1e-9 with the QCD solver."""
    import oracle

    opts = {"qcd_bulk": dict(conformal=False, shear=True, bulk=True, theta=2.0),
            "conformal_shear": dict(conformal=True, shear=True, bulk=False, theta=1.8),
            "qcd_ideal": dict(conformal=False, shear=False, bulk=False, theta=2.0)}[physics]
    nx, ny, nz = shape
    kw = dict(nx=nx, ny=ny, nz=nz, dx=0.3, dy=0.3, dz=0.3, dt=0.01, etabar=0.16, **opts)
    G, O = gvh.Lattice(**kw), oracle.OracleLattice(**kw)
    prim = rich_state(G, seed=13, spacing=6.0 / max(nx, ny))
    G.set_primitive(prim)
    O.set_primitive(prim)
    G.step(0.5, 0.01)
    O.step(0.5, 0.01)
    assert G.status() == 0
    sg, so = G.get_state(), O.get_state()
    for k in G.field_names:
        assert rel_err(G.interior(sg[k]), O.interior(so[k])) <= (1e-12 if opts["conformal"] else 1e-9), k
    tol = 1e-12 if opts["conformal"] else 1e-9
    a, b = G.max_propagation_speed(), O.max_propagation_speed()
    assert abs(a - b) <= tol * max(b, 1e-30)


@pytest.mark.parametrize("shape", [(21, 19, 17), (37, 32, 16), (37, 64, 16), (97, 90, 1)],
                         ids=lambda s: "x".join(map(str, s)))
def test_mixed_small_lattice_kernels_match_a_batch(shape):
    """The mixed path on the small-lattice kernels against a batch's one-thread-per-cell kernel, three
    steps. The mixed path's bar (test_zz_no_alloc): the same FP32 expressions, whose multiply-add
    contraction may differ between kernels."""
    nx, ny, nz = shape
    L = gvh.Lattice(nx, ny, nz, 0.3, 0.3, 0.3, 0.01, 0.16, precision="mixed", tau0=0.5)
    prim = rich_state(L, seed=5, spacing=6.0 / max(nx, ny))
    L.set_primitive(prim)
    B = gvh.Batch(64 << 20, precision="mixed")
    eid = B.add_event(nx, ny, nz, 0.3, 0.3, 0.3, 0.01, 0.16, prim, tau0=0.5)
    for n in range(3):
        L.step(0.5 + n * 0.01, 0.01)
    B.step(3)
    a, b = L.get_state(), B.get_state(eid)
    for k in L.field_names:
        assert rel_err(L.interior(a[k]), L.interior(b[k])) <= 1e-6, k
