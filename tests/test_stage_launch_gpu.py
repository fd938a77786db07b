"""How the stage kernels are launched: steps queued back to back, whose kernels overlap their
edges, and steps captured into a CUDA graph, must give what steps with a wait between them give,
bit for bit."""
import ctypes

import numpy as np
import pytest

import gvh
from helpers import rich_state
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
