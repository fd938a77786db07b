"""What a program pays once: a handle loads the stage kernels it takes and no others; the
allocation-free step loads the rest at its first call on a device."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)

CHILD = r"""
import ctypes, sys
sys.path[:0] = [sys.argv[1], sys.argv[1] + "/gpu-vh_b200", sys.argv[1] + "/tests"]
import torch
import gvh
from helpers import rich_state
from test_zz_no_alloc import bound, stack
free = lambda: torch.cuda.mem_get_info()[0]
kw = dict(nx=12, ny=10, nz=7, dx=0.3, dy=0.3, dz=0.3, dt=0.01, etabar=0.16)
G = gvh.Lattice(**kw)
G.set_primitive(rich_state(G, seed=31))
G.step(0.5, 0.01)
s = G.get_state()
t = [torch.tensor(stack(G, s, n), device="cuda") for n in
     (G.qnames, ["e"], ["p"], ["utp", "uxp", "uyp", "unp"], ["ut", "ux", "uy", "un"])]
nxt = torch.empty_like(t[4])
torch.cuda.synchronize()
def noalloc():
    before = free()
    rc = bound().gvh_rk2_step_noalloc(ctypes.byref(G.lattice), ctypes.byref(G.hydro), ctypes.byref(G.options), 0.5, 0.01,
                                      0.0, *[x.data_ptr() for x in t], nxt.data_ptr(), None, None)
    torch.cuda.synchronize()
    assert rc == 0
    return before - free()
first = noalloc()
print(bound().gvh_rk2_step_noalloc_max_bytes(), first, noalloc())
"""


def test_a_handle_loads_its_own_kernels_only():
    r = subprocess.run([sys.executable, "-c", CHILD, ROOT], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    scratch, first, second = map(int, r.stdout.split()[-3:])
    assert first > scratch  # the step's static scratch and the kernels that the handle did not load
    assert second == 0
