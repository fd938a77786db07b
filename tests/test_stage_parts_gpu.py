"""The stage kernels of small lattices (eight warps per 32 cells, four or two threads per cell)
against the one-thread-per-cell kernel, which a batch and large lattices take. A stage reaches two
cells along each axis, so after one step (two stages) of a small lattice cut out of a large one the
cells four and more from its edges must hold what the large one's do: bit for bit on the mixed
path, whose kernels make the same sums, to rounding in FP64."""
import numpy as np
import pytest

import gvh
from helpers import rich_state

pytestmark = pytest.mark.gpu

HBARC = 0.197326938
LARGE, AT = (61, 60, 40), (9, 8, 7)  # one thread per cell on 148 SMs (more than 56,832 cells)
SMALL = {8: (21, 19, 17), 4: (37, 32, 16), 2: (37, 40, 20)}

QCD, CONF = dict(conformal=False, theta=2.0), dict(conformal=True, theta=1.8)
FULL, SHEAR, IDEAL = dict(shear=True, bulk=True), dict(shear=True, bulk=False), dict(shear=False, bulk=False)
# options, T_reg [GeV], state; T_reg above the whole lattice's temperature regulates every cell
CASES = {
    "qcd_bulk": ({**QCD, **FULL}, 0.0, {}),
    "qcd_shear": ({**QCD, **SHEAR}, 0.0, {}),
    "qcd_ideal": ({**QCD, **IDEAL}, 0.0, {}),
    "conformal_shear": ({**CONF, **SHEAR}, 0.0, {}),
    "conformal_ideal": ({**CONF, **IDEAL}, 0.0, {}),
    "qcd_bulk_regulated": ({**QCD, **FULL}, 2.0, dict(pi=0.3)),
    "qcd_shear_regulated": ({**QCD, **SHEAR}, 0.5, dict(pi=0.3)),
    "qcd_bulk_cartesian": ({**QCD, **FULL, "cartesian": True}, 0.0, {}),
    "conformal_shear_cartesian": ({**CONF, **SHEAR, "cartesian": True}, 0.0, {}),
}


def stepped(shape, prim, opts, T_reg, precision):
    L = gvh.Lattice(*shape, 0.3, 0.3, 0.3, 0.01, 0.16, precision=precision, **opts)
    L.set_primitive(prim if isinstance(prim, dict) else prim(L))
    L.enable_validity()
    L.step(0.5, 0.01, T_reg / HBARC)
    return L, L.get_state(), L.get_validity()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("case", list(CASES))
def test_parts_equal_the_one_thread_kernel(case, precision):
    opts, T_reg, st = CASES[case]
    made = {}

    def large_state(L):
        made.update(rich_state(L, seed=5, spacing=0.1, **st))
        return made

    B, big, big_v = stepped(LARGE, large_state, opts, T_reg, precision)
    for parts, (nx, ny, nz) in SMALL.items():
        i, j, k = AT
        cut = {n: np.ascontiguousarray(v.reshape(B.ncz, B.ncy, B.ncx)[k:k + nz + 4, j:j + ny + 4, i:i + nx + 4]).reshape(-1)
               for n, v in made.items()}
        L, small, small_v = stepped((nx, ny, nz), cut, opts, T_reg, precision)
        assert L.status() == 0 and B.status() == 0

        def pair(a, b, m):  # the cells m and more from the small lattice's edges
            return (L.interior(a)[m:-m, m:-m, m:-m],
                    B.interior(b)[k + m:k + nz - m, j + m:j + ny - m, i + m:i + nx - m])

        for n in L.field_names:
            a, b = pair(small[n], big[n], 4)
            assert a.size
            if precision == "mixed":
                np.testing.assert_array_equal(a, b, err_msg=f"{parts} {n}")
            else:  # sums of at most four terms in another order, through the recovery
                assert np.max(np.abs(a - b)) <= 1e-13 * max(np.max(np.abs(b)), 1e-300), (parts, n)
        for n in L.VALIDITY_NAMES:  # central differences of the new u: one cell further
            a, b = pair(small_v[n], big_v[n], 5)
            if precision == "mixed":
                np.testing.assert_array_equal(a, b, err_msg=f"{parts} {n}")
                continue
            fin = np.isfinite(b)
            assert np.array_equal(np.isfinite(a), fin), (parts, n)
            if fin.any():  # the validity tests' bar
                assert np.max(np.abs(a[fin] - b[fin])) <= 1e-9 * max(np.max(np.abs(b[fin])), 1e-300), (parts, n)
