"""The work that users of this library have it do, as measurable cases.

A case is one call pattern on one lattice (or one set of lattices):

  step     a lattice in the layout of the C ABI's device arrays: gather into the handle, RK2 steps,
           scatter back (the seam of the drop-in twoStepRungeKutta, which takes one step per call;
           more steps stand for a program that looks at the state every few steps)
  noalloc  RK2 steps on caller-owned arrays (gvh_rk2_step_noalloc)
  batch    events admitted to a batch, advanced together, read back and retired (one wave of the
           serving loop)
  surface  the freeze-out hypersurface of one slab: both time levels into the handle, the slab's
           rows or its surface.dat text out
  loop     the run loop with its stop test and surface.dat

Initial states are seeded Glauber-hotspot events with a transverse flow, a longitudinal flow and
dissipative currents that satisfy u_mu pi^{mu nu} = 0, at an early or a late proper time (late:
dilute, with cells below the closed-form recovery's threshold)."""
from __future__ import annotations

import ctypes
import math
import os
import shutil
import sys
import tempfile
import weakref
from dataclasses import replace

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "gpu-vh_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import gvh  # noqa: E402
from gvh import workloads  # noqa: E402

HBARC = 0.197326938
PHYSICS = {  # conformal, shear, bulk, theta
    "qcd_bulk": (False, True, True, 2.0),
    "qcd_shear": (False, True, False, 2.0),
    "qcd_ideal": (False, False, False, 2.0),
    "conformal_shear": (True, True, False, 1.8),
    "conformal_ideal": (True, False, False, 1.8),
}
SERVING_GRIDS = ((61, 61, 1, 0.2), (101, 101, 31, 0.15), (131, 131, 61, 0.1))


def _step(name, nx, ny, nz, dx, dz, physics, precision, steps, late=False, etabar=0.16, T_reg_GeV=0.0, kind="step"):
    return dict(name=name, kind=kind, nx=nx, ny=ny, nz=nz, dx=dx, dz=dz, dt=dx / 10, physics=physics,
                precision=precision, steps=steps, late=late, etabar=etabar, T_reg_GeV=T_reg_GeV)


def listed():
    return [
        # the smallest lattice in use (the smoke check's), one step per call: launches and latency
        _step("step_12x10x6_qcd_bulk", 12, 10, 6, 0.3, 0.3, "qcd_bulk", "fp64", 1),
        # the small conformal event of the benchmark, state read every ten steps
        _step("step_33x33x17_conformal", 33, 33, 17, 0.2, 0.2, "conformal_shear", "fp64", 10, etabar=0.2),
        # a 2+1D event on the plain FP64 path
        _step("step_61x61x1_qcd_bulk", 61, 61, 1, 0.2, 0.1, "qcd_bulk", "fp64", 10),
        # a caller with its own device arrays and no allocation at step time
        _step("noalloc_41x41x21_qcd_bulk", 41, 41, 21, 0.2, 0.2, "qcd_bulk", "fp64", 4, kind="noalloc"),
        # ideal hydrodynamics (no dissipative currents), an even lattice
        _step("step_96x80x40_qcd_ideal", 96, 80, 40, 0.15, 0.15, "qcd_ideal", "fp64", 2),
        # a late, dilute event of the serving mix's middle grid, regulated, mixed precision
        _step("step_101x101x31_late_mixed", 101, 101, 31, 0.15, 0.1, "qcd_bulk", "mixed", 2, late=True,
              etabar=0.12, T_reg_GeV=0.13),
        # the full event of the benchmark: plain FP64, and mixed precision
        _step("step_131x131x61_fp64", 131, 131, 61, 0.1, 0.1, "qcd_bulk", "fp64", 2),
        _step("step_131x131x61_mixed", 131, 131, 61, 0.1, 0.1, "qcd_bulk", "mixed", 2),
        # one wave of the serving mix: two events of each grid
        dict(name="batch_serving_mix_mixed", kind="batch", small=2, middle=2, large=2, precision="mixed", steps=4),
        # many 2+1D events at once
        dict(name="batch_16x61x61x1_fp64", kind="batch", small=16, middle=0, large=0, precision="fp64", steps=40),
        # the full event's freeze-out surface, one slab, as text
        dict(_step("surface_131x131x61_text", 131, 131, 61, 0.1, 0.1, "qcd_bulk", "fp64", 1, late=True,
                   kind="surface"), rows=False),
        # a 2+1D event through the run loop, surface.dat written
        _step("loop_61x61x1_surface", 61, 61, 1, 0.2, 0.1, "qcd_bulk", "fp64", 40, late=True, kind="loop"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step"] * 5 + ["noalloc", "batch", "surface", "loop"])
    precision = rng.choice(["fp64", "mixed"])
    if kind == "batch":
        small, middle, large = rng.randint(1, 12), rng.randint(0, 3), rng.randint(0, 2)
        return dict(kind="batch", small=small, middle=middle, large=large, precision=precision,
                    steps=rng.randint(2, 4))
    physics = rng.choice(["qcd_bulk"] * 4 + ["qcd_shear", "qcd_ideal", "conformal_shear", "conformal_ideal"])
    two_d = rng.random() < 0.25
    hi = {"noalloc": 49, "loop": 91}.get(kind, 131)
    nx, ny = _log_int(rng, 10, hi), _log_int(rng, 10, hi)
    nz = 1 if two_d else _log_int(rng, 5, {"noalloc": 31, "loop": 15}.get(kind, 61))
    dx = rng.choice([0.1, 0.15, 0.2])
    steps = 1 if nx * ny * nz > 400000 else rng.randint(1, 6)
    late = rng.random() < 0.4
    if kind == "surface":
        nx, ny, nz, late, physics = max(nx, 31), max(ny, 31), 1 if two_d else max(nz, 9), True, "qcd_bulk"
    if kind == "loop":
        nx, ny, late, physics, steps = max(nx, 31), max(ny, 31), True, "qcd_bulk", rng.randint(11, 32)
    c = _step("", nx, ny, nz, dx, 0.1, physics, precision, steps, late=late, etabar=round(rng.uniform(0.08, 0.24), 4),
              T_reg_GeV=rng.choice([0.0, 0.13]), kind=kind)
    del c["name"]
    if kind == "surface":
        c["rows"] = rng.random() < 0.5
    return c


# ---- initial states (torch, from the seed alone) ----------------------------------------

_PA = [-0.25181736420168666, 9737.845799644809, 1.077580993288114e6, 3.1729694865420084e6, 1.6357487344679043e6,
       334334.4309240126, 41913.439282708554, 6340.448389300905, 141.5073484468774, 0.7158279081255019,
       0.0009417586777847889, 3.1188455176941583e-7, 1.9531729608963267e-11]
_PB = [45829.44617893836, 4.0574329080826794e6, 2.0931169138134286e7, 1.3512402226067686e7, 1.7851642641834426e6,
       278581.2989342773, 26452.34905933697, 499.04919730607065, 2.3405487982094204, 0.002962497695527404,
       9.601103399348206e-7, 5.928138360995685e-11, 3.2581066229887368e-18]
_CA = [5.191934309650155e-32, 4.123605749683891e-23, 3.1955868410879504e-16, 1.4170364808063119e-10,
       6.087136671592452e-6, 0.02969737949090831, 15.382615282179595, 460.6487249985994, 1612.4245252438795,
       275.0492627924299, 58.60283714484669, 6.504847576502024, 0.03009027913262399, 8.189430244031285e-6]
_CB = [1.4637868900982493e-30, 6.716598285341542e-22, 3.5477700458515908e-15, 1.1225580509306008e-9,
       0.00003551782901018317, 0.13653226327408863, 60.85769171450653, 1800.5461219450308, 15190.225535036281,
       590.2572000057821, 293.99144775704605, 21.461303090563028, 0.09301685073435291, 0.000024810902623582917]
_TA = [1.510073201405604e-29, 8.014062800678687e-18, 2.4954778310451065e-10, 0.000063810382643387,
       0.4873490574161924, 207.48582344326206, 6686.07424325115, 14109.766109389702, 1471.6180520527757,
       14.055788949565482, 0.015421252394182246, 1.5780479034557783e-6]
_TB = [7.558667139355393e-28, 1.3686372302041508e-16, 2.998130743142826e-9, 0.0005036835870305458,
       2.316902328874072, 578.0778724946719, 11179.193315394154, 17965.67607192861, 1051.0730543534657,
       5.916312075925817, 0.003778342768228011, 1.8472801679382593e-7]


def _poly(c, x):
    a = torch.full_like(x, c[-1])
    for k in reversed(c[:-1]):
        a = a * x + k
    return a


def _pressure(e, conformal):
    return e / 3 if conformal else _poly(_PA, e) / _poly(_PB, e)


def _workload(case, seed):
    conformal, shear, bulk, theta = PHYSICS[case["physics"]]
    return replace(workloads.CONFIG2, name="case", nx=case["nx"], ny=case["ny"], nz=case["nz"], dx=case["dx"],
                   dy=case["dx"], dz=case["dz"], dtau=case["dt"], conformal=conformal, shear=shear, bulk=bulk,
                   etabar=case["etabar"], theta=theta, seed=int(seed) & 0x3fffffff)


def _tau(case):
    return 4.0 if case["late"] else 0.6


def _fields(case, seed, dev, level=0):
    """The state's fields on the interior, [field][z][y][x]: conserved components, e, p, u, u one step
    earlier. level 1 is a time level a little later (the upper one of a slab)."""
    conformal, shear, bulk, _ = PHYSICS[case["physics"]]
    w = _workload(case, seed)
    late = case["late"]
    hs = workloads.hotspot_sources(w, b=3.0 + (int(seed) % 7), e0_GeV=1.5 if late else 40.0,
                                   sigma_hot=1.2 if late else 0.4, background_GeV=0.012 if late else 0.05)
    f64 = dict(dtype=torch.float64, device=dev)
    tau = _tau(case) + level * case["dt"]
    shape = (case["nz"], case["ny"], case["nx"])
    ax = [(torch.arange(n, **f64) - (n - 1) / 2) * d for n, d in zip(shape, (case["dz"], case["dx"], case["dx"]))]
    z, y, x = ax
    hx, hy, hw = (torch.tensor(np.asarray(a), **f64) for a in (hs.x, hs.y, hs.w))
    s2 = 2 * hs.sigma ** 2
    gx = torch.exp(-(x[None, :] - hx[:, None]) ** 2 / s2)
    gy = torch.exp(-(y[None, :] - hy[:, None]) ** 2 / s2) * hw[:, None]
    plane = (gy.T @ gx) * hs.scale
    fz = torch.exp(-torch.clamp(z.abs() - hs.eta_flat, min=0) ** 2 / (2 * hs.sigma_eta ** 2))
    e = (fz[:, None, None] * plane[None] + hs.background) * (1 + case["dt"] / tau) ** (-1.2 * level) + 1e-3
    rng = np.random.default_rng(int(seed) + 17)
    Z, Y, X = (a.reshape([-1 if k == m else 1 for m in range(3)]) for k, a in enumerate(ax))
    rate = (0.18 if late else 0.06) * (1 + 0.1 * rng.random())
    ux = rate * X * torch.exp(-(X ** 2 + Y ** 2) / 60) * torch.ones_like(e) + 0.02 * torch.sin(1.1 * Y + rng.random())
    uy = 1.2 * rate * Y * torch.exp(-(X ** 2 + Y ** 2) / 60) * torch.ones_like(e) + 0.02 * torch.sin(0.9 * X + rng.random())
    un = (0.02 / tau) * torch.tanh(Z) * torch.cos(0.3 * X) * torch.ones_like(e)  # 0 on a 2+1D lattice

    def ut_of(a, b, c):
        return torch.sqrt(1 + a * a + b * b + tau * tau * c * c)

    ut = ut_of(ux, uy, un)
    back = 1 - case["dt"] / tau
    up = [ut_of(ux * back, uy * back, un * back), ux * back, uy * back, un * back]
    p = _pressure(e, conformal)
    out, pi, Pi = [], None, torch.zeros_like(e)
    if shear:
        amp = [0.08 * (0.5 + rng.random()) for _ in range(5)]
        ph = [rng.uniform(0, 6.28) for _ in range(5)]
        wave = [a * p * torch.cos(0.5 * X + h) * torch.cos(0.4 * Y + 2 * h) for a, h in zip(amp, ph)]
        pixx, pixy, piyy = wave[0] + 0.05 * p, 0.5 * wave[1], wave[2] + 0.05 * p
        flat = 0.0 if case["nz"] == 1 else 1.0
        pixn, piyn = flat * 0.2 * wave[3] / tau, flat * 0.2 * wave[4] / tau
        pinn = -0.1 * p / tau ** 2
        t2 = tau * tau
        pitx = (pixx * ux + pixy * uy + t2 * pixn * un) / ut
        pity = (pixy * ux + piyy * uy + t2 * piyn * un) / ut
        pitn = (pixn * ux + piyn * uy + t2 * pinn * un) / ut
        pitt = (pitx * ux + pity * uy + t2 * pitn * un) / ut
        pi = [pitt, pitx, pity, pitn, pixx, pixy, pixn, piyy, piyn, pinn]
    if bulk:
        Pi = -0.03 * p
    h = e + p + Pi
    T = [h * ut * ut - (p + Pi), h * ut * ux, h * ut * uy, h * ut * un]
    if pi:
        T = [a + b for a, b in zip(T, pi)]
    out = T + (pi or []) + ([Pi] if bulk else []) + [e, p, ut, ux, uy, un] + up
    return torch.stack([a.expand(shape) for a in out]).contiguous()


def _ghosted(f):
    for axis in (1, 2, 3):
        n = f.shape[axis]
        at = torch.clamp(torch.arange(-2, n + 2, device=f.device), 0, n - 1)
        f = f.index_select(axis, at)
    return f.reshape(f.shape[0], -1).contiguous()


def _lattice(case):
    conformal, shear, bulk, theta = PHYSICS[case["physics"]]
    return gvh.Lattice(case["nx"], case["ny"], case["nz"], case["dx"], case["dx"], case["dz"], case["dt"],
                       case["etabar"], theta=theta, conformal=conformal, shear=shear, bulk=bulk,
                       precision=case["precision"], tau0=_tau(case))


def _rows(t):
    n, b = t.shape[0], t.shape[1] * t.element_size()
    return (ctypes.c_void_p * n)(*[t.data_ptr() + k * b for k in range(n)])


def _bind(L):
    vp, ip, dp = ctypes.c_void_p, ctypes.c_int, ctypes.c_double
    L.gvh_gather_state_device.argtypes = [vp, vp, ip, ip]
    L.gvh_scatter_state_device.argtypes = [vp, vp, ip, ip]
    L.gvh_rk2_step_noalloc.argtypes = [ctypes.POINTER(gvh.LatticeParams), ctypes.POINTER(gvh.HydroParams),
                                       ctypes.POINTER(gvh.Options), dp, dp, dp, vp, vp, vp, vp, vp, vp, vp, vp]
    return L


def _ok(rc):
    if rc != 0:
        raise RuntimeError("call failed (%d): %s" % (rc, gvh.load().gvh_last_error().decode()))


class State(dict):
    """What one case keeps between passes (weak-referenceable, so that files can follow its life)."""


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    lib = _bind(gvh.load())
    st = State(case=case, lib=lib)
    kind = case["kind"]
    if kind == "batch":
        arena = 0
        grids = [g for g, n in zip(SERVING_GRIDS, (case["small"], case["middle"], case["large"])) for _ in range(n)]
        b = gvh.Batch(1 << 20, precision=case["precision"], theta=2.0)
        for nx, ny, nz, _ in grids:
            arena += b.event_bytes(nx, ny, nz) + 256
        b.close()
        st["batch"] = b = gvh.Batch(arena + (1 << 20), precision=case["precision"], theta=2.0)
        rng = np.random.default_rng(int(seed))
        st["events"] = []
        for nx, ny, nz, dx in grids:
            w = replace(workloads.CONFIG2, nx=nx, ny=ny, nz=nz, dx=dx, dy=dx, dz=0.1, dtau=dx / 10,
                        seed=int(rng.integers(1 << 30)))
            hs = workloads.hotspot_sources(w, b=float(rng.uniform(0, 12)))
            etabar = float(rng.uniform(0.08, 0.24))
            out = torch.empty((b.nq + 10, (nx + 4) * (ny + 4) * (nz + 4)), dtype=torch.float64, device=dev)
            st["events"].append(((nx, ny, nz, dx, dx, 0.1, dx / 10, etabar), hs, out, _rows(out)))
        return st
    f = _fields(case, seed, dev)
    t = _tau(case)
    if kind == "noalloc":
        conformal, shear, bulk, theta = PHYSICS[case["physics"]]
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        o = gvh.Options()
        lib.gvh_default_options(ctypes.byref(o))
        o.eos = gvh.GVH_EOS_CONFORMAL if conformal else gvh.GVH_EOS_QCD
        o.shear, o.bulk, o.theta = int(shear), int(bulk), theta
        o.precision = gvh.GVH_PRECISION_MIXED if case["precision"] == "mixed" else gvh.GVH_PRECISION_FP64
        f = f.reshape(f.shape[0], -1)
        nq = f.shape[0] - 10
        st["opts"] = o
        st["lat"] = gvh.LatticeParams(nx, ny, nz, nx + 4, ny + 4, nz + 4, 0, case["dx"], case["dx"], case["dz"],
                                      case["dt"])
        st["hyd"] = gvh.HydroParams(t, case["etabar"], 0.15, 0, 0.0)
        st["q0"], st["ep0"] = f[:nq].clone(), f[nq:nq + 2].clone()
        st["u0"] = torch.stack([f[nq + 6:nq + 10], f[nq + 2:nq + 6], torch.zeros_like(f[nq + 2:nq + 6])])
        st["q"], st["ep"], st["u"] = (torch.empty_like(st[k]) for k in ("q0", "ep0", "u0"))
        return st
    st["L"] = L = _lattice(case)
    st["stream"] = s = torch.cuda.Stream(dev)
    L.set_stream(s.cuda_stream)
    st["in"] = g = _ghosted(f)
    st["in_rows"] = _rows(g)
    if kind == "surface":
        st["upper"] = _ghosted(_fields(case, seed, dev, level=1))
        st["upper_rows"] = _rows(st["upper"])
        st["surface"] = S = gvh.Surface(L, gvh.energy_density_of_temperature(0.15))
        S.set_outputs(rows=bool(case["rows"]), text=not case["rows"])
        # where a pass puts what it found (the crossed hypercubes are a thin shell of the lattice)
        most = case["nx"] * case["ny"] * case["nz"] // 4 + 4096
        st["found"] = np.zeros((most, gvh.SURFACE_COLUMNS)) if case["rows"] else np.zeros(most * 200, np.uint8)
        return st
    st["out"] = torch.empty_like(g)
    st["out_rows"] = _rows(st["out"])
    if kind == "loop":
        st["dir"] = d = tempfile.mkdtemp(prefix="gvh_loop_")
        weakref.finalize(st, shutil.rmtree, d, True)
    return st


_GROUPS = (("T", 0, 4), ("e", -10, -9), ("p", -9, -8), ("u", -8, -4), ("u_previous", -4, None))


def _grouped(f):
    """[field][cell] as a dict of the state's quantities."""
    d = {k: f[a:b] for k, a, b in _GROUPS}
    nq = f.shape[0] - 10
    if nq >= 14:
        d["pi"] = f[4:14]
    if nq == 15:
        d["Pi"] = f[14:15]
    return d


def run(st):
    case, lib = st["case"], st["lib"]
    kind, t0, dt = case["kind"], 0.6 if case["kind"] == "batch" else _tau(case), case.get("dt")
    if kind == "batch":
        b = st["batch"]
        ids = [b.add_event_hotspots(*a, hs, tau0=t0) for a, hs, _, _ in st["events"]]
        b.step(case["steps"])
        for i, (_, _, out, rows) in zip(ids, st["events"]):
            rc = lib.gvh_batch_get_state(b._h, i, rows, len(rows))
            if rc != 0:
                raise RuntimeError("gvh_batch_get_state: %d" % rc)
            b.remove_event(i)
        return [{"q": out[:-10], "e_p_u": out[-10:]} for _, _, out, _ in st["events"]]
    T_reg = case["T_reg_GeV"] / HBARC
    if kind == "noalloc":
        q, ep, u = st["q"], st["ep"], st["u"]
        q.copy_(st["q0"])
        ep.copy_(st["ep0"])
        u.copy_(st["u0"])
        prev, cur, nxt = u[0], u[1], u[2]
        stream = torch.cuda.current_stream().cuda_stream
        for n in range(case["steps"]):
            _ok(lib.gvh_rk2_step_noalloc(ctypes.byref(st["lat"]), ctypes.byref(st["hyd"]), ctypes.byref(st["opts"]),
                                         t0 + n * dt, dt, T_reg, q.data_ptr(), ep[0].data_ptr(), ep[1].data_ptr(),
                                         prev.data_ptr(), cur.data_ptr(), nxt.data_ptr(), None, stream))
            prev, cur, nxt = cur, nxt, prev
        return _grouped(torch.cat([q, ep, cur, prev]))
    L, n = st["L"], len(st["in_rows"])
    _ok(lib.gvh_gather_state_device(L._h, st["in_rows"], n, 8))
    if kind == "surface":
        S = st["surface"]
        S.set_lower()
        _ok(lib.gvh_gather_state_device(L._h, st["upper_rows"], n, 8))
        count = S.find(t0, t0)
        found = st["found"]
        if case["rows"]:
            found[:count] = S.rows()
            return {"count": count, "rows": found}
        text, size = ctypes.c_void_p(), ctypes.c_longlong()
        lib.gvh_surface_get_text(S._h, ctypes.cast(ctypes.byref(text), ctypes.POINTER(ctypes.c_char_p)),
                                 ctypes.byref(size))
        ctypes.memmove(found.ctypes.data, text, min(size.value, found.nbytes))
        return {"count": count, "bytes": size.value, "text": found}
    if kind == "loop":
        rep = L.run_loop(case["steps"], output_dir=st["dir"], surface=True, tau0=t0, T_fo_GeV=0.15,
                         T_reg_GeV=case["T_reg_GeV"])
        _ok(lib.gvh_scatter_state_device(L._h, st["out_rows"], n, 8))
        return {"state": _grouped(st["out"]), "elements": rep["surface_elements"], "steps": rep["steps"]}
    for k in range(case["steps"]):
        L.step(t0 + k * dt, dt, T_reg)
    _ok(lib.gvh_scatter_state_device(L._h, st["out_rows"], n, 8))
    return _grouped(st["out"])


# ---- what a pass cannot do without ------------------------------------------------------

def _cell_work(physics, steps):
    """(bytes, flops) of `steps` RK2 steps of one cell. Bytes: stage 1 reads q, e, u, u_previous and
    writes q, e, u; stage 2 reads those, u and q of the step's start and writes q, e, u: 5 nq + 28
    values of 8 bytes. Flops per step: two stages of source, 3 x 2 x nq limited fluxes and 13 primitive
    recoveries (QCD: two Newton updates each on average)."""
    conformal, shear, bulk, _ = PHYSICS[physics]
    nq = 4 + (10 if shear else 0) + (1 if bulk else 0)
    flops = 2 * (13 * (30 if conformal else 260) + 3 * nq * 45 + (900 if shear else 150))
    return steps * 8 * (5 * nq + 28), steps * flops


def work(case):
    kind = case["kind"]
    if kind == "batch":
        total = [0, 0]
        for (nx, ny, nz, _), n in zip(SERVING_GRIDS, (case["small"], case["middle"], case["large"])):
            b, f = _cell_work("qcd_bulk", case["steps"])
            total[0] += n * (nx * ny * nz * b + (nx + 4) * (ny + 4) * (nz + 4) * 25 * 8)
            total[1] += n * nx * ny * nz * f
        return {"bytes": total[0], "flops": total[1]}
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    cells, ghosted = nx * ny * nz, (nx + 4) * (ny + 4) * (nz + 4)
    _, shear, bulk, _ = PHYSICS[case["physics"]]
    nf = 14 + (10 if shear else 0) + (1 if bulk else 0)
    if kind == "surface":  # both levels in, the corners' energies and the ten fields of the crossed cubes
        return {"bytes": 2 * cells * nf * 8 + 4 * cells * 8, "flops": 0}
    steps = case["steps"] + (1 if kind == "loop" else 0)
    b, f = _cell_work(case["physics"], steps)
    return {"bytes": cells * b + 2 * (cells if kind == "noalloc" else ghosted) * nf * 8, "flops": cells * f}


# ---- the same values in 64 bits with torch alone ----------------------------------------

def _shift(f, axis, d):
    n = f.shape[axis]
    if n == 1:
        return f
    return f.index_select(axis, torch.clamp(torch.arange(n, device=f.device) + d, 0, n - 1))


def _slope(theta, x, y, z):
    """Generalised minmod slope of three neighbours."""
    a, b, c = theta * (y - x), (z - x) / 2, theta * (z - y)
    m = torch.minimum(torch.minimum(a.abs(), b.abs()), c.abs())
    return torch.where((a > 0) & (b > 0) & (c > 0), m, torch.where((a < 0) & (b < 0) & (c < 0), -m, 0 * m))


def _recover(conformal, t, q, guess):
    """e, p, u^mu of a conserved state by Newton's method from the guess (stop test 1e-3)."""
    nq = q.shape[0]
    pi = q[4:8] if nq >= 14 else torch.zeros_like(q[:4])
    Pi = q[14] if nq == 15 else torch.zeros_like(q[0])
    M0, M1, M2, M3 = q[0] - pi[0], q[1] - pi[1], q[2] - pi[2], q[3] - pi[3]
    M = M1 * M1 + M2 * M2 + t * t * M3 * M3
    closed = M0 - M / M0
    if conformal:
        e = (torch.sqrt((4 * M0 * M0 - 3 * M).abs()) - M0).abs()
    else:
        e = guess.clone()
        live = torch.nonzero((guess > 0.1).reshape(-1)).reshape(-1)
        flat = e.reshape(-1)
        m0, m, bulk = M0.reshape(-1), M.reshape(-1), Pi.reshape(-1)
        for it in range(2000):
            if live.numel() == 0:
                break
            e0, a0, am, ab = flat[live], m0[live], m[live], bulk[live]
            c = _pressure(e0, False) / e0
            g = _poly(_CA, e0) / _poly(_CB, e0) - c
            A, B = a0 * (1 - c) + ab, a0 * (a0 + ab) - am
            H = torch.sqrt((A * A + 4 * c * B).abs())
            D = (A - H) / (2 * c)
            slope = 1 - g * (B + D * H - g * c * D * a0 / e0) / (c * e0 * H)
            e1 = e0 - (0.9 if it >= 200 else 1.0) * (e0 + D) / slope
            flat[live] = e1
            live = live[~((e1 - e0).abs() <= 1e-3 * e1.abs())]
    e = torch.where(guess <= 0.1, closed, e)
    p = _pressure(e, conformal)
    low = e < 1e-7
    e, p = torch.where(low, 1e-7 + 0 * e, e), torch.where(low, 1e-7 + 0 * p, p)
    P = p + Pi
    E = 1 / (e + P)
    ut = torch.sqrt(((M0 + P) * E).abs())
    return e, p, torch.stack([ut, M1 * E / ut, M2 * E / ut, M3 * E / ut])


_PAIR = {(0, 0): 4, (0, 1): 5, (0, 2): 6, (0, 3): 7, (1, 1): 8, (1, 2): 9, (1, 3): 10, (2, 2): 11, (2, 3): 12,
         (3, 3): 13}


def _source(case, t, q, e, p, u, up):
    conformal, shear, bulk, theta = PHYSICS[case["physics"]]
    h = (case["dz"], case["dx"], case["dx"])
    zero = torch.zeros_like(e)

    def grad(f):  # limited derivatives along x, y, eta
        return [_slope(theta, _shift(f, k, -1), f, _shift(f, k, 1)) / h[k] for k in (2, 1, 0)]

    du = [grad(u[m]) for m in range(4)]  # du[m][axis]
    dp = grad(p)
    pi = {k: (q[c] if shear else zero) for k, c in _PAIR.items()}
    pi.update({(b, a): v for (a, b), v in list(pi.items())})
    Pi = q[14] if bulk else zero
    ut, un = u[0], u[3]
    v = [u[k] / ut for k in (1, 2, 3)]
    dkvk = sum((du[k + 1][k] - v[k] * du[0][k]) / ut for k in range(3))
    tnn = (e + p + Pi) * un * un + (p + Pi) / t / t + pi[3, 3]
    S = [-(q[0] / t + t * tnn) + dkvk * (pi[0, 0] - p - Pi) - sum(v[k] * dp[k] for k in range(3)),
         -q[1] / t - dp[0] + dkvk * pi[0, 1], -q[2] / t - dp[1] + dkvk * pi[0, 2],
         -3 * q[3] / t - dp[2] / t ** 2 + dkvk * pi[0, 3]]
    if not shear:
        return torch.stack(S)
    # Israel-Stewart right-hand sides; index 3 is eta with the metric factor t^2
    T = (e / 13.8997) ** 0.25 if conformal else _poly(_TA, e) / _poly(_TB, e)
    f02, f033, f16 = float(np.float32(0.2)), float(np.float32(0.333333)), float(np.float32(1.6))
    t2 = t * t
    dtu = [(u[m] - up[m]) / case["dt"] for m in range(4)]
    conv = [ut * dtu[m] + sum(u[k + 1] * du[m][k] for k in range(3)) for m in range(4)]  # u.d u^m
    Dlow = [conv[0] + t * un * un, -conv[1], -conv[2], -t2 * conv[3] - 2 * t * ut * un]
    expansion = ut / t + dtu[0] + du[1][0] + du[2][1] + du[3][2]
    th3 = expansion / 3
    a = conv  # accelerations without the connection terms
    s = {(0, 0): -t * ut * un ** 2 + (dtu[0] - ut * a[0]) + (ut ** 2 - 1) * th3}
    for k, m in ((1, 1), (2, 2)):
        s[0, k] = -(t * un ** 2 * u[k]) / 2 + (dtu[k] - du[0][k - 1]) / 2 - (u[k] * a[0] + ut * a[k]) / 2 + ut * u[k] * th3
        s[k, k] = -(du[k][k - 1] + u[k] * a[k]) + (1 + u[k] ** 2) * th3
        s[k, 3] = -ut * u[k] * un / t - (du[3][k - 1] + du[k][2] / t2) / 2 - (un * a[k] + u[k] * a[3]) / 2 + u[k] * un * th3
    s[0, 3] = -un * (2 * ut ** 2 + t2 * un ** 2) / (2 * t) + (dtu[3] - du[0][2] / t2) / 2 - (un * a[0] + ut * a[3]) / 2 + ut * un * th3
    s[1, 2] = -(du[2][0] + du[1][1]) / 2 - (u[2] * a[1] + u[1] * a[2]) / 2 + u[1] * u[2] * th3
    s[3, 3] = -ut * (1 + 2 * t2 * un ** 2) / t ** 3 - du[3][2] / t2 - un * a[3] + (1 / t2 + un ** 2) * th3
    s.update({(j, i): x for (i, j), x in list(s.items())})
    Dn = Dlow[3]
    wx = (-dtu[1] - du[0][0] + ut * a[1] - u[1] * a[0] - t * un ** 2 * u[1]) / 2
    wy = (-dtu[2] - du[0][1] + ut * a[2] - u[2] * a[0] - t * un ** 2 * u[2]) / 2
    wn = (-t2 * dtu[3] - 2 * t * un - du[0][2] - ut * Dn - t2 * un * a[0] - t ** 3 * un ** 3) / 2
    wxy = (du[2][0] - du[1][1] + u[1] * a[2] - u[2] * a[1]) / 2
    wxn = (t2 * du[3][0] - du[1][2] - u[1] * Dn - t2 * un * a[1]) / 2
    wyn = (t2 * du[3][1] - du[2][2] - u[2] * Dn - t2 * un * a[2]) / 2
    W = {(0, 1): wx, (0, 2): wy, (0, 3): wn, (1, 2): wxy, (1, 3): wxn, (2, 3): wyn, (1, 0): wx, (2, 0): wy,
         (3, 0): wn / t2, (2, 1): -wxy, (3, 1): -wxn / t2, (3, 2): -wyn / t2}  # W[i, j] = omega^i_j
    low = (1, -1, -1, -t2)  # metric signs of a lowered index
    ps = sum(low[i] * low[j] * pi[i, j] * s[i, j] for i in range(4) for j in range(4))
    metric = (-1.0, 1.0, 1.0, 1 / t2)
    rhs = []
    for i, j in _PAIR:
        I1 = sum((pi[i, k] * u[j] + pi[j, k] * u[i]) * Dlow[k] for k in range(4))
        I3 = sum((pi[i, k] * W[j, k] if k != j else 0) + (pi[j, k] * W[i, k] if k != i else 0) for k in range(4))
        I4 = sum(low[k] * (pi[i, k] * s[j, k] + pi[j, k] * s[i, k]) for k in range(4)) / 2
        I4 = I4 + ((metric[i] if i == j else 0) + u[i] * u[j]) * ps / 3
        x = 2 * f02 * (e + p) * s[i, j] - pi[i, j] * f02 * T / case["etabar"]
        x = x - (I1 + 1.33333 * expansion * pi[i, j] - I3 + 1.42857 * I4 - 1.2 * Pi * s[i, j])
        # the connection of the eta direction
        for c, o in ((i, j), (j, i)):
            if c == 0:
                x = x - un * t * pi[o, 3]
            if c == 3:
                x = x - (ut * pi[o, 3] + un * pi[o, 0]) / t
        rhs.append(x / ut + pi[i, j] * dkvk)
    if bulk:
        cs2 = zero if conformal else _poly(_CA, e) / _poly(_CB, e)
        d = f033 - cs2
        y = T / 1.01355
        hot = 0.9 * torch.exp(-(y - 1) / 0.025) + 0.25 * torch.exp(-(y - 1) / 0.13) + 0.001
        cold = 0.9 * torch.exp((y - 1) / 0.0025) + 0.22 * torch.exp((y - 1) / 0.022) + 0.03
        zeta = torch.where(y > 1.05, hot, torch.where(y < 0.995, cold, -13.77 * y * y + 27.55 * y - 13.45))
        x = -15 * d * d * (e + p) * expansion - Pi * 15 * d * d * T / zeta - 0.666667 * Pi * expansion + f16 * d * ps
        rhs.append(x / ut + Pi * dkvk)
    return torch.stack(S + rhs)


def _euler(case, t, q, e, p, u, up):
    conformal, shear, bulk, theta = PHYSICS[case["physics"]]
    out = q + case["dt"] * _source(case, t, q, e, p, u, up)
    for k, axis in ((1, 2), (2, 1), (3, 0)):  # u index, tensor axis of one field
        d = case["dz"] if k == 3 else case["dx"]
        ta = axis + 1  # with the component axis in front
        slope = _slope(theta, _shift(q, ta, -1), q, _shift(q, ta, 1))
        plus, minus = q + slope / 2, q - slope / 2  # the cell's states at its two faces
        n = q.shape[ta]
        at = torch.arange(n, device=q.device).reshape([-1 if m == ta else 1 for m in range(4)])
        # beyond the edge the ghost cells repeat the last cell, with slope 0
        right = torch.where(at == n - 1, q, _shift(minus, ta, 1))
        left = torch.where(at == 0, q, _shift(plus, ta, -1))

        def flux(L, R):
            uL, uR = _recover(conformal, t, L, e)[2], _recover(conformal, t, R, e)[2]
            wL, wR = uL[k] / uL[0], uR[k] / uR[0]
            a = torch.maximum(wL.abs(), wR.abs())
            return (wR * R + wL * L - a * (R - L)) / 2

        inc = (flux(left, minus) - flux(plus, right)) / d
        if shear:
            der = (_shift(q, ta, 1) - _shift(q, ta, -1)) / d / 2
            v = u[k] / u[0]
            for m in range(4):
                lo, hi = (min(m, k), max(m, k))
                inc[m] = inc[m] + der[_PAIR[0, m]] * v - der[_PAIR[lo, hi]]
            if bulk:
                inc[0] = inc[0] - v * der[14]
                inc[k] = inc[k] - (der[14] / t ** 2 if k == 3 else der[14])
        out = out + case["dt"] * inc
    return out


def _regulated(case, t, q, e, p, u, e_reg):
    if q.shape[0] < 14:
        return q
    pi = {k: q[c] for k, c in _PAIR.items()}
    pi.update({(b, a): x for (a, b), x in list(pi.items())})
    low = (1, -1, -1, -t * t)
    pipi = sum(low[i] * low[j] * pi[i, j] ** 2 for i in range(4) for j in range(4))
    size = pipi.abs().sqrt()
    worst = size / torch.sqrt(e * e + 3 * p * p)
    trace = sum(low[i] * pi[i, i] for i in range(4))
    for x in [trace] + [sum(low[j] * pi[i, j] * u[j] for j in range(4)) for i in range(4)]:
        worst = torch.fmax(worst, x / (0.1 * size))
    fac = torch.where(worst.abs() < 1e-7, 1 + 0 * worst, torch.tanh(worst) / worst)
    fac = torch.where(e > e_reg, 1 + 0 * fac, fac)
    return torch.cat([q[:4], q[4:14] * fac, q[14:]])


def _rk2(case, t, q, e, p, u, up):
    conformal = PHYSICS[case["physics"]][0]
    T = case.get("T_reg_GeV", 0.0) / HBARC
    e_reg = _e_of_T(conformal, T)
    t1 = t + case["dt"]
    qs = _euler(case, t, q, e, p, u, up)
    es, ps, us = _recover(conformal, t1, qs, e)
    qs = _regulated(case, t1, qs, es, ps, us, e_reg)
    qn = (_euler(case, t1, qs, es, ps, us, u) + q) / 2
    en, pn, un = _recover(conformal, t1, qn, es)
    return _regulated(case, t1, qn, en, pn, un, e_reg), en, pn, un, u


def _e_of_T(conformal, T):
    if conformal:
        return 13.8997 * T ** 4
    num = [-0.011958188410851651, 119.89423098138208, -3156.9475699248055, 32732.86844374939, -187899.8994764422,
           712537.3610845465, -1.557049803609345e6, 1.4852519861308339e6, 532132.6079941876, -1.963099445042592e6,
           -4484.44579242679, 1.7984228830058286e6, 119345.25619517374, -1.3499773937058165e6, -207838.4995663606,
           654970.2138652403, -78643.00334616247, 40274.00078068926, 422619.58977657766, -409688.07836393174,
           -62005.75915066359, 46788.14270090656, 40784.330477857235, -12589.47744840392]
    den = [31630.074365558292, -127100.88940643385, 173528.1225422275, -39403.297956865215, -85582.57873541754,
           9320.560804233442, 50882.74198960172, 20335.926473421183, -14897.725710713818, -23836.484117457,
           -13726.013896090335, 4517.908673107615, 18056.19917986404, 14954.82860467155, 2569.623976952738,
           -9304.046211514986, -15606.429173842751, 8383.710735812094, 1591.3177623932843, -678.748230997762,
           -33.58687934953277, 3.2520554133126285, -0.19647288043440464, 0.005443394551264717]
    return sum(c * T ** k for k, c in enumerate(num)) / sum(c * T ** k for k, c in enumerate(den))


def exact(case, seed):
    kind = case["kind"]
    dev = torch.device("cuda", torch.cuda.current_device())
    if kind == "surface":
        return None  # a branchy geometric construction; its values come with its rows
    if kind == "batch":
        return None  # the same step as the lattices', on hotspot states rounded to float
    if kind == "loop" and case["nx"] * case["ny"] * case["nz"] * case["steps"] > 20_000_000:
        return None
    f = _fields(case, seed, dev)
    nq = f.shape[0] - 10
    s = (f[:nq], f[nq], f[nq + 1], f[nq + 2:nq + 6], f[nq + 6:nq + 10])
    steps = case["steps"] + (1 if kind == "loop" else 0)
    t0 = _tau(case)
    for n in range(steps):
        s = _rk2(case, t0 + n * case["dt"], *s)
    q, e, p, u, up = s
    out = torch.cat([q, e[None], p[None], u, up])
    if kind == "noalloc":
        return _grouped(out.reshape(out.shape[0], -1))
    g = _grouped(_ghosted(out))
    return {"state": g, "elements": None, "steps": None} if kind == "loop" else g
