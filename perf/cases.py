"""The work a user of this framework has it do, as cases that can be timed.

Three kinds of case:

  step      set the state of a handle, take `steps` full time steps (filter and `nkrk` Runge-Kutta stages), read the
            state back: what a driver (`bench.py`), a request of the server or a coupled code does.  A run is in the
            middle of its course when the pass begins: a time step is in hand, the frame moves, and a pass of ten
            steps or more begins where a new time step is taken, as one step in ten does.
  granular  the reference's own procedures one by one on the work field rr of every block (`mpigo`, `deriv` and
            `filte`), as a Fortran driver linked against the library calls them.
  lines     the allocation-free derivative of a set of lines in the caller's own device arrays.

A case is plain values.  Sizes come from the presets, the serving and batch workloads and the tests, or are ragged
neighbours of them.  States are a uniform freestream with smooth random disturbances of about a hundredth (density,
velocity and pressure), functions of the position, so they agree on the points that blocks share.
"""
import math
import random

import numpy as np
import torch

from tandemproject_gb300.config import FP64, MIXED, CaseConfig
from tandemproject_gb300.grid import aerofoil_grid
from tandemproject_gb300.solver import F_RR, Batch, Case, load_library

_PRECISION = {"fp64": FP64, "mixed": MIXED}


# ---- the cases -----------------------------------------------------------------------------------------------------
def _step(name, nx, ny, nz, precision, steps, smgrid=0.0, **kw):
    """nx: points along xi of the upstream, aerofoil and wake blocks; ny, nz: along eta and zeta."""
    c = {"name": name, "kind": "step", "nx0": nx[0], "nx1": nx[1], "nx2": nx[2], "ny0": ny[0], "ny1": ny[1], "nz": nz,
         "precision": precision, "steps": steps, "smgrid": smgrid, "viscous": True, "les": False, "turbulence": 0.0,
         "mach": 0.24, "aoa": 0.0, "thick": 12.0, "ncase": 1}
    return dict(c, **kw)


def listed():
    return [
        # a handful of short lines from a code that may not allocate: the cost of the call itself
        {"name": "lines_small", "kind": "lines", "nlines": 40, "len": 97},
        # as many points as that entry point takes, odd lines
        {"name": "lines_large", "kind": "lines", "nlines": 3327, "len": 601},
        # the reference's procedures one by one, on its smallest grid here (odd in every direction)
        {"name": "granular_0p2m", "kind": "granular", "nx0": 49, "nx1": 121, "nx2": 49, "ny0": 40, "ny1": 40,
         "nz": 13, "smgrid": 0.0},
        # a quick check on that grid: launches and latency count
        _step("fp64_0p2m", (49, 121, 49), (40, 40), 13, "fp64", 10),
        # the 0.61 M-point grid of the parity runs, with the LES terms
        _step("fp64_les_0p6m", (91, 201, 91), (40, 40), 20, "fp64", 10, les=True),
        # an inviscid run, ragged blocks: no viscous sweeps
        _step("fp64_euler_1p9m", (171, 259, 173), (81, 75), 20, "fp64", 10, smgrid=0.004, viscous=False),
        # the headline workload: FP64 with inflow turbulence
        _step("fp64_turb_8p8m", (384, 384, 384), (120, 120), 32, "fp64", 10, smgrid=0.0025, turbulence=0.025),
        # the smallest request of the server, mixed precision
        _step("mixed_turb_0p9m", (160, 160, 160), (56, 56), 16, "mixed", 10, smgrid=0.00625, turbulence=0.02,
              mach=0.3, aoa=4.0, thick=15.0),
        # one step between a copy in and a copy out: a coupled code that takes the state every step
        _step("mixed_coupled_3p3m", (251, 263, 247), (97, 93), 23, "mixed", 1, smgrid=0.004),
        # the largest case of one handle
        _step("mixed_25m", (640, 640, 640), (200, 200), 32, "mixed", 10, smgrid=0.002),
        # many cases of uneven sizes stepped together
        _step("mixed_batch5_17m", (290, 290, 290), (91, 91), 24, "mixed", 10, smgrid=0.0035, turbulence=0.03,
              ncase=5),
        # the same in FP64, small cases
        _step("fp64_batch3_4m", (167, 167, 167), (58, 58), 21, "fp64", 10, smgrid=0.006, ncase=3),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["lines", "granular", "step", "step", "step", "step", "batch"])
    if kind == "lines":
        n = _log_int(rng, 7, 4096)
        return {"kind": "lines", "nlines": _log_int(rng, 1, 2_000_000 // n), "len": n}
    nz = rng.randint(13, 48)
    if kind != "batch" and rng.random() < 0.25:
        # neighbours of the smallest grids: short blocks up- and downstream of the aerofoil's
        nx = rng.randint(115, 205)
        nxs, nys, sm = (nx * 2 // 5 + rng.randint(0, 6), nx, nx * 2 // 5 + rng.randint(0, 6)), (40, 40), 0.0075
        nz = min(nz, 29)
    else:
        # at least 56 points along eta: coarser H-grids of other shapes fold in the wake
        total = _log_int(rng, 400_000, 1_500_000 if kind == "granular" else 3_000_000 if kind == "batch" else 9_000_000)
        ny = max(56, int(math.sqrt(total / (6.0 * nz * 3.2))))
        nx = max(115, total // (6 * nz * ny))
        nxs = tuple(nx - rng.randint(0, nx // 10) for _ in range(3))
        nys = (ny + rng.randint(0, ny // 10), ny + rng.randint(0, ny // 10))
        while sum(nxs) * sum(nys) * nz > 9_000_000:
            nz -= 1
        sm = min(0.0075, max(0.002, 1.0 / nxs[1]))
    if kind == "granular":
        c = _step("", nxs, nys, nz, "fp64", 1, smgrid=sm)
        return {"kind": "granular", **{k: c[k] for k in ("nx0", "nx1", "nx2", "ny0", "ny1", "nz", "smgrid")}}
    precision = rng.choice(["fp64", "mixed"])
    viscous = rng.random() > 0.15
    c = _step("", nxs, nys, nz, precision, rng.choice([1, 2, 5, 10]), smgrid=sm, viscous=viscous,
              les=viscous and rng.random() < 0.15, turbulence=rng.choice([0.0, round(rng.uniform(0.005, 0.05), 4)]),
              mach=round(rng.uniform(0.2, 0.4), 3), aoa=round(rng.uniform(0.0, 8.0), 2),
              thick=round(rng.uniform(8.0, 18.0), 2), ncase=rng.randint(2, 4) if kind == "batch" else 1)
    del c["name"]
    return c


# ---- preparing -----------------------------------------------------------------------------------------------------
def _config(case, k=0):
    """Case k of a handle: the cases of a batch are shorter by a ninth each along xi and differ in their physics."""
    f = (8.0 / 9.0) ** k
    nx = [int(case["nx%d" % i] * f) for i in range(3)]
    ny = [case["ny%d" % i] for i in range(2)]
    kw = {"smgrid": case["smgrid"]} if case["smgrid"] else {}
    if "precision" in case:
        kw.update(precision=_PRECISION[case["precision"]], nviscous=int(case["viscous"]), les=int(case["les"]),
                  turb_intensity=case["turbulence"], mach=case["mach"] * (1 - 0.05 * k), aoa_deg=case["aoa"] + 0.5 * k,
                  thick=case["thick"] - 0.5 * k, turb_seed=1234 + k)
    return CaseConfig(lxibk=tuple(n - 1 for n in nx), letbk=tuple(n - 1 for n in ny), lzebk=(case["nz"] + 2 * k - 1,),
                      nsmf=0, timf=1.0, **kw)


_grids = {}


def _grid(cfg):
    """The last grids, kept on the host: a program that starts many cases on one grid reads it once."""
    key = repr(cfg)
    if key not in _grids:
        while sum(sum(b.size for b in g) for g in _grids.values()) > 150_000_000:
            _grids.pop(next(iter(_grids)))
        _grids[key] = [np.ascontiguousarray(b) for b in aerofoil_grid(cfg)]
    return _grids[key]


def _waves(x, y, z, span, rng, n=3):
    """A sum of n plane waves, periodic over the span, of unit rms."""
    s = 0
    for _ in range(n):
        kx, ky, kz = rng.uniform(-6, 6), rng.uniform(-6, 6), 2 * math.pi * rng.choice([0, 1, 2]) / span
        s = s + torch.sin(kx * x + ky * y + kz * z + rng.uniform(0, 2 * math.pi))
    return s * math.sqrt(2.0 / n)


def _state(grids, spans, seed):
    """[5][points of all blocks] on the host (pinned): rho, rho u, rho v, rho w, rho E."""
    rng = random.Random(seed)
    out = torch.empty((5, sum(b.size // 3 for g in grids for b in g)), dtype=torch.float64, pin_memory=True)
    at = 0
    for g, span in zip(grids, spans):
        waves = rng.getrandbits(60)
        for b in g:
            x, y, z = torch.from_numpy(b.reshape(3, -1)).cuda()
            r = random.Random(waves)
            rho = 1.0 + 0.01 * _waves(x, y, z, span, r)
            u, v, w = (0.01 * _waves(x, y, z, span, r) for _ in range(3))
            p = (1.0 + 0.01 * _waves(x, y, z, span, r)) / 1.4
            q = torch.stack([rho, rho * u, rho * v, rho * w, p / 0.4 + 0.5 * rho * (u * u + v * v + w * w)])
            out[:, at:at + q.shape[1]].copy_(q)
            at += q.shape[1]
    return out


def _points(case):
    return sum(_config(case, k).npoints for k in range(case.get("ncase", 1)))


class _Handle:
    """A handle with its grids set, initialised."""

    def __init__(self, case):
        cfgs = [_config(case, k) for k in range(case.get("ncase", 1))]
        self.grids = [_grid(c) for c in cfgs]
        self.spans = [c.span for c in cfgs]
        self.h = Batch(cfgs) if len(cfgs) > 1 else Case(cfgs[0])
        for b, xyz in enumerate(x for g in self.grids for x in g):
            self.h.set_grid(b, xyz)
        self.h.init()


def _lines_input(case, seed):
    g = torch.Generator().manual_seed(seed)
    n, m = case["nlines"], case["len"]
    x = torch.linspace(0, 1, m, dtype=torch.float64)
    amp = torch.rand((n, 4), generator=g, dtype=torch.float64)
    ph = torch.rand((n, 4), generator=g, dtype=torch.float64)
    f = torch.ones((n, m), dtype=torch.float64)
    for k in range(4):
        f += 0.3 * amp[:, k:k + 1] * torch.sin(2 * math.pi * ((k + 1) * 2 * x + ph[:, k:k + 1]))
    return f


def prepare(case, seed):
    if case["kind"] == "lines":
        f = _lines_input(case, seed).cuda()
        return {"kind": "lines", "lib": load_library(), "in": f, "out": torch.empty_like(f), "nlines": case["nlines"],
                "len": case["len"], "stream": torch.cuda.current_stream().cuda_stream}
    hd = _Handle(case)
    c = hd.h
    q = _state(hd.grids, hd.spans, seed)
    if case["kind"] == "granular":
        # u, v, w of every block, the fields whose derivatives the driver takes
        rr, at = [], 0
        for b in range(len(c.dims)):
            n = c.npts(b)
            rr.append((q[1:4, at:at + n] / q[0:1, at:at + n]).numpy().copy())
            at += n
        return {"kind": "granular", "h": c, "rr": rr}
    q = q.numpy()
    # the time step of this grid and state (the second step of a run takes it)
    c.set_state_all(q)
    c.step(2)
    dt = min(c.case_time(k)[4] for k in range(c.ncase)) if isinstance(c, Batch) else c.get_time()[4]
    out = torch.empty(q.shape, dtype=torch.float64, pin_memory=True).numpy()
    n0 = 11 if case["steps"] >= 10 else 12
    c.set_time((n0, 1 if n0 == 11 else 11, dt, dt, dt, 0.5))
    torch.cuda.synchronize()
    return {"kind": "step", "h": c, "q": q, "out": out, "steps": case["steps"], "time": (n0, 1 if n0 == 11 else 11, dt, dt, dt, 0.5)}


# ---- one pass ------------------------------------------------------------------------------------------------------
def run(state):
    if state["kind"] == "lines":
        rc = state["lib"].ati_deriv_lines_noalloc(state["in"].data_ptr(), state["out"].data_ptr(), state["nlines"],
                                                  state["len"], state["stream"])
        if rc:
            raise RuntimeError("ati_deriv_lines_noalloc: status %d" % rc)
        return state["out"]
    c = state["h"]
    if state["kind"] == "granular":
        nb = len(c.dims)
        for b in range(nb):
            c.set_field(b, F_RR, state["rr"][b])
        # the gradient of rr(:,1) along zeta, eta and xi, as the viscous terms take it ...
        c.mpigo(0, 1, 0)
        for nn in (3, 2, 1):
            c.deriv(nn, 1, 2)
        grad = [c.get_field(b, F_RR) for b in range(nb)]
        # ... and the three-direction filter of rr(:,1)
        for b in range(nb):
            c.set_field(b, F_RR, state["rr"][b])
        c.mpigo(1, 1, 0)
        for nn in (1, 2, 3):
            c.filte(nn, 1)
        return {"gradient": grad, "filtered": [c.get_field(b, F_RR) for b in range(nb)]}
    c.set_time(state["time"])
    c.set_state_all(state["q"])
    c.step(state["steps"])
    return c.get_state_all(state["out"])


# ---- what a pass cannot do without ----------------------------------------------------------------------------------
def work(case):
    if case["kind"] == "lines":
        n = case["nlines"] * case["len"]
        return {"bytes": 16 * n, "flops": 17 * n}
    n = _points(case)
    if case["kind"] == "granular":
        # three fields in and out twice; three derivatives and three filters of one field
        return {"bytes": 2 * 2 * 3 * 8 * n, "flops": (3 * 17 + 3 * 20) * n}
    # a stage reads qa, qo, the metrics (9 planes) and the Jacobian and writes qa; the filter reads and writes qa
    stage = 8 * (5 + 5 + 9 + 1 + 5)
    # 15 flux derivatives of 17 operations and the fluxes and the update; 12 gradients and the stresses on top
    flops = 15 * 17 + 150 + (12 * 17 + 110 if case["viscous"] else 0)
    per_step = 4 * stage + 8 * 10
    return {"bytes": n * (case["steps"] * per_step + 2 * 40), "flops": n * case["steps"] * (4 * flops + 15 * 20)}


# ---- the same in 64 bits, without the framework's code --------------------------------------------------------------
_AL, _BE = 0.5862704032801503, 0.09549533555017055
_ABC = (0.6431406736919156, 0.2586011023495066, 0.007140953479797375)
_ROW = ((-3.456878182643609, 5.839043358834730, 1.015886726041007, -0.2246526470654333, 0.08564940889936562,
         -0.01836710059356763),
        (-0.3177447290722621, -0.02807631929593225, 1.593461635747659, 0.2533027046976367, -0.03619652460174756,
         0.004080281419108407),
        (-0.1219006056449124, -0.6301651351188667, 0.6521195063966084, 0.3938843551210350, 0.01904944407973912,
         -0.001027260523947668))
_LHS = ((0, 0, 1, 5.912678614078549, 3.775623951744012),
        (0, 0.08360703307833438, 1, 2.058102869495757, 0.9704052014790193),
        (0.03250008295108466, 0.3998040493524358, 1, 0.7719261277615860, 0.1626635931256900))


def _compact(f):
    """Compact first derivative of the rows of f (one-sided rows at both ends), by banded elimination."""
    n, m = f.shape
    a = np.zeros((m, 5))
    a[:] = (_BE, _AL, 1, _AL, _BE)
    b = np.zeros((m, n))
    g = f.T
    for k, w in enumerate(_ABC):
        b[3:m - 3] += w * (g[4 + k:m - 2 + k] - g[2 - k:m - 4 - k])
    for r in range(3):
        a[r], a[m - 1 - r] = _LHS[r], _LHS[r][::-1]
        others = [q for q in range(7) if q != r]
        b[r] = sum(w * (g[q] - g[r]) for w, q in zip(_ROW[r], others))
        b[m - 1 - r] = sum(w * (g[m - 1 - r] - g[m - 1 - q]) for w, q in zip(_ROW[r], others))
    for i in range(m):
        for d in (1, 2):
            if i + d < m:
                w = a[i + d, 2 - d] / a[i, 2]
                for q in range(3):
                    if 0 <= 2 - d + q < 5:
                        a[i + d, 2 - d + q] -= w * a[i, 2 + q]
                b[i + d] -= w * b[i]
    x = np.zeros((m + 2, n))
    for i in range(m - 1, -1, -1):
        x[i] = (b[i] - a[i, 3] * x[i + 1] - a[i, 4] * x[i + 2]) / a[i, 2]
    return np.ascontiguousarray(x[:m].T)


def exact(case, seed):
    """The derivative of a set of lines; a whole step in plain 64-bit arrays would take minutes."""
    if case["kind"] != "lines":
        return None
    return _compact(_lines_input(case, seed).numpy())
