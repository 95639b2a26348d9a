"""What the step is timed on: whole runs through the public entry points.

A pass is what a program that uses this framework does with one scenario, or
with a batch of them: the DATA arrays (or a checkpoint) go to the device, the
loop body runs for a number of steps, and the results come back to host
memory.  The kinds of scenario are those of the test and benchmark
configurations -- flat dam break, tilted slab, lake at rest, mudflow on a bumpy
slope, the batched ensemble and the serving mix -- with terrain, rheology and
release drawn from the seed.

``exact`` integrates the same equations (main/optim_par.cpp:128-682) with torch
in 64 bits, scattering with index_add.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from amsc_b200.batch import Batch
from amsc_b200.dampm import STATE_FIELDS, Solver, pinned_array
from amsc_b200.data import DATA
from amsc_b200.serving import Request, Server

UPLOAD = ("x", "y", "Mp", "Ap", "vpx", "vpy", "hp", "mom_px", "mom_py", "Vp")
MOVING = ("x", "y", "vpx", "vpy", "hp", "F_11", "F_12", "F_22")
DEPTHS = ("x", "y", "hp")
FRAME = MOVING + ("mom_px", "mom_py", "Ap", "Zp", "hpZ", "apx", "apy", "dZxp", "dZyp", "Fpx",
                  "Fpy", "Fric_px", "Fric_py")
FRAME_NODES = ("vvxL", "vvyL", "Mv", "HV")
FOREVER = 2_000_000_000  # a loop bound that no run reaches


def listed():
    return [
        # the smallest use: 4096 particles of a flat dam break, fixed dt, where
        # a step is a chain of short kernels
        {"name": "dambreak_64", "kind": "dam", "cells": 64, "steps": 50},
        # the reference's scaling fixture of 10000 (Bingham + Voellmy, 100 steps)
        {"name": "slab_10000", "kind": "slab", "n": 10000, "steps": 100},
        # lake at rest over a bump: still-water level, adaptive dt, a spacing
        # that is no power of two, an odd particle count
        {"name": "lake_50", "kind": "lake", "cells": 50, "spacing": 0.17, "steps": 100},
        # an ordinary mudflow, 0.25M particles, adaptive dt
        {"name": "mudflow_512", "kind": "mudflow", "cells": 512, "h": 0.5, "steps": 100},
        # a ragged one: odd grid, spacing no power of two
        {"name": "mudflow_777", "kind": "mudflow", "cells": 777, "h": 0.37, "steps": 100},
        # the largest: the 2048 x 2048 mudflow of the benchmark, 4.0M particles
        {"name": "mudflow_2048", "kind": "mudflow", "cells": 2048, "h": 0.5, "steps": 160},
        # the same kind with particles merged and split every 10 steps
        {"name": "mergesplit_1024", "kind": "mergesplit", "cells": 1024, "h": 0.5, "steps": 100},
        # output: every 10th step is recorded and its fields are written out
        {"name": "frame_512", "kind": "frame", "cells": 512, "h": 0.5, "steps": 10},
        # restart from a checkpoint on the host, a short advance, the whole
        # state back (a host-coupled program)
        {"name": "restart_1024", "kind": "restart", "cells": 1024, "h": 0.5, "steps": 16},
        # ensembles of independent scenarios at a fixed dt, in both precisions
        {"name": "ensemble_96", "kind": "ensemble", "members": 96, "mix": 1, "precision": "fp64",
         "steps": 320},
        {"name": "ensemble_96_fp32", "kind": "ensemble", "members": 96, "mix": 1,
         "precision": "fp32", "steps": 128},
        # a serving burst: adaptive dt, requests finish one by one and make
        # room for the ones that queue
        {"name": "serving_20", "kind": "serving", "requests": 20, "mix": 2, "t_end": 4.0,
         "precision": "fp64"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("dam", "slab", "lake", "mudflow", "mudflow", "mudflow", "mergesplit",
                       "frame", "restart", "ensemble", "ensemble", "serving"))
    h = rng.choice((0.5, 0.5, 0.25, 0.37, 1.0))
    precision = rng.choice(("fp64", "fp32"))
    if kind == "dam":
        return {"kind": kind, "cells": 16 * rng.randint(2, 16), "steps": rng.randint(20, 100)}
    if kind == "slab":
        return {"kind": kind, "n": _log_int(rng, 1000, 100000), "steps": rng.randint(20, 100)}
    if kind == "lake":
        return {"kind": kind, "cells": rng.randint(20, 120),
                "spacing": round(rng.uniform(0.05, 0.2), 3), "steps": rng.randint(20, 100)}
    if kind == "mudflow":
        return {"kind": kind, "cells": _log_int(rng, 128, 1800), "h": h,
                "steps": rng.randint(40, 120)}
    if kind == "mergesplit":
        return {"kind": kind, "cells": _log_int(rng, 128, 1024), "h": h,
                "steps": 10 * rng.randint(2, 10)}
    if kind == "frame":
        return {"kind": kind, "cells": _log_int(rng, 64, 700), "h": h, "steps": 10}
    if kind == "restart":
        return {"kind": kind, "cells": _log_int(rng, 128, 1024), "h": h,
                "steps": rng.randint(1, 32)}
    if kind == "ensemble":
        return {"kind": kind, "members": _log_int(rng, 2, 96), "mix": rng.randint(10, 1 << 20),
                "precision": precision, "steps": rng.randint(24, 200)}
    return {"kind": kind, "requests": rng.randint(3, 20), "mix": rng.randint(10, 1 << 20),
            "t_end": round(rng.uniform(1.0, 4.0), 2), "precision": precision}


# ---------------------------------------------------------------------------
# scenarios: (arrays in DATA order, scalars) from a case and a seed
# ---------------------------------------------------------------------------
def _scalars(**kw):
    s = {"Nex": 1, "Ney": 1, "hx": 1.0, "hy": 1.0, "rho": 1000.0, "g": 9.81, "T": 1e30,
         "xi": 200.0, "mu": 50.0, "phi": 20.0, "tauy": 30.0, "BINGHAM_ON": 1.0,
         "FRICTION_ON": 1.0, "CFL": 0.4, "BC_FLAG": 1, "MERGE_SPLIT_ON": 0, "eq_level": 0.0,
         "DT_FIXED": 0.0, "NSTEPS": FOREVER, "ms_alpha": 0.9, "ms_beta": 0.30,
         "ms_split_hp_min": 0.0, "ms_shear_split": 1e30, "ms_hp_min": 0.05, "ms_max_dv": 0.01,
         "ms_min_level": -2, "ms_max_level": 2, "ms_min_particles_per_cell": 2,
         "ms_call_interval": 10, "ms_max_ops": 1e9, "ms_pair_dist": 0.0, "ms_variant": 0,
         "ms_stretch_thresh": 1e7}
    s.update(kw)
    return s


def _particles(x, y, hp, area, rho):
    z = np.zeros(x.size)
    Ap = np.full(x.size, area)
    Vp = Ap * hp
    Mp = rho * Vp
    return {"x": x, "y": y, "Mp": Mp, "Ap": Ap, "vpx": z, "vpy": z, "hp": hp, "mom_px": z * Mp,
            "mom_py": z * Mp, "Vp": Vp}


def _lattice(xs, ys):
    """All pairs, y fastest."""
    return np.repeat(xs, ys.size), np.tile(ys, xs.size)


def _bumps(n, h, slope, bumps, amp, sig, rng):
    """Z = slope*(L - x) + Gaussian bumps and its gradient, node r + c*(n+1)."""
    x = np.arange(n + 1) * h
    A, S = rng.uniform(*amp, bumps), rng.uniform(*sig, bumps)
    cx, cy = rng.uniform(0, n * h, bumps), rng.uniform(0, n * h, bumps)
    dx, dy = x[:, None] - cx, x[:, None] - cy
    ex, ey = A * np.exp(-(dx ** 2) / (2 * S ** 2)), np.exp(-(dy ** 2) / (2 * S ** 2))
    Z = ex @ ey.T + slope * (n * h - x)[:, None]
    gx = (-ex * dx / S ** 2) @ ey.T - slope
    gy = ex @ (-ey * dy / S ** 2).T
    return {"Z": Z.reshape(-1), "dZdx": gx.reshape(-1), "dZdy": gy.reshape(-1)}


def _ellipse(n, h, ppc, cx, cy, a, b, peak):
    """ppc x ppc particles per cell inside an ellipse, parabolic depth."""
    offs = (np.arange(ppc) + 0.5) / ppc * h

    def axis(c, w):
        cells = np.arange(max(math.floor((c - w) / h), 0), min(math.ceil((c + w) / h), n))
        return (cells[:, None] * h + offs).reshape(-1)

    xs, ys = axis(cx, a), axis(cy, b)
    r2 = ((xs - cx) / a)[:, None] ** 2 + ((ys - cy) / b)[None, :] ** 2
    ix, iy = np.nonzero(r2 < 1.0)
    return xs[ix], ys[iy], peak * (1.0 - r2[ix, iy])


def _dam(case, rng):
    n, h = case["cells"], 0.25
    offs = np.array([0.25, 0.75]) * h
    x, y = _lattice((np.arange(n // 4)[:, None] * h + offs).reshape(-1),
                    (np.arange(n)[:, None] * h + offs).reshape(-1))
    x = x + rng.uniform(-0.1, 0.1, x.size) * h
    y = y + rng.uniform(-0.1, 0.1, x.size) * h
    arrays = _particles(x, y, rng.uniform(0.95, 1.05, x.size), h * h / 4, 1000.0)
    for k in ("Z", "dZdx", "dZdy"):
        arrays[k] = np.zeros((n + 1) ** 2)
    return arrays, _scalars(Nex=n, Ney=n, hx=h, hy=h, BINGHAM_ON=0.0, FRICTION_ON=0.0,
                            DT_FIXED=1e-3)


def _slab(case, rng):
    n, s = int(round(math.sqrt(case["n"]) / 2)), 0.5
    slope = math.tan(math.radians(rng.uniform(1.0, 3.0)))
    xs = 1.0 + s / 2 + s * np.arange(2 * (n - 2))
    x, y = _lattice(xs, xs)
    hp = rng.uniform(4.0, 6.0) + rng.uniform(-0.01, 0.01, x.size)
    arrays = _particles(x, y, hp, s * s, 1200.0)
    nodes = np.repeat(np.arange(n + 1.0), n + 1)
    arrays.update(Z=100.0 - slope * nodes, dZdx=np.full(nodes.size, -slope),
                  dZdy=np.zeros(nodes.size))
    return arrays, _scalars(Nex=n, Ney=n, rho=1200.0, mu=2000.0, DT_FIXED=1e-3)


def _lake(case, rng):
    n, L = case["cells"], 10.0
    h = L / n
    amp, cx, cy = rng.uniform(3.0, 6.0), rng.uniform(4.0, 6.0), rng.uniform(4.0, 6.0)

    def bed(x, y):
        return amp * np.exp(-0.4 * ((x - cx) ** 2 + (y - cy) ** 2))

    xs = case["spacing"] * np.arange(int(L / case["spacing"]) + 1)
    x, y = _lattice(xs, xs)
    X, Y = _lattice(np.arange(n + 1) * h, np.arange(n + 1) * h)
    Z = bed(X, Y)
    arrays = _particles(x, y, 10.0 - bed(x, y), case["spacing"] ** 2, 1200.0)
    arrays.update(Z=Z, dZdx=-0.8 * (X - cx) * Z, dZdy=-0.8 * (Y - cy) * Z)
    return arrays, _scalars(Nex=n, Ney=n, hx=h, hy=h, rho=1200.0, BINGHAM_ON=0.0,
                            FRICTION_ON=0.0, CFL=0.1, BC_FLAG=0, eq_level=10.0)


def _mudflow(case, rng):
    n, h = case["cells"], case["h"]
    s = n * h / 1024.0
    arrays = _particles(*_ellipse(n, h, 4, 0.5 * n * h, n * h - 150.0 * s, 200.0 * s, 100.0 * s,
                                  5.0), (h / 4) ** 2, 1800.0)
    arrays.update(_bumps(n, h, 0.3, 32, (0.0, 20.0 * min(s, 1.0)), (10.0 * s, 60.0 * s), rng))
    sc = _scalars(Nex=n, Ney=n, hx=h, hy=h, rho=1800.0, xi=500.0, tauy=rng.uniform(300.0, 700.0))
    if case["kind"] == "mergesplit":
        a0 = (h / 4) ** 2
        sc.update(MERGE_SPLIT_ON=1, ms_alpha=math.sqrt(2.0 * a0) / h,
                  ms_beta=math.sqrt(0.5 * a0) / h, ms_pair_dist=0.25)
    return arrays, sc


def _member(size_rng, rng, fixed, t_end):
    """One scenario of a batch: its size from size_rng, its values from rng."""
    n = int(round(math.exp(size_rng.uniform(math.log(64), math.log(512)))))
    frac, ratio = size_rng.uniform(0.02, 0.10), size_rng.uniform(1.0, 2.0)
    u, v = size_rng.uniform(0.0, 1.0), size_rng.uniform(0.0, 1.0)
    b = math.sqrt(frac / (math.pi * ratio)) * n
    a = min(ratio * b, 0.45 * n)
    x, y, hp = _ellipse(n, 1.0, 2, a + 1.0 + u * max(n - 2 * a - 2.0, 0.0),
                        b + 1.0 + v * max(n - 2 * b - 2.0, 0.0), a, b, rng.uniform(2.0, 8.0))
    rho = rng.uniform(1500.0, 2200.0)
    arrays = _particles(x, y, hp, 0.25, rho)
    arrays.update(_bumps(n, 1.0, rng.uniform(0.2, 0.5), 8, (0.0, 15.0), (5.0, 40.0), rng))
    return arrays, _scalars(Nex=n, Ney=n, rho=rho, xi=rng.uniform(200.0, 2000.0),
                            mu=rng.uniform(10.0, 200.0), phi=rng.uniform(15.0, 35.0),
                            tauy=rng.uniform(100.0, 2000.0), DT_FIXED=fixed, T=t_end)


def _members(case, seed):
    sizes, rng = np.random.default_rng(case["mix"]), np.random.default_rng(seed)
    if case["kind"] == "ensemble":
        return [_member(sizes, rng, 0.02, 1e30) for _ in range(case["members"])]
    return [_member(sizes, rng, 0.0, case["t_end"]) for _ in range(case["requests"])]


_SINGLE = {"dam": _dam, "slab": _slab, "lake": _lake}


def _scenario(case, seed):
    return _SINGLE.get(case["kind"], _mudflow)(case, np.random.default_rng(seed))


# ---------------------------------------------------------------------------
# the program around the entry points
# ---------------------------------------------------------------------------
def _pinned(a):
    p = pinned_array(a.size)
    p[:] = a
    return p


def prepare(case, seed):
    if case["kind"] in ("ensemble", "serving"):
        data = [DATA(a, s) for a, s in _members(case, seed)]
        st = {"case": case, "data": data}
        if case["kind"] == "ensemble":
            st["batch"] = Batch(sum(d.np for d in data), sum(d.nnodes for d in data), len(data),
                                precision=case["precision"])
        else:
            # room for about two thirds of the requests at a time, and always
            # for the largest of them
            sizes = [(390 * d.np / 0.55, 56 * d.nnodes / 0.45) for d in data]
            room = max(0.66 * max(map(sum, zip(*sizes))), 1.1 * max(map(max, sizes)))
            st["server"] = Server(room, max_scenarios=len(data), precision=case["precision"])
        return st
    arrays, scalars = _scenario(case, seed)
    d = DATA(arrays, scalars)
    solver = Solver(d, merge_split=case["kind"] == "mergesplit")
    st = {"case": case, "solver": solver, "np": d.np}
    room = d.np if case["kind"] != "mergesplit" else 2 * d.np
    names = FRAME if case["kind"] == "frame" else MOVING
    if case["kind"] == "restart":
        st["checkpoint"] = solver.get_state({k: pinned_array(d.np) for k in STATE_FIELDS})
        names = STATE_FIELDS
    else:
        st["input"] = [_pinned(arrays[k]) for k in UPLOAD]
        st["pointers"] = [a.ctypes.data_as(ctypes.POINTER(ctypes.c_double)) for a in st["input"]]
    st["out"] = {k: _pinned(np.zeros(room)) for k in names}
    return st


def _upload(st):
    """New particles for the solver, as its constructor uploads them."""
    s = st["solver"]
    if s.lib.dampm_upload_particles(s.h, st["np"], *st["pointers"]) != 0:
        raise RuntimeError(s.lib.dampm_last_error(s.h).decode())


def _run_ensemble(st):
    b = st["batch"]
    handles = [b.add(d) for d in st["data"]]
    b.step(st["case"]["steps"])
    out = {k: np.concatenate([b.download(h, k) for h in handles]) for k in DEPTHS}
    for h in handles:
        b.remove(h)
    b.compact()
    return out


def _run_serving(st):
    served = st["server"].run([Request(k, d, 0.0) for k, d in enumerate(st["data"])])
    return {"status": np.array([r.status == "done" for r in served]),
            "results": [r.result for r in served]}


def run(st):
    case = st["case"]
    kind, steps = case["kind"], case["steps"] if "steps" in case else 0
    if kind == "ensemble":
        return _run_ensemble(st)
    if kind == "serving":
        return _run_serving(st)
    s, out = st["solver"], st["out"]
    if kind == "restart":
        s.set_state(st["checkpoint"])
        s.step(steps)
        return s.get_state(out)
    _upload(st)
    if kind == "frame":
        s.step(steps - 2)
        s.lib.dampm_record_outputs(s.h, 1)
        s.step(1)
        s.stage_download(out)
        s.step(1)
        s.lib.dampm_record_outputs(s.h, 0)
        nodes = {k: s.download_nodal(k) for k in FRAME_NODES}
        s.staged_wait()
        return {"particles": out, "nodes": nodes}
    s.step(steps)
    s.stage_download(out)
    s.staged_wait()
    return {"particles": out, **s.status()}


def _counts(case):
    """(particles, nodes) of a case."""
    k = case["kind"]
    if k in ("ensemble", "serving"):
        m = _members(case, 0)
        return sum(a["x"].size for a, _ in m), sum(a["Z"].size for a, _ in m)
    n = case.get("cells") or int(round(math.sqrt(case["n"]) / 2))
    if k == "dam":
        return n * n, (n + 1) ** 2
    if k == "slab":
        return (2 * (n - 2)) ** 2, (n + 1) ** 2
    if k == "lake":
        return (int(10.0 / case["spacing"]) + 1) ** 2, (n + 1) ** 2
    # the ellipse covers pi * 200 * 100 of 1024 * 1024, 16 particles per cell
    return int(16 * math.pi * 20000 / 1024 ** 2 * n * n), (n + 1) ** 2


def work(case):
    """Per step each particle's state is read (11 values) and its moving part
    written (8), the bed is read and the nodal velocities written and read
    (per node that the flow touches, a quarter of a particle's share); about
    580 operations a particle.  A serving request takes about 30 steps per
    second of simulated time."""
    particles, _ = _counts(case)
    steps = case["steps"] if "steps" in case else 30 * case["t_end"]
    real = 4 if case.get("precision") == "fp32" else 8
    return {"bytes": steps * particles * (19 + 5 / 4) * real, "flops": steps * particles * 580.0}


# ---------------------------------------------------------------------------
# the same equations in 64 bits, with torch
# ---------------------------------------------------------------------------
class _Reference:
    def __init__(self, arrays, sc):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.sc, self.it, self.t, self.dt = sc, 0, 0.0, 0.0
        for k, v in arrays.items():
            setattr(self, k, torch.from_numpy(np.ascontiguousarray(v)).to(dev))
        self.nr, self.nc = sc["Ney"], sc["Nex"]
        self.bin()
        zp = sum(N * self.Z[n] for N, n in zip(self.shape()[0], self.nodes))
        diff = sc["eq_level"] - zp
        zero = torch.zeros_like(zp)
        self.H = torch.where(diff > 0, diff, zero) if sc["eq_level"] > 0 else zero
        self.F11 = self.F22 = -0.5 * sc["rho"] * sc["g"] * self.still()
        self.F12, self.fbx, self.fby = zero, zero, zero

    def bin(self):
        sc = self.sc
        self.r = torch.clamp(torch.floor(self.y / sc["hy"]), 0, self.nr - 1).long()
        self.c = torch.clamp(torch.floor(self.x / sc["hx"]), 0, self.nc - 1).long()
        n = self.r + self.c * (self.nr + 1)
        self.nodes = (n, n + 1, n + self.nr + 1, n + self.nr + 2)

    def shape(self):
        hx, hy = self.sc["hx"], self.sc["hy"]
        a = (self.x - self.c * hx) / hx
        b = (self.y - self.r * hy) / hy
        N = ((1 - a) * (1 - b), (1 - a) * b, a * (1 - b), a * b)
        Nx = (-(1 - b) / hx, -b / hx, (1 - b) / hx, b / hx)
        Ny = (-(1 - a) / hy, (1 - a) / hy, -a / hy, a / hy)
        return N, Nx, Ny

    def still(self):
        return torch.where(self.hp > 1e-10, self.hp - self.H * self.H / self.hp,
                           torch.zeros_like(self.hp))

    def time_step(self):
        sc = self.sc
        if sc["DT_FIXED"] > 0:
            return sc["DT_FIXED"]
        if self.it == 0:
            return 1e-3
        wave = math.sqrt(sc["g"] * float(self.hp.max()))
        cel = wave + max(float(self.vpx.abs().max()), float(self.vpy.abs().max()))
        return sc["CFL"] * min(sc["hx"], sc["hy"]) / (1e-2 + cel)

    def step(self):
        sc = self.sc
        dt = self.dt = self.time_step()
        self.it += 1
        self.bin()
        N, Nx, Ny = self.shape()

        def scatter(values):
            out = torch.zeros_like(self.Z)
            for n, v in zip(self.nodes, values):
                out.index_add_(0, n, v)
            return out

        dzx = sum(g * self.Z[n] for g, n in zip(Nx, self.nodes))
        dzy = sum(g * self.Z[n] for g, n in zip(Ny, self.nodes))
        wb = torch.where(self.hp > 1e-10, 1 - self.H / self.hp, torch.ones_like(self.hp))
        M = scatter([w * self.Mp for w in N])
        px, py = scatter([w * self.mom_px for w in N]), scatter([w * self.mom_py for w in N])
        fx = -sc["g"] * self.Vp * sc["rho"] * dzx * wb + self.Ap * self.fbx
        fy = -sc["g"] * self.Vp * sc["rho"] * dzy * wb + self.Ap * self.fby
        fx = scatter([w * fx - (gx * self.F11 + gy * self.F12) * self.Vp
                      for w, gx, gy in zip(N, Nx, Ny)])
        fy = scatter([w * fy - (gx * self.F12 + gy * self.F22) * self.Vp
                      for w, gx, gy in zip(N, Nx, Ny)])
        act = M > 1e-2
        Ms = torch.where(act, M, torch.ones_like(M))
        vx = torch.where(act, dt * fx / Ms + (dt * fx + px) / Ms, torch.zeros_like(M))
        vy = torch.where(act, dt * fy / Ms + (dt * fy + py) / Ms, torch.zeros_like(M))
        if sc["BC_FLAG"]:
            vx.view(self.nc + 1, -1)[[0, 1, self.nc - 1, self.nc]] = 0
            vy.view(self.nc + 1, -1)[:, [0, 1, self.nr - 1, self.nr]] = 0
        at_x, at_y = [vx[n] for n in self.nodes], [vy[n] for n in self.nodes]
        u = self.vpx = sum(w * a for w, a in zip(N, at_x))
        v = self.vpy = sum(w * a for w, a in zip(N, at_y))
        eps = 1e-10
        self.x = torch.clamp(self.x + dt * u, eps, self.nc * sc["hx"] - eps)
        self.y = torch.clamp(self.y + dt * v, eps, self.nr * sc["hy"] - eps)
        _, Nx, Ny = self.shape()  # the new position in the old cell
        ux, uy = (sum(g * a for g, a in zip(G, at_x)) for G in (Nx, Ny))
        wx, wy = (sum(g * a for g, a in zip(G, at_y)) for G in (Nx, Ny))
        self.hp = torch.clamp(self.hp / (1 + dt * (ux + wy)), min=1e-2)
        self.stress(ux, uy, wx, wy)
        self.mom_px, self.mom_py = u * self.Mp, v * self.Mp
        self.Ap = torch.where(self.hp > 1e-2, self.Vp / self.hp, torch.zeros_like(self.hp))
        self.friction()
        self.t += dt

    def stress(self, ux, uy, wx, wy):
        sc, u, v, hp = self.sc, self.vpx, self.vpy, self.hp
        speed = torch.sqrt(u * u + v * v)
        alf = torch.where(hp > 1e-3, 6 * sc["mu"] * speed / ((hp + 0.001) * sc["tauy"]), 0 * hp)
        A, B, C = 1.5, -114.0 / 32.0 - alf, 65.0 / 32.0
        plug = (-B - torch.sqrt(B * B - 4 * A * C)) / (2 * A)
        zx, zy = (torch.where(hp > 1e-3, 1.5 / (2 + plug) * (w / (hp + 0.001)), 0 * hp)
                  for w in (u, v))
        xy = 0.5 * (uy + wx)
        second = 0.5 * (ux * ux + wy * wy + (ux + wy) ** 2) + zx * zx + zy * zy + xy * xy
        safe = torch.where(second != 0, second, torch.ones_like(second))
        k = torch.where(second != 0, sc["tauy"] / torch.sqrt(safe) + 2 * sc["mu"], 0 * second)
        pres = 0.5 * sc["rho"] * sc["g"] * self.still()
        self.F11 = sc["BINGHAM_ON"] * k * ux - pres
        self.F12 = sc["BINGHAM_ON"] * k * xy
        self.F22 = sc["BINGHAM_ON"] * k * wy - pres

    def friction(self):
        sc, u, v, hp = self.sc, self.vpx, self.vpy, self.hp
        speed = torch.sqrt(u * u + v * v)
        moving = (speed > 1e-10) & (sc["FRICTION_ON"] > 0)
        s = (sc["rho"] * sc["g"] * hp * math.tan(sc["phi"] * math.pi / 180.0)
             + sc["rho"] * sc["g"] * speed * speed / sc["xi"])
        per = torch.where(moving, -sc["FRICTION_ON"] * s
                          / torch.where(moving, speed, torch.ones_like(speed)), 0 * speed)
        self.fbx, self.fby = per * u, per * v

    def field(self, name):
        v = getattr(self, {"F_11": "F11", "F_12": "F12", "F_22": "F22"}.get(name, name))
        return v.cpu().numpy()


def _advance(arrays, scalars, steps):
    r = _Reference(arrays, scalars)
    for _ in range(steps):
        r.step()
    return r


def exact(case, seed):
    kind = case["kind"]
    if kind in ("mergesplit", "serving"):
        return None  # which particles merge, and when a request ends, is no computed number
    if kind in ("mudflow", "restart") and case["steps"] > 10:
        return None  # the yield stress has amplified the last digit of any arithmetic to percents
    if kind == "ensemble":
        m = _members(case, seed)
        if sum(a["x"].size for a, _ in m) > 2_000_000 or len(m) * case["steps"] > 13_000:
            return None
        refs = [_advance(a, s, case["steps"]) for a, s in m]
        return {k: np.concatenate([r.field(k) for r in refs]) for k in DEPTHS}
    arrays, scalars = _scenario(case, seed)
    if kind == "restart":
        r = _advance(arrays, scalars, case["steps"])
        return {k: r.field(k) for k in STATE_FIELDS}
    if kind == "frame":  # the particles as the last step begins
        r = _advance(arrays, scalars, case["steps"] - 1)
        return {"particles": {k: r.field(k) if k in MOVING else None for k in FRAME},
                "nodes": {k: None for k in FRAME_NODES}}
    r = _advance(arrays, scalars, case["steps"])
    return {"particles": {k: r.field(k) for k in MOVING}, "it": r.it, "t": r.t, "dt": r.dt,
            "np": int(r.x.numel())}
