"""The work whose speed is measured: what a user of the framework has it do,
through its public entry points (the simFDTD ops, StepN, Batch, Server).

A case is one run of a simulation, or of several: `prepare` sets the handles
up (grid, media, sources, probes: what a program has in hand before it
steps), `run` resets the fields, takes every step and reads the results
back: the probe record and the six fields.  The field buffers are the
program's own and are filled through the C ABI (fdtd_output_vis), as a C
program does it.  The long 512-class run does not reset: it goes on from
where the last pass ended.  The served case and the whole-solve case pay for
set-up inside the pass, as their users do.

`exact` restates the scheme (Yee curl, CPML, TF/SF modes 1-5, current
source, per-cell magnetic media) in float64 with plain torch and numpy.
"""
import ctypes
import math

import numpy as np
import torch

from maxwell_solver_gb300 import simFDTD
from maxwell_solver_gb300._native import load
from maxwell_solver_gb300.batch import Batch
from maxwell_solver_gb300.serve import Server

C0 = 299792458.0
MU0 = 4 * math.pi * 1e-7
EPS0 = 1 / C0 / C0 / MU0
FIELDS = 6


def _case(name, kind, dims, steps, pml, mode, media, probes=8, current=0, magnetic=False, count=1,
          warm=0):
    """kind: step (StepN), ops (one call per reference op), solve (StepN with
    the set-up and deletion inside the pass), batch, serve.  mode: TF/SF 0-5.
    media: spheres, layers, cells (another value in every cell).  current: 0,
    or the field component (1-3) driven by a line current.  warm: steps taken
    in prepare by a run that goes on from pass to pass."""
    return {"name": name, "kind": kind, "I": dims[0], "J": dims[1], "K": dims[2], "steps": steps,
            "pml": pml, "mode": mode, "media": media, "probes": probes, "current": current,
            "magnetic": magnetic, "count": count, "warm": warm}


def listed():
    return [
        # a script's own time loop, six op calls a step, on the smallest grid
        # used: call overhead and launches
        _case("op_loop_48", "ops", (48, 44, 40), 60, 10, 3, "spheres"),
        # the 64^3 configuration: 500 steps in one call, bound by latency
        _case("run_64", "step", (64, 64, 64), 500, 10, 3, "spheres"),
        # a geoelectric script's loop: layered earth, a line current added by
        # an op of its own in every step, no plane wave
        _case("op_loop_current", "ops", (120, 104, 96), 150, 10, 0, "layers", current=2),
        # odd sizes, oblique incidence: a medium scattering run
        _case("run_odd_oblique", "step", (131, 117, 109), 300, 9, 5, "spheres", probes=16),
        # magnetic media per cell
        _case("run_magnetic", "step", (160, 144, 130), 200, 10, 2, "spheres", magnetic=True),
        # an inhomogeneous medium without repeats: coefficients per cell
        _case("run_inhomogeneous", "step", (176, 160, 129), 200, 12, 4, "cells"),
        # the 256^3 configuration: oblique wave on spheres, 64 probes
        _case("run_256", "step", (256, 256, 256), 300, 12, 5, "spheres", probes=64),
        # a large flat layered model driven by a line current
        _case("run_current_flat", "step", (400, 360, 120), 150, 16, 0, "layers", current=1),
        # the 512-class configuration, going on through its 4000 steps
        _case("run_512", "step", (512, 512, 448), 200, 16, 1, "layers", probes=256, warm=50),
        # many small solves of different sizes and lengths advanced together
        _case("batch_48", "batch", (32, 0, 128), 600, 8, 5, "spheres", probes=0, count=48),
        # a queue of requests, set-up and results included
        _case("serve_10", "serve", (48, 0, 160), 500, 10, 5, "spheres", count=10),
        # one solve from its material arrays to its results
        _case("solve_200", "solve", (200, 185, 168), 250, 10, 1, "spheres", probes=32),
    ]


def draw(rng):
    kind = rng.choices(("step", "ops", "solve", "batch", "serve"), (8, 2, 2, 2, 1))[0]
    pml = rng.randint(8, 16)
    if kind in ("batch", "serve"):
        lo = rng.randint(32, 56)
        c = _case("", kind, (lo, 0, rng.randint(lo + 24, 128 if kind == "batch" else 160)),
                  rng.randint(200, 600), rng.randint(8, 10), 5, "spheres",
                  probes=0 if kind == "batch" else 8,
                  count=rng.randint(8, 28) if kind == "batch" else rng.randint(4, 10))
        del c["name"]
        return c
    top = {"step": 400, "ops": 160, "solve": 224}[kind]
    base = math.exp(rng.uniform(math.log(44), math.log(top)))
    dims = tuple(max(2 * pml + 16, int(base * rng.uniform(0.8, 1.2))) for _ in range(3))
    cells = dims[0] * dims[1] * dims[2]
    steps = max(20, min(500 if kind != "ops" else 120, int(4e9 / cells * rng.uniform(0.4, 1.0))))
    mode = rng.choice((0, 1, 2, 3, 4, 5, 5))
    media = rng.choice(("spheres", "spheres", "layers", "cells") if cells < 2e7
                       else ("spheres", "layers"))
    c = _case("", kind, dims, steps, pml, mode, media, probes=rng.choice((0, 8, 64)),
              current=0 if mode else rng.randint(1, 3),
              magnetic=cells < 2e7 and rng.random() < 0.15)
    del c["name"]
    return c


# ------------------------------------------------------------------ inputs

def _spec(case, seed, member=0):
    """The inputs of one simulation, from the seed alone."""
    r = np.random.default_rng([int(seed), int(member), 17])
    s = {k: case[k] for k in ("steps", "pml", "mode", "media", "probes", "current", "magnetic")}
    if case["kind"] in ("batch", "serve"):
        # the mix (sizes, lengths, media kinds) belongs to the case; what is
        # computed in it to the seed
        q = np.random.default_rng([int(member), case["I"], case["K"], case["count"]])
        s["dims"] = tuple(int(x) for x in q.integers(case["I"], case["K"] + 1, 3))
        s["steps"] = int(q.integers(case["steps"] // 2, case["steps"] + 1))
        if case["kind"] == "serve" and q.random() < 0.5:
            s["media"], s["mode"] = "layers", 1
    else:
        s["dims"] = (case["I"], case["J"], case["K"])
    I, J, K = s["dims"]
    p = s["pml"]
    s["delX"], s["fctr"] = 1e-3, float(np.float32(r.uniform(10e9, 30e9)))
    s["delT"] = 0.99 * s["delX"] / (math.sqrt(3.0) * C0)
    s["T"] = 4000 if case["warm"] else s["steps"]
    s["width"] = p + 5
    s["angles"] = (float(r.uniform(0.2, math.pi - 0.2)), float(r.uniform(0, 2 * math.pi)),
                   float(r.uniform(0, 2 * math.pi)))
    # media as shape rows [kind, eps_r, sigma, g0..g5]
    rows = []
    if s["media"] == "layers":
        top = K - p - 2 - int(0.45 * K)
        while top > 0:
            lo = max(0, top - int(r.integers(10, 81)))
            rows.append([2, np.float32(r.uniform(5, 30)), np.float32(10 ** r.uniform(-4, 0)),
                         lo, top, 0, 0, 0, 0])
            top = lo
    else:
        room = (min(I, J, K) - 2 * (p + 2)) / 2
        for _ in range(min(40, 2 + I * J * K // 400000)):
            rad = min(float(r.uniform(4, 20)), max(room - 1, 1.0))
            c = [float(r.uniform(p + 2 + rad, n - p - 2 - rad)) for n in (I, J, K)]
            rows.append([1, np.float32(r.uniform(1.5, 10)), np.float32(10 ** r.uniform(-4, 0)),
                         *c, rad, 0, 0])
    s["rows"] = rows
    if s["media"] == "cells":
        s["eps"] = [r.uniform(1, 10, I * J * K).astype(np.float32) for _ in range(3)]
        s["sig"] = [(10 ** r.uniform(-4, -1, I * J * K)).astype(np.float32) for _ in range(3)]
    if s["magnetic"]:
        mu = np.ones((K, J, I), dtype=np.float32)
        mu[K // 3:2 * K // 3, J // 3:2 * J // 3, I // 3:2 * I // 3] = r.uniform(1.5, 5)
        sm = np.where(mu > 1, np.float32(r.uniform(10, 100)), np.float32(0)).astype(np.float32)
        s["mu"], s["sm"] = mu.ravel(), sm.ravel()
    n = np.arange(s["T"], dtype=np.float64)
    tau = 20.0 / math.pi * s["delX"] / C0
    t = n * s["delT"] - (3 + r.uniform(0, 0.5)) * tau
    s["pw"] = (-(t / tau) * np.exp(-(t / tau) ** 2) * r.uniform(0.5, 2)).astype(np.float32)
    s["cur"] = np.exp(-(n - 20 - r.uniform(0, 4)) ** 2 / 50).astype(np.float32)
    # a line of cells along the driven component, under the centre
    m = (I // 2, J // 2, K // 2)
    box = [m[0], m[0], m[1], m[1], m[2], m[2]]
    if s["current"]:
        a = s["current"] - 1
        w = s["dims"][a]
        box[2 * a], box[2 * a + 1] = w // 4, w - w // 4
    s["box"] = box
    lim = [d - 2 * p for d in s["dims"]]
    s["loc"] = np.stack([r.integers(1, max(2, lim[a] - 1), s["probes"]) for a in range(3)],
                        axis=1).astype(np.int32)
    return s


def _create(s, arrays=False):
    """A handle set up for the spec.  arrays: the media as UpdateMaterial
    arrays (s["media6"]) instead of shapes."""
    I, J, K = s["dims"]
    P = simFDTD("CreateSimulation")
    simFDTD("SetParams", P, np.float64([s["pml"], s["width"]]))
    simFDTD("SetConst", P, np.float32([s["fctr"], s["delX"], s["delT"]]),
            np.int32([s["T"], I, J, K, s["probes"]]))
    simFDTD("SetSource", P, s["cur"])
    if s["probes"]:
        simFDTD("SetAntennaLocations", P, np.asfortranarray(s["loc"]))
    if s["media"] == "cells":
        for a in range(3):
            simFDTD("UpdateMaterial", P, np.int32(1 + a), s["sig"][a])
            simFDTD("UpdateMaterial", P, np.int32(4 + a), s["eps"][a])
    elif arrays:
        for f in range(6):
            simFDTD("UpdateMaterial", P, np.int32(1 + f), s["media6"][f])
    else:
        simFDTD("SetShapes", P, np.float32([1, 0]), np.float64(s["rows"]).reshape(-1, 9))
    simFDTD("ReadySimulation", P)
    if s["magnetic"]:
        simFDTD("SetMagnetic", P, s["mu"], s["mu"], s["mu"], s["sm"], s["sm"], s["sm"])
    if s["mode"] == 5:
        simFDTD("SetIncidence", P, np.float64(s["angles"]))
    if s["mode"]:
        simFDTD("Init1D", P, np.float32(1), s["pw"])
    return P


class _State:
    """The specs, the handles and the buffers one program holds."""

    def __init__(self, case, seed):
        self.case, self.lib = case, load()
        self.specs = [_spec(case, seed, m) for m in range(case["count"])]
        self.P, self.batch, self.server, self.at = [], None, None, 0
        kind = case["kind"]
        if kind == "serve":
            self.server = Server(hbm_budget=64 << 30)
            return
        # page-locked, as a program that reads fields again and again keeps them
        self.fields = [[torch.zeros(int(np.prod(s["dims"])), dtype=torch.float32,
                                    pin_memory=torch.cuda.is_available()).numpy()
                        for _ in range(1 if kind == "batch" else FIELDS)] for s in self.specs]
        if kind == "solve":
            s = self.specs[0]
            if s["media"] != "cells":
                eps, sig = (x.cpu().numpy().ravel() for x in _shapes_on_grid(s, torch.float32))
                s["media6"] = [sig, sig, sig, eps, eps, eps]
            return
        self.P = [_create(s) for s in self.specs]
        if kind == "batch":
            self.batch = Batch()
        if case["warm"]:
            simFDTD("StepN", self.P[0], np.int32([0, case["warm"], case["mode"]]))
            self.at = case["warm"]

    def read(self, m, P, ez_only=False):
        """The probe record and the six fields of one handle (or Ez alone)."""
        s, f = self.specs[m], self.fields[m]
        out = {}
        if s["probes"]:
            out["probes"] = simFDTD("OutputProbes", P, np.uint32(s["T"] * s["probes"] * 6))
        for c in (2,) if ez_only else range(FIELDS):
            to = f[0 if ez_only else c]
            if self.lib.fdtd_output_vis(int(P[0]), to.ctypes.data_as(ctypes.c_void_p), to.size,
                                        c + 1):
                raise RuntimeError(self.lib.fdtd_last_error())
            out["EH"[c // 3] + "xyz"[c % 3]] = to
        return out

    def __del__(self):
        if self.batch is not None:
            self.batch.close()
        if self.server is not None:
            self.server.close()
        for P in self.P:
            simFDTD("DeleteSimulation", P)


def prepare(case, seed):
    return _State(case, seed)


def _op_loop(s, P):
    """The reference scripts' time loop."""
    mode, cur, box = s["mode"], s["current"], np.int32(s["box"])
    for n in range(s["steps"]):
        simFDTD("UpdateH_All", P)
        if mode:
            simFDTD("UpdateH_PlaneWave", P, np.int32([n, mode]))
        simFDTD("UpdateH_PML", P)
        simFDTD("UpdateE_All", P)
        if mode:
            simFDTD("UpdateE_PlaneWave", P, np.int32([n, mode]))
        simFDTD("UpdateE_PML", P)
        if cur:
            simFDTD("AddCurrents", P, np.int32([n, cur]), box)


def _step_n(s, P, first, count):
    at = np.int32([first, count, s["mode"]])
    if s["current"]:
        simFDTD("StepN", P, at, np.int32([s["current"], *s["box"]]))
    else:
        simFDTD("StepN", P, at)


def run(state):
    case, specs = state.case, state.specs
    kind = case["kind"]
    if kind == "serve":
        srv = state.server
        tickets = [srv.submit_request(s["dims"], s["steps"], s["fctr"], s["delX"], s["delT"],
                                      s["pml"], s["mode"], s["pw"], s["rows"], (1.0, 0.0),
                                      s["loc"], 3, angles=s["angles"]) for s in specs]
        done = [srv.result(t) for t in tickets]
        return [{"probes": d["probes"], "Ez": d["field"]} for d in done]
    if kind == "batch":
        for s, P in zip(specs, state.P):
            simFDTD("ResetFieldAll", P)
            state.batch.add(P, 0, s["steps"], s["mode"])
        state.batch.run()
        state.batch.clear()
        return [state.read(m, P, ez_only=True) for m, P in enumerate(state.P)]
    s = specs[0]
    if kind == "solve":
        P = _create(s, arrays=True)
        _step_n(s, P, 0, s["steps"])
        out = state.read(0, P)
        simFDTD("DeleteSimulation", P)
        return out
    P = state.P[0]
    if case["warm"] and state.at + s["steps"] <= s["T"]:
        _step_n(s, P, state.at, s["steps"])
        state.at += s["steps"]
        return state.read(0, P)
    simFDTD("ResetFieldAll", P)
    if kind == "ops":
        _op_loop(s, P)
    else:
        _step_n(s, P, 0, s["steps"])
        state.at = s["steps"]
    return state.read(0, P)


def work(case):
    """Per step every field is read and written once (48 B a cell), the
    coefficients are read (a 2-byte material id, six floats where every cell
    has its own, two more bytes for magnetic media) and the CPML's recurrences
    are read and written; the fields are read back once.  Operations: the two
    curls' 36 a cell."""
    total_b = total_f = 0
    for m in range(case["count"]):
        q = _spec({**case, "media": "layers", "magnetic": False}, 0, m)
        I, J, K = q["dims"]
        cells, p = I * J * K, q["pml"]
        coef = (24 if case["media"] == "cells" else 2) + (2 if case["magnetic"] else 0)
        psi = 2 * 2 * p * (J * K + I * K + I * J) * 16
        total_b += q["steps"] * (cells * (48 + coef) + psi)
        total_b += cells * 4 * (1 if case["kind"] in ("batch", "serve") else FIELDS)
        total_f += q["steps"] * cells * 36
    return {"bytes": total_b, "flops": total_f}


# ------------------------------------------------------------------- float64

def _shapes_on_grid(s, dt):
    """eps_r, sigma as [K, J, I] tensors from the spec's shape rows."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    I, J, K = s["dims"]
    ax = [torch.arange(n, device=dev, dtype=torch.float64) for n in (I, J, K)]
    eps = torch.ones((K, J, I), device=dev, dtype=dt)
    sig = torch.zeros((K, J, I), device=dev, dtype=dt)
    for kind, e, g, *a in s["rows"]:
        if kind == 1:
            d = [((x + 0.5 - c) ** 2) for x, c in zip(ax, a)]
            m = (d[0][None, None, :] + d[1][None, :, None]) + d[2][:, None, None] <= a[3] * a[3]
            eps[m], sig[m] = float(e), float(g)
        else:
            eps[int(a[0]):int(a[1])], sig[int(a[0]):int(a[1])] = float(e), float(g)
    return eps, sig


def _cpml(s):
    """b, c at the slab positions of E and H (2p each)."""
    p, dx, dt = s["pml"], float(np.float32(s["delX"])), float(np.float32(s["delT"]))
    smax = 0.8 * 4 / (math.sqrt(MU0 / EPS0) * dx)

    def at(ns, na):
        sg, al = smax * (ns / (p - 1)) ** 3, 0.08 * (na / (p - 1))
        b = math.exp(-(sg + al) * dt / EPS0)
        return b, (sg / (sg + al) * (b - 1) if sg + al else 0.0)

    e = [at(p - i - 1, i) for i in range(p)]
    h = [at(p - i - 1.5, i + 0.5) for i in range(p - 1)] + [(0.0, 0.0)]
    e, h = e + e[::-1], h + h[:p - 1][::-1] + [(0.0, 0.0)]
    return [np.array([v[k] for v in t]) for t in (e, h) for k in (0, 1)]


def _line_axis(s, inverse, bE, cE, bH, cH):
    """The axis modes' 1D run: E before each step, H after its update."""
    p, T, S = s["pml"], s["T"], max(s["dims"])
    dx, dt = float(np.float32(s["delX"])), float(np.float32(s["delT"]))
    ce, ch = dt / EPS0 / dx, dt / MU0 / dx
    E, H, pE, pH = (np.zeros(n) for n in (S, S, 2 * p, 2 * p))
    oe, oh = np.zeros((T, S)), np.zeros((T, S))
    th = np.arange(2 * p - 1)
    te = np.arange(1, 2 * p)
    ih, ie = np.where(th < p, th, th + S - 2 * p), np.where(te < p, te, te + S - 2 * p)
    src = p + 3 if inverse else S - (p + 3)
    for n in range(T):
        oe[n] = E
        H[:-1] += ch * (E[1:] - E[:-1])
        pH[th] = bH[th] * pH[th] + cH[th] * (E[ih + 1] - E[ih])
        H[ih] += ch * pH[th]
        oh[n] = H
        E[1:] += ce * (H[1:] - H[:-1])
        pE[te] = bE[te] * pE[te] + cE[te] * (H[ie] - H[ie - 1])
        E[ie] += ce * pE[te]
        E[src] += float(s["pw"][n])
    return oe, oh


def _line_oblique(s, lo, hi):
    """The oblique wave's 1D run in its window, and the window's geometry."""
    t, f, q = s["angles"]
    dx, dt, T = float(np.float32(s["delX"])), float(np.float32(s["delT"])), s["T"]
    k = np.array([math.sin(t) * math.cos(f), math.sin(t) * math.sin(f), math.cos(t)])
    th = np.array([math.cos(t) * math.cos(f), math.cos(t) * math.sin(f), -math.sin(t)])
    e = math.cos(q) * th + math.sin(q) * np.array([-math.sin(f), math.cos(f), 0.0])
    span = float(np.sum(np.abs(k) * (np.array(hi) - np.array(lo))))
    r0 = [lo[a] if k[a] >= 0 else hi[a] for a in range(3)]
    dx1 = dx * math.sqrt(float(np.sum(k ** 4)))
    if C0 * dt / dx1 > 0.995:
        dx1 = C0 * dt / 0.995
    w = 2 * math.pi * float(np.float32(s["fctr"]))
    kn = w / C0
    rhs = (dx / (C0 * dt) * math.sin(w * dt / 2)) ** 2
    for _ in range(60):
        x = kn * k * dx / 2
        step = (np.sum(np.sin(x) ** 2) - rhs) / np.sum(k * dx * np.sin(x) * np.cos(x))
        kn -= step
        if abs(step) < 1e-15 * abs(kn):
            break
    speed = math.sin(w * dt / 2) * dx1 / (C0 * dt * math.sin(kn * dx1 / 2))
    if speed * C0 * dt / dx1 > 0.999:
        speed = 0.999 * dx1 / (C0 * dt)
    rho = dx / dx1
    x0, W = 4 * rho, math.ceil((span + 2.6) * rho + 4 * float(np.float32(rho))) + 4
    src = T + 8
    mb = src + 2
    n1 = mb + W + T + 8
    E, H = np.zeros(n1), np.zeros(n1)
    cE, cH = speed * dt / EPS0 / dx1, speed * dt / MU0 / dx1
    oe, oh = np.zeros((T, W)), np.zeros((T, W))
    for n in range(T):
        oe[n] = E[mb:mb + W]
        H[:-1] -= cH * (E[1:] - E[:-1])
        oh[n] = H[mb:mb + W]
        E[1:-1] -= cE * (H[1:-1] - H[:-2])
        E[src] += float(s["pw"][n]) * speed * dx / dx1
    return k, e, np.cross(k, e), r0, rho, x0, W, oe, oh


def _simulate(s, steps):
    """Fields [6][K, J, I] after `steps` steps and the probe record, float64."""
    f64 = torch.float64
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    I, J, K = s["dims"]
    p, dx, dt = s["pml"], float(np.float32(s["delX"])), float(np.float32(s["delT"]))
    if s["media"] == "cells":
        eps = [torch.tensor(x, device=dev, dtype=f64).view(K, J, I) for x in s["eps"]]
        sig = [torch.tensor(x, device=dev, dtype=f64).view(K, J, I) for x in s["sig"]]
        mat = [(2 * EPS0 * e, g * dt) for e, g in zip(eps, sig)]
    else:
        eps, sig = _shapes_on_grid(s, f64)
        mat = [(2 * EPS0 * eps, sig * dt)]
    den = torch.full((I,), 1 / dx, device=dev, dtype=f64)
    den[I - 1] = 0
    Ca = [(a - g) / (a + g) for a, g in mat]
    Cb = [2 * dt / (a + g) * den for a, g in mat]
    if len(mat) == 1:
        Ca, Cb = Ca * 3, Cb * 3
    del eps, sig, mat
    if s["magnetic"]:
        mu = torch.tensor(s["mu"], device=dev, dtype=f64).view(K, J, I)
        g = torch.tensor(s["sm"], device=dev, dtype=f64).view(K, J, I) * dt / (2 * MU0 * mu)
        Da, Db = (1 - g) / (1 + g), dt / (MU0 * mu) / (1 + g) / dx
    else:
        Da, Db = None, dt / MU0 / dx
    bE, cE, bH, cH = _cpml(s)
    vec = {k: torch.tensor(v, device=dev) for k, v in
           (("bE", bE), ("cE", cE), ("bH", bH), ("cH", cH))}
    F = [torch.zeros((K, J, I), device=dev, dtype=f64) for _ in range(6)]
    E, H = F[:3], F[3:]
    n = (I, J, K)

    def sl(axis, a, b, rest):
        """Slice [a, b) on the axis, `rest` on the others (tensor order)."""
        out = list(rest)
        out[2 - axis] = slice(a, b)
        return tuple(out)

    def shape(axis, v):
        return v.view([-1 if 2 - axis == d else 1 for d in range(3)])

    # the slabs of one axis: (first, last + 1, first table position)
    slabs_h = [[(0, p, 0), (m - p, m - 1, p)] for m in n]
    slabs_e = [[(1, p, 1), (m - p, m, p)] for m in n]
    psi = {}

    def recur(fam, axis, q, k, d, pos):
        b = shape(axis, vec["b" + fam][pos:pos + d.shape[2 - axis]])
        c = shape(axis, vec["c" + fam][pos:pos + d.shape[2 - axis]])
        key = (fam, axis, q, k)
        psi[key] = b * psi[key] + c * d if key in psi else c * d
        return psi[key]

    at = lambda C, w: C[w] if isinstance(C, torch.Tensor) else C  # noqa: E731
    hin = (slice(0, K - 1), slice(0, J - 1), slice(0, I - 1))
    ein = (slice(1, K - 1), slice(1, J - 1), slice(1, I - 1))

    def up(w, axis, by):
        w = list(w)
        w[2 - axis] = slice(w[2 - axis].start + by, w[2 - axis].stop + by)
        return tuple(w)

    lo = [s["width"]] * 3
    hi = [m - s["width"] - 1 for m in n]
    (i0, j0, k0), (i1, j1, k1) = lo, hi
    mode = s["mode"]
    if mode in (1, 2, 3, 4):
        oe, oh = (torch.tensor(v, device=dev) for v in _line_axis(s, mode == 4, bE, cE, bH, cH))
        off = max(n) - (K if mode < 3 else I)
        oe, oh = oe[:, off:], oh[:, off:]
    if mode == 5:
        kv, pe, ph, r0, rho, x0, W, oe, oh = _line_oblique(s, lo, hi)
        oe, oh = torch.tensor(oe, device=dev), torch.tensor(oh, device=dev)
        planes = []  # (family, slice, component, sign, window index, fraction, amplitude)
        for ax in range(3):
            u, v = (ax + 1) % 3, (ax + 2) % 3
            for side in (0, 1):
                for q, (ce, chh) in enumerate(((u, v), (v, u))):
                    sign = 1.0 if (q == 0) == (side == 0) else -1.0
                    end = [hi[a] + (0 if a == ce else 1) for a in range(3)]
                    ex = hi[ax] if side else lo[ax]
                    hx = hi[ax] if side else lo[ax] - 1
                    for fam, own, oth in (("H", hx, ex), ("E", ex, hx)):
                        half = [0.5 if (a == ce) == (fam == "H") else 0.0 for a in range(3)]
                        if fam == "E":
                            half = [0.0 if a == chh else 0.5 for a in range(3)]
                        x = torch.full((), x0 - (0.5 if fam == "E" else 0.0), device=dev, dtype=f64)
                        for a in range(3):
                            g = (torch.tensor([float(oth)], device=dev, dtype=f64) if a == ax else
                                 torch.arange(lo[a], end[a], device=dev, dtype=f64))
                            x = x + shape(a, rho * kv[a] * (g + half[a] - r0[a]))
                        m = x.floor().clamp(0, W - 2).long()
                        w = [slice(lo[a], end[a]) for a in (2, 1, 0)]
                        w[2 - ax] = slice(own, own + 1)
                        planes.append((fam, tuple(w), chh if fam == "H" else ce, sign, m, x - m,
                                       pe[ce] if fam == "H" else ph[chh]))

    def oblique(fam, step):
        row = (oe if fam == "H" else oh)[step]
        for g, w, c, sign, m, fr, amp in planes:
            if g != fam:
                continue
            inc = sign * amp * (row[m] + fr * (row[m + 1] - row[m]))
            if fam == "H":
                H[c][w] += at(Db, w) * inc
            else:
                E[c][w] += Cb[c][w] * inc

    def face(fam, c, sign, x, y, z, inc):
        """c of the family += sign * coefficient * inc over a box (slices or
        one index each)."""
        w = tuple(v if isinstance(v, slice) else slice(v, v + 1) for v in (z, y, x))
        if fam == "H":
            H[c][w] += sign * at(Db, w) * inc
        else:
            E[c][w] += sign * Cb[c][w] * inc

    X, Y, Z = (slice(a, b + 1) for a, b in zip(lo, hi))
    Xs, Ys, Zs = (slice(a, b) for a, b in zip(lo, hi))
    record = np.zeros((s["T"], s["probes"], 6))
    loc = torch.tensor(s["loc"].astype(np.int64) + p, device=dev)
    kept = []
    for step in range(steps):
        if s["probes"]:
            kept.append(torch.stack([f[loc[:, 2], loc[:, 1], loc[:, 0]] for f in F], dim=1))
        # H: curl, plane wave, CPML
        D = {}
        for a in range(3):
            for c in range(3):
                if c != a:
                    D[c, a] = E[c][up(hin, a, 1)] - E[c][hin]
        for c in range(3):
            a, b = (c + 1) % 3, (c + 2) % 3
            h = H[c][hin]
            if Da is not None:
                h *= Da[hin]
            h += at(Db, hin) * (D[a, b] - D[b, a])
        if mode == 5:
            oblique("H", step)
        elif mode == 3:
            r = oe[step]
            face("H", 0, 1, X, j0 - 1, Zs, r[X]), face("H", 0, -1, X, j1, Zs, r[X])
            face("H", 1, -1, i0 - 1, Y, Zs, r[i0]), face("H", 1, 1, i1, Y, Zs, r[i1])
        elif mode == 4:
            r = oe[step]
            face("H", 0, -1, X, Ys, k0 - 1, r[X]), face("H", 0, 1, X, Ys, k1, r[X])
            face("H", 2, 1, i0 - 1, Ys, Z, r[i0]), face("H", 2, -1, i1, Ys, Z, r[i1])
        elif mode == 1:
            r = oe[step]
            face("H", 0, -1, X, Ys, k0 - 1, r[k0]), face("H", 0, 1, X, Ys, k1, r[k1])
            z = r[Z].view(-1, 1, 1)
            face("H", 2, 1, i0 - 1, Ys, Z, z), face("H", 2, -1, i1, Ys, Z, z)
        elif mode == 2:
            r = oe[step]
            face("H", 1, 1, Xs, Y, k0 - 1, r[k0]), face("H", 1, -1, Xs, Y, k1, r[k1])
            z = r[Z].view(-1, 1, 1)
            face("H", 2, -1, Xs, j0 - 1, Z, z), face("H", 2, 1, Xs, j1, Z, z)
        for a in range(3):
            for q, (b, e, pos) in enumerate(slabs_h[a]):
                w = sl(a, b, e, hin)
                u, v = (a + 1) % 3, (a + 2) % 3
                # component u takes +dE_v along a, component v takes -dE_u
                H[u][w] += at(Db, w) * recur("H", a, q, 0, D[v, a][w], pos)
                H[v][w] -= at(Db, w) * recur("H", a, q, 1, D[u, a][w], pos)
        # E: curl, plane wave, CPML, current
        D = {}
        for a in range(3):
            for c in range(3):
                if c != a:
                    d = torch.zeros((K, J, I), device=dev, dtype=f64)
                    w = sl(a, 1, n[a], (slice(None),) * 3)
                    d[w] = H[c][w] - H[c][sl(a, 0, n[a] - 1, (slice(None),) * 3)]
                    D[c, a] = d
        for c in range(3):
            a, b = (c + 1) % 3, (c + 2) % 3
            w = [slice(None)] * 3
            w[2 - a] = w[2 - b] = slice(1, None)
            w = tuple(w)
            E[c][w] = Ca[c][w] * E[c][w] + Cb[c][w] * (D[b, a][w] - D[a, b][w])
        if mode == 5:
            oblique("E", step)
        elif mode == 3:
            r = oh[step]
            face("E", 0, 1, Xs, Y, k0, r[Xs]), face("E", 0, -1, Xs, Y, k1, r[Xs])
            face("E", 2, -1, i0, Y, Zs, r[i0 - 1]), face("E", 2, 1, i1, Y, Zs, r[i1])
        elif mode == 4:
            r = oh[step]
            face("E", 0, 1, Xs, j0, Z, r[Xs]), face("E", 0, -1, Xs, j1, Z, r[Xs])
            face("E", 1, -1, i0, Ys, Z, r[i0 - 1]), face("E", 1, 1, i1, Ys, Z, r[i1])
        elif mode == 1:
            r = oh[step]
            face("E", 1, -1, X, Ys, k0, r[k0 - 1]), face("E", 1, 1, X, Ys, k1, r[k1])
            z = r[Zs].view(-1, 1, 1)
            face("E", 2, 1, X, j0, Zs, z), face("E", 2, -1, X, j1, Zs, z)
        elif mode == 2:
            r = oh[step]
            face("E", 0, -1, Xs, Y, k0, r[k0 - 1]), face("E", 0, 1, Xs, Y, k1, r[k1])
            z = r[Zs].view(-1, 1, 1)
            face("E", 2, 1, i0, Y, Zs, z), face("E", 2, -1, i1, Y, Zs, z)
        for a in (1, 2, 0):
            for q, (b, e, pos) in enumerate(slabs_e[a]):
                w = sl(a, b, e, ein)
                u, v = (a + 1) % 3, (a + 2) % 3
                E[u][w] -= Cb[u][w] * recur("E", a, q, 0, D[v, a][w], pos)
                E[v][w] += Cb[v][w] * recur("E", a, q, 1, D[u, a][w], pos)
        if s["current"]:
            c, bx = s["current"] - 1, s["box"]
            w = tuple(slice(bx[2 * a], bx[2 * a + 1] + 1) for a in (2, 1, 0))
            E[c][w] -= Cb[c][w] * float(s["cur"][step]) / dx
    if kept:
        record[:steps] = torch.stack(kept).cpu().numpy()
    return F, record.ravel()


def _values(F, which):
    """The named fields' values; None for one that is rounding residue only
    (a component that the wave does not excite: nothing in 64 bits)."""
    norm = [float(f.norm()) for f in F]
    out = {}
    for c in which:
        top = max(norm[:3] if c < 3 else norm[3:])
        out["EH"[c // 3] + "xyz"[c % 3]] = (F[c].cpu().numpy().ravel() if norm[c] > 1e-5 * top
                                            else None)
    return out


def exact(case, seed):
    done = case["steps"] + case["warm"]
    if case["count"] == 1 and case["I"] * case["J"] * case["K"] * done > 3e10:
        return None
    specs = [_spec(case, seed, m) for m in range(case["count"])]
    if case["count"] == 1:
        s = specs[0]
        F, rec = _simulate(s, done)
        out = _values(F, range(FIELDS))
        return {"probes": rec, **out} if s["probes"] else out
    out = []
    for m, s in enumerate(specs):
        # the first few of a mix: each takes its steps one by one
        if m >= 4:
            out.append({"probes": None, "Ez": None} if case["kind"] == "serve" else {"Ez": None})
            continue
        F, rec = _simulate(s, s["steps"])
        one = _values(F, (2,))
        out.append({"probes": rec, **one} if case["kind"] == "serve" else one)
    return out
