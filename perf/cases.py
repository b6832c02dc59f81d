"""Timed workloads of the SSG solver library.

Every case is one pass through a public entry point as a user's program makes
it: forward modelling of a shot set (``SSGSolver.forward``), one FWI gradient
evaluation (``SSGSolver.gradient``), the adjoint source of recorded gathers
(``solver.adjoint_source``) and the host-side step of an inversion iteration
(``optim.search_direction`` with the gradient's smoothing and taper). The
solver handle, its model and the prepared geometry are what a program keeps
between calls; the observed data and gradients are on the device for the
gradient entries, and modelling returns host seismograms, ready to be written
as SU files.

``exact`` restates the acoustic solvers (forward and, through autograd, the
gradient), the envelope adjoint source and the L-BFGS step in 64 bits. The
elastic solvers with anisotropy have no such value: their absorbing layer's
damping ratios are the outcome of a threshold search in single precision, so a
64-bit evaluation may end one search step away and damp differently. The DTW
adjoint source has none either: it follows the discrete path that a dynamic
program chooses.
"""
from __future__ import annotations

import math

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

from owl_b200 import _lib as L
from owl_b200 import optim
from owl_b200.geometry import Receiver, Shot, Source
from owl_b200.solver import MisfitOpts, RunOpts, SSGSolver, adjoint_source

DX = {"ac2d": 10.0, "ac3d": 10.0, "el2d": 5.0, "el3d": 10.0}
DT = {"ac2d": 1e-3, "ac3d": 9e-4, "el2d": 5e-4, "el3d": 8e-4}
F0 = {"ac2d": 10.0, "ac3d": 12.0, "el2d": 15.0, "el3d": 10.0}
MEDIUM = {"ac2d": L.OWL_ACOUSTIC_ISO_2D, "ac3d": L.OWL_ACOUSTIC_ISO_3D,
          "el2d": L.OWL_ELASTIC_VHTIORT_2D, "el3d": L.OWL_ELASTIC_VHTIORT_3D}
NCOMP = {"ac2d": 1, "ac3d": 1, "el2d": 2, "el3d": 3}
CKPT = {"fp32": L.OWL_CKPT_FP32, "fp16": L.OWL_CKPT_FP16, "bf16": L.OWL_CKPT_BF16}
# floating-point operations of one time step per cell: the staggered
# derivatives (3 per coefficient pair) and the updates
DERIVS = {"ac2d": 4, "ac3d": 6, "el2d": 8, "el3d": 18}
UPDATES = {"ac2d": 8, "ac3d": 11, "el2d": 20, "el3d": 45}


def _wave(task, medium, nx, nz, nt, shots, nrec, ny=1, pml=20, half=4, fs=False, ckpt="fp32", every=50):
    return {"task": task, "medium": medium, "nx": nx, "ny": ny, "nz": nz, "nt": nt, "shots": shots, "nrec": nrec,
            "pml": pml, "half": half, "fs": fs, "ckpt": ckpt, "every": every}


def listed():
    def named(name, case):
        return {"name": name, **case}

    return [
        # one shot on a small section: a quick look at one gather, latency counts
        named("ac2d_one_shot", _wave("forward", "ac2d", 151, 101, 500, 1, 76, pml=15)),
        # the synthetic data of a 2D line, the plain modelling workload
        named("ac2d_line_modelling", _wave("forward", "ac2d", 401, 201, 1000, 16, 401)),
        # one FWI gradient evaluation of a 2D line, the benchmark workload: 32
        # shots, 2000 steps, single-precision checkpoints every 50 steps
        named("ac2d_line_gradient", _wave("gradient", "ac2d", 401, 201, 2000, 32, 301)),
        # a marine-type gradient: free surface, 16th order, odd sizes, few
        # shots, half-precision checkpoints
        named("ac2d_surface_gradient", _wave("gradient", "ac2d", 287, 173, 701, 5, 144, pml=16, half=8, fs=True,
                                             ckpt="fp16", every=40)),
        # 3D acoustic modelling of one shot into an areal spread
        named("ac3d_modelling", _wave("forward", "ac3d", 241, 201, 250, 1, 2500, ny=221)),
        # 3D acoustic gradient of one shot
        named("ac3d_gradient", _wave("gradient", "ac3d", 141, 121, 200, 1, 1600, ny=131, pml=15, ckpt="fp16")),
        # land modelling: VTI with a flat free surface, explosions and vertical forces, two components
        named("el2d_line_modelling", _wave("forward", "el2d", 601, 301, 1000, 16, 301, fs=True)),
        # gradient of the same medium in the Thomsen parameters
        named("el2d_line_gradient", _wave("gradient", "el2d", 301, 151, 800, 8, 151, fs=True, ckpt="fp16")),
        # 3D orthorhombic modelling, three components
        named("el3d_modelling", _wave("forward", "el3d", 149, 121, 150, 1, 900, ny=137, pml=15)),
        # 3D orthorhombic gradient in the nine moduli and the density
        named("el3d_gradient", _wave("gradient", "el3d", 105, 81, 120, 1, 400, ny=97, pml=12, ckpt="fp16")),
        # travel-time adjoint source of two recorded gathers by dynamic time warping
        named("dtw_adjoint_source", {"task": "adjoint", "misfit": "dtw", "gathers": 2, "traces": 81, "nt": 1001,
                                     "dt": 2e-3, "tlag": 0.1}),
        # what follows a gradient in every iteration: smoothing, taper and the
        # L-BFGS direction from the stored models and gradients
        named("lbfgs_step", {"task": "direction", "method": "l-bfgs", "nx": 401, "nz": 201, "models": 6,
                             "sigma": 3.0}),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _load(case):
    """a measure of a case's cost: cell updates weighted by the medium and the task"""
    if case["task"] == "direction":
        return 100.0 * case["nx"] * case["nz"] * case["models"]
    if case["task"] == "adjoint":
        return 0.0
    weight = {"ac2d": 1.0, "ac3d": 1.6, "el2d": 3.0, "el3d": 12.0}[case["medium"]]
    return weight * (5.0 if case["task"] == "gradient" else 1.0) * _cells(case) * case["nt"] * case["shots"]


def draw(rng):
    """One more case of the same ranges: sizes uniform in their logarithm, odd ones among them."""
    most = max(_load(c) for c in listed())
    kind = rng.choice(["ac2d", "ac2d", "ac2d", "el2d", "el2d", "ac3d", "el3d", "adjoint", "direction"])
    if kind == "direction":
        return {"task": "direction", "method": rng.choice(["l-bfgs", "l-bfgs", "cg"]), "nx": _log(rng, 101, 901),
                "nz": _log(rng, 65, 401), "models": rng.randint(2, 11), "sigma": round(rng.uniform(1.0, 6.0), 2)}
    if kind == "adjoint":
        misfit = rng.choice(["dtw", "envelope", "envelope"])
        nt = _log(rng, 301, 1001) if misfit == "dtw" else _log(rng, 301, 2001)
        return {"task": "adjoint", "misfit": misfit, "gathers": rng.randint(1, 3), "traces": _log(rng, 11, 81),
                "nt": nt, "dt": 2e-3, "tlag": round(rng.uniform(0.03, 0.1), 3)}
    task = rng.choice(["forward", "gradient"])
    half = 8 if kind == "ac2d" and rng.random() < 0.25 else 4
    fs = kind in ("ac2d", "el2d") and rng.random() < 0.5
    if kind in ("ac2d", "el2d"):
        nx, ny, nz = _log(rng, 120, 601), 1, _log(rng, 64, 301)
        nt, shots = _log(rng, 200, 2000), _log(rng, 1, 32)
        nrec = rng.randint(max(2, nx // 8), nx)
    else:
        top = 200 if kind == "ac3d" else 120
        nx, ny, nz = _log(rng, 48, top), _log(rng, 48, top), _log(rng, 48, top)
        nt, shots = _log(rng, 60, 250), rng.randint(1, 2)
        nrec = rng.randint(8, nx // 3) ** 2
    pml = rng.randint(10, 20)
    every = rng.choice([25, 40, 50])
    ckpt = rng.choice(["fp32", "fp32", "fp16", "bf16"])
    case = _wave(task, kind, nx, nz, nt, shots, nrec, ny=ny, pml=pml, half=half, fs=fs, ckpt=ckpt, every=every)
    if _load(case) > most:  # as many shots, then steps, as the largest listed case's cost allows
        case["shots"] = max(1, int(shots * most / _load(case)))
    if _load(case) > most:
        case["nt"] = max(50, int(nt * most / _load(case)))
    return case


# ------------------------------ inputs ---------------------------------------
def _smooth(shape, rng, waves=3):
    """a smooth random field in [-1, 1]: a few long cosines along each axis"""
    out = np.zeros(shape, dtype=np.float32)
    for _ in range(waves):
        f = np.float32(rng.uniform(0.5, 1.0) / waves)
        for ax, n in enumerate(shape):
            k, ph = rng.uniform(0.5, 2.5), rng.uniform(0, 2 * np.pi)
            c = np.cos(2 * np.pi * k * np.arange(n) / n + ph).astype(np.float32)
            f = f * c.reshape([-1 if a == ax else 1 for a in range(len(shape))])
        out = out + f
    return out


def _model(case, seed):
    """the medium's parameter fields in the order of SSGSolver.set_model, each (nz, nx) or (nz, ny, nx)"""
    rng = np.random.default_rng(seed)
    m = case["medium"]
    shape = (case["nz"], case["nx"]) if case["ny"] == 1 else (case["nz"], case["ny"], case["nx"])
    depth = np.linspace(0.0, 1.0, case["nz"], dtype=np.float32).reshape((-1,) + (1,) * (len(shape) - 1))
    if m in ("ac2d", "ac3d"):
        vp = 1500.0 + 2500.0 * depth + 120.0 * _smooth(shape, rng)
        vp = np.broadcast_to(vp, shape).astype(np.float32)
        return [vp, (310.0 * vp ** 0.25 * (1.0 + 0.02 * _smooth(shape, rng))).astype(np.float32)]
    if m == "el2d":
        vp = np.broadcast_to(1800.0 + 2600.0 * depth + 60.0 * _smooth(shape, rng), shape).astype(np.float32)
        eps = (0.09 + 0.08 * _smooth(shape, rng)).astype(np.float32)
        delta = (0.02 + 0.06 * _smooth(shape, rng)).astype(np.float32)
        return [vp, (vp / 1.8).astype(np.float32), eps, delta, np.zeros_like(vp),
                (310.0 * vp ** 0.25).astype(np.float32)]
    vp = np.broadcast_to(2000.0 + 2900.0 * depth, shape).astype(np.float32)
    vs, rho = vp / 1.73, 310.0 * vp ** 0.25
    fac = [1.0 + 0.07 * (1.0 + _smooth(shape, rng)) for _ in range(4)]
    c33, c44, c12 = rho * vp ** 2, rho * vs ** 2, rho * (vp ** 2 - 2 * vs ** 2)
    return [np.ascontiguousarray(f, dtype=np.float32)
            for f in (c33 * fac[0], c12, c12, c33 * fac[1], c12, c33, c44, c44 * fac[2], c44 * fac[3], rho)]


def _positions(case):
    """(sources, receivers) as (x, y, z) metres: sources off the grid nodes, receivers on them"""
    m = case["medium"]
    d, nx, ny = DX[m], case["nx"], case["ny"]
    wide, deep = (nx - 1) * d, (ny - 1) * d
    n = case["shots"]
    src = [(0.08 * wide + 0.84 * wide * ((k + 0.37) / n), 0.5 * deep + (0.13 * d if ny > 1 else 0.0), 2.0 * d)
           for k in range(n)]
    if ny == 1:
        cols = np.unique(np.linspace(0, nx - 1, case["nrec"]).round().astype(int))
        rec = [(d * int(i), 0.0, 0.0 if m == "el2d" else 2.0 * d) for i in cols]
    else:
        side = max(2, int(math.isqrt(case["nrec"])))
        cols = np.unique(np.linspace(2, nx - 3, side).round().astype(int))
        rows = np.unique(np.linspace(2, ny - 3, side).round().astype(int))
        rec = [(d * int(i), d * int(j), 2.0 * d) for j in rows for i in cols]
    return src, rec


def _shots(case):
    m = case["medium"]
    src, rec = _positions(case)
    recs = [Receiver(x=x, y=y, z=z) for x, y, z in rec]
    out = []
    for k, (x, y, z) in enumerate(src):
        force = (m == "el2d" and k % 2 == 1) or m == "el3d"
        mech = "force" if force else "explosion"
        out.append(Shot(k + 1, [Source(x=x, y=y, z=z, f0=F0[m], mechanism=mech)], recs))
    return out


def _observed(case, seed):
    """band-limited arrivals with a move-out, (shot, component, receiver, time) flattened"""
    rng = np.random.default_rng(seed + 77)
    m = case["medium"]
    src, rec = _positions(case)
    t = np.arange(case["nt"], dtype=np.float32) * np.float32(DT[m])
    r = np.asarray(rec, dtype=np.float32)
    scale = {"ac2d": 1e-4, "ac3d": 1e-4, "el2d": 1e-8, "el3d": 1e-9}[m]
    out = []
    for s in src:
        off = np.sqrt(((r - np.asarray(s, dtype=np.float32)) ** 2).sum(axis=1))
        for _ in range(NCOMP[m]):
            g = 0.0
            for v, w in ((1700.0, 1.0), (2600.0, 0.4)):
                arg = (np.pi * F0[m] * (t[None, :] - (off[:, None] / v + 1.0 / F0[m] + rng.uniform(0, 0.03)))) ** 2
                g = g + w * rng.uniform(0.7, 1.3) * (1.0 - 2.0 * arg) * np.exp(-np.minimum(arg, 80.0))
            out.append((scale * g).astype(np.float32).ravel())
    return np.concatenate(out)


def _gathers(case, seed):
    """synthetic and observed gathers: the observed ones shifted and scaled slowly along the spread"""
    rng = np.random.default_rng(seed)
    ntr, nt, dt = case["gathers"] * case["traces"], case["nt"], case["dt"]
    t = np.arange(nt) * dt
    syn, obs = np.zeros((ntr, nt)), np.zeros((ntr, nt))
    f0, span = 12.0, (nt - 1) * dt
    for w in range(5):
        t0 = span * rng.uniform(0.15, 0.8) + np.linspace(0.0, 0.1 * span, ntr)
        a = rng.uniform(-1.0, 1.0, ntr) * 0.2 + rng.choice([-1.0, 1.0])
        lag = 0.02 * np.sin(np.linspace(0, 6, ntr) + w) + rng.uniform(-0.01, 0.01)
        for target, tc, amp in ((syn, t0, a), (obs, t0 + lag, a * rng.uniform(0.8, 1.2))):
            arg = (np.pi * f0 * (t[None, :] - tc[:, None])) ** 2
            target += amp[:, None] * (1.0 - 2.0 * arg) * np.exp(-arg)
    noise = 1e-3 * rng.standard_normal((2, ntr, nt))
    return (syn + noise[0]).astype(np.float32), (obs + noise[1]).astype(np.float32)


def _history(case, seed):
    """models and gradients of the iterations so far, oldest first, flat with z fastest"""
    rng = np.random.default_rng(seed)
    shape = (case["nx"], case["nz"])
    x = 2500.0 + 400.0 * _smooth(shape, rng)
    curv = 1.0 + 0.5 * _smooth(shape, rng)
    target = x + 60.0 * _smooth(shape, rng)
    models, grads = [], []
    for _ in range(case["models"]):
        g = curv * (x - target) + 0.05 * rng.standard_normal(shape)
        models.append(x.astype(np.float32).ravel())
        grads.append(g.astype(np.float32).ravel())
        x = x - 0.35 * g + 0.5 * _smooth(shape, rng)
    prev = (-grads[0] + 0.1 * rng.standard_normal(grads[0].shape)).astype(np.float32)
    return models, grads, prev


# ------------------------------ the passes -----------------------------------
def prepare(case, seed):
    dev = torch.device("cuda")
    if case["task"] == "adjoint":
        syn, obs = _gathers(case, seed)
        gp = [case["traces"] * g for g in range(case["gathers"] + 1)]
        mo = MisfitOpts(misfit=L.MISFIT_NAMES[case["misfit"]], dt=case["dt"], tlag_max=case["tlag"])
        return {"case": case, "syn": torch.from_numpy(syn).to(dev), "obs": torch.from_numpy(obs).to(dev),
                "gp": gp, "mo": mo}
    if case["task"] == "direction":
        models, grads, prev = _history(case, seed)
        up = lambda a: torch.from_numpy(a).to(dev)  # noqa: E731
        return {"case": case, "models": [up(a) for a in models], "grads": [up(a) for a in grads], "prev": up(prev)}
    m = case["medium"]
    d = DX[m]
    s = SSGSolver(MEDIUM[m], case["nx"], case["nz"], d, d, DT[m], case["nt"], pml=case["pml"], fdhalf=case["half"],
                  free_surface=case["fs"], f0_max=F0[m], max_shots=case["shots"], ny=case["ny"],
                  aniso={"el2d": L.OWL_ANISO_THOMSEN, "el3d": L.OWL_ANISO_CIJ}.get(m, 0))
    s.set_model(*_model(case, seed))
    ps = s.prepare(_shots(case))
    state = {"case": case, "solver": s, "ps": ps}
    if case["task"] == "gradient":
        state["obs"] = torch.from_numpy(_observed(case, seed)).to(dev)
        state["opts"] = RunOpts(checkpoint_interval=case["every"], checkpoint_precision=CKPT[case["ckpt"]])
    return state


def run(state):
    case = state["case"]
    if case["task"] == "forward":
        return state["solver"].forward(state["ps"])
    if case["task"] == "gradient":
        misfit, grad = state["solver"].gradient(state["ps"], state["obs"], opts=state["opts"])
        return {"misfit": misfit, "grad": grad}
    if case["task"] == "adjoint":
        adj, traces, gathers = adjoint_source(state["mo"], state["gp"], state["syn"], state["obs"])
        return {"adj": adj, "trace_misfit": traces, "gather_misfit": gathers}
    # the newest gradient is processed on a copy (the raw one stays in the history), then enters the direction
    nx, nz = case["nx"], case["nz"]
    g = state["grads"][-1].clone()
    field = g.view(nx, nz).t()
    optim.process(field, L.OWL_GRAD_SMOOTH, [case["sigma"], case["sigma"], 0.0])
    optim.process(field, L.OWL_GRAD_TAPER, [8, 8, 12, 12, 0, 0])
    srch = optim.search_direction(L.SEARCH_NAMES[case["method"]], state["models"], state["grads"][:-1] + [g],
                                  prev_srch=state["prev"])
    return {"gradient": g, "direction": srch}


def _cells(case):
    p = 2 * case["pml"]
    return (case["nx"] + p) * (case["nz"] + p) * (case["ny"] + p if case["ny"] > 1 else 1)


def work(case):
    if case["task"] == "direction":
        n = case["nx"] * case["nz"]
        rad = math.ceil(3 * case["sigma"])
        pairs = case["models"] - 1 if case["method"] == "l-bfgs" else 1
        return {"bytes": 4.0 * n * (2 * case["models"] + 2), "flops": n * (4.0 * (2 * rad + 1) + 14.0 * pairs)}
    if case["task"] == "adjoint":
        n = case["gathers"] * case["traces"] * case["nt"]
        if case["misfit"] == "dtw":  # every sample's candidates against the allowed slopes' runs, at least one pass
            m = 2 * int(case["tlag"] / case["dt"] + 0.5) + 1
            return {"bytes": 12.0 * n, "flops": 20.0 * n * m}
        return {"bytes": 12.0 * n, "flops": 4 * 5.0 * n * math.log2(max(2, case["nt"]))}
    m = case["medium"]
    nm = case["nx"] * case["nz"] * case["ny"]
    nparam = {"ac2d": 2, "ac3d": 2, "el2d": 6, "el3d": 10}[m]
    traces = 4.0 * len(_positions(case)[1]) * NCOMP[m] * case["shots"] * case["nt"]
    step = DERIVS[m] * 3.0 * case["half"] + UPDATES[m]
    steps = float(_cells(case)) * case["nt"] * case["shots"]
    if case["task"] == "forward":
        return {"bytes": 4.0 * nparam * nm + traces, "flops": step * steps}
    # a gradient: the forward, its adjoint, and the correlations
    return {"bytes": 8.0 * nparam * nm + traces, "flops": (2 * step + 6.0 * nparam) * steps}


# ------------------------------ 64-bit values --------------------------------
def exact(case, seed):
    if case["task"] == "direction":
        return _exact_direction(case, seed)
    if case["task"] == "adjoint":
        return _exact_envelope(case, seed) if case["misfit"] == "envelope" else None
    if case["medium"] in ("el2d", "el3d"):
        return None
    return _exact_acoustic(case, seed)


def _exact_direction(case, seed):
    models, grads, prev = _history(case, seed)
    models = [a.astype(np.float64) for a in models]
    grads = [a.astype(np.float64) for a in grads]
    g = grads[-1].reshape(case["nx"], case["nz"])
    sg = case["sigma"]
    rad = max(1, math.ceil(3 * float(np.float32(sg))))
    w = np.exp(-0.5 * np.arange(-rad, rad + 1.0) ** 2 / float(np.float32(sg)) ** 2)
    w /= w.sum()
    for ax in (1, 0):
        p = np.pad(g, [(rad, rad) if a == ax else (0, 0) for a in range(2)], mode="edge")
        n = g.shape[ax]
        g = sum(w[k] * np.take(p, range(k, k + n), axis=ax) for k in range(2 * rad + 1))
    for ax, ln in ((1, 8), (0, 12)):
        t = np.arange(ln) / ln
        ramp = np.ones(g.shape[ax])
        ramp[:ln] *= 0.42 - 0.5 * np.cos(np.pi * t) + 0.08 * np.cos(2 * np.pi * t)
        ramp = ramp * ramp[::-1]
        g = g * ramp.reshape((-1, 1) if ax == 0 else (1, -1))
    g = g.ravel()
    grads[-1] = g
    if case["method"] == "cg":
        gp = grads[-2]
        beta = max(0.0, float(np.dot(g - gp, g)) / float(np.dot(gp, gp)))
        return {"gradient": g, "direction": -g + beta * prev.astype(np.float64)}
    q, alpha, ys = g.copy(), {}, {}
    pairs = [(models[i + 1] - models[i], grads[i + 1] - grads[i]) for i in range(len(models) - 1)]
    for i in range(len(pairs) - 1, -1, -1):
        s, y = pairs[i]
        ys[i] = float(np.dot(y, s))
        alpha[i] = float(np.dot(s, q)) / ys[i]
        q -= alpha[i] * y
    s, y = pairs[-1]
    q *= float(np.dot(y, s)) / float(np.dot(y, y))
    for i, (s, y) in enumerate(pairs):
        q += s * (alpha[i] - float(np.dot(y, q)) / ys[i])
    return {"gradient": g, "direction": -q}


def _exact_envelope(case, seed):
    syn, obs = (a.astype(np.float64) for a in _gathers(case, seed))
    n = case["nt"]
    h = np.zeros(n)
    h[0] = 1.0
    h[1:(n + 1) // 2] = 2.0
    if n % 2 == 0:
        h[n // 2] = 1.0

    def analytic(x):
        return np.fft.ifft(np.fft.fft(x, axis=1) * h, axis=1)

    e1, z = np.abs(analytic(obs)), analytic(syn)
    e2 = np.abs(z)
    coef = (e2 - e1) / (e2 + float(np.float32(1e-2)) * e2.max(axis=1, keepdims=True))
    adj = syn * coef - analytic(z.imag * coef).imag
    tm = ((e1 - e2) ** 2).sum(axis=1)
    return {"adj": adj, "trace_misfit": tm, "gather_misfit": tm.reshape(case["gathers"], -1).sum(axis=1)}


_COEF = {4: (1.217990, -0.09382142, 0.01507536, -0.001700324),
         8: (1.259312, -0.1280347, 0.03841945, -0.01473229, 0.005924913, -0.002248618, 0.0007179226, -0.0001400855)}


def _taps(pos, d):
    """nearest node (1-based) and the nine Kaiser-windowed sinc weights around it"""
    q = float(np.float32(np.float32(pos) / np.float32(d)))
    g = int(math.floor(q + 0.5)) + 1
    x = q - (g - 1)
    t = np.arange(-4, 5) - x
    b = float(np.float32(6.31))
    win = np.where(np.abs(t) <= 4, np.i0(b * np.sqrt(np.maximum(0.0, 1.0 - (t / 4) ** 2))) / np.i0(b), 0.0)
    return g, np.sinc(t) * win


def _exact_acoustic(case, seed):
    """The acoustic solver in 64 bits: every derivative a product with the
    operator's matrix over the padded axis, the gradient by autograd over
    recomputed segments of the time loop."""
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    f64 = dict(dtype=torch.float64, device=dev)
    m, P, R, nt, S = case["medium"], case["pml"], case["half"], case["nt"], case["shots"]
    d, dt = float(np.float32(DX[m])), float(np.float32(DT[m]))
    three = case["ny"] > 1
    n = [case["nz"], case["ny"], case["nx"]] if three else [case["nz"], case["nx"]]
    dim, N = len(n), [k + 2 * P for k in n]
    vp, rho = (torch.from_numpy(np.ascontiguousarray(a)).to(**f64).requires_grad_(case["task"] == "gradient")
               for a in _model(case, seed))
    coef = np.asarray(_COEF[R], dtype=np.float32).astype(np.float64)

    def matrices(size):
        to_p, to_v = np.zeros((size, size)), np.zeros((size, size))
        for k, c in enumerate(coef, 1):
            for i in range(size):
                for j, w in ((i + k, c), (i + 1 - k, -c)):
                    if 0 <= j < size:
                        to_p[i, j] += w / d
                for j, w in ((i + k - 1, c), (i - k, -c)):
                    if 0 <= j < size:
                        to_v[i, j] += w / d
        return torch.from_numpy(to_p).to(**f64), torch.from_numpy(to_v).to(**f64)

    ops = [matrices(k) for k in N]

    def along(mat, f, ax):  # mat applied along spatial axis ax of (shots, ...)
        if ax == dim - 1:
            return f @ mat.T
        if ax == 0:
            return (mat @ f.reshape(f.shape[0], f.shape[1], -1)).reshape(f.shape)
        return mat @ f

    # absorbing layers: (a, b) along each axis at whole and half nodes
    v = vp.detach().cpu().numpy()
    vmax = max(float(v.take(e, axis=a).max()) for a in range(dim) for e in (0, -1))
    amax = float(np.float32(F0[m])) * math.pi

    def damping(size, ax, half):
        a, b = np.zeros(size + 2 * P), np.zeros(size + 2 * P)
        for i in range(-P + 1, size + P + 1):
            if half:
                dist = abs(i - 1.5) if i <= 1 else i - size - 0.5 if i >= size + 1 else None
            else:
                dist = 1.0 - i if i < 1 else float(i - size) if i >= size + 1 else None
            if dist is None or (case["fs"] and ax == 0 and i <= 1):
                continue
            nd = dist / P
            alpha = max(amax * (1.0 - nd), 0.25 * amax)
            damp = vmax * 3.0 * math.log(1e5) / (2.0 * P * d) * nd * nd
            a[i + P - 1] = -2.0 * dt * damp / (2.0 + dt * (alpha + damp))
            b[i + P - 1] = (2.0 - dt * (alpha + damp)) / (2.0 + dt * (alpha + damp))
        shape = [1] + [-1 if q == ax else 1 for q in range(dim)]
        return torch.from_numpy(a).to(**f64).reshape(shape), torch.from_numpy(b).to(**f64).reshape(shape)

    pml_p = [damping(n[q], q, False) for q in range(dim)]
    pml_v = [damping(n[q], q, True) for q in range(dim)]

    # coefficients over the padded grid
    def pad(f, lo):
        mode = [P + 1 - lo, P] * dim
        return torch.nn.functional.pad(f[None, None], mode, mode="replicate")[0, 0]

    bk = dt * pad(rho, 1) * pad(vp, 1) ** 2
    wide = pad(rho, 0)
    inner = tuple(slice(1, None) for _ in range(dim))
    bv = []
    for q in range(dim):
        low = tuple(slice(0, -1) if a == q else slice(1, None) for a in range(dim))
        bv.append(dt / (0.5 * (wide[inner] + wide[low])))
    mirror = live_p = None
    live_v = [None] * dim
    if case["fs"]:
        keep = torch.ones(N[0], **f64)
        keep[:P + 1] = 0  # rows up to the surface row 1
        mz = torch.zeros(N[0], N[0], **f64)
        for i in range(P + 1, N[0]):
            mz[i, i] = 1.0
        for j in range(2, P + 2):
            mz[(2 - j) + P - 1, j + P - 1] = -1.0
        mirror = mz
        live_p = keep.reshape([1, -1] + [1] * (dim - 1))
        on = torch.ones(N[0], **f64)
        on[:P] = 0
        live_v = [live_p] + [on.reshape([1, -1] + [1] * (dim - 1))] * (dim - 1)

    # sources, receivers
    src, rec = _positions(case)
    order = (2, 1, 0) if three else (2, 0)
    inj = torch.zeros([S] + N, **f64)
    for s, pos in enumerate(src):
        taps = [_taps(pos[c], d) for c in order]
        box = taps[0][1]
        for t in taps[1:]:
            box = np.multiply.outer(box, t[1])
        lo = [t[0] - 4 + P - 1 for t in taps]
        where = tuple(slice(max(0, o), o + 9) for o in lo)
        cut = tuple(slice(max(0, -o), None) for o in lo)
        part = torch.from_numpy(np.ascontiguousarray(box[cut])).to(**f64)
        if case["fs"]:
            first = P + 1 - where[0].start
            if first > 0:
                part[:first] = 0
        inj[(s,) + where] += part
    idx = torch.zeros(len(rec), dtype=torch.long, device=dev)
    for a, c in enumerate(order):
        node = torch.tensor([int(round(r[c] / d)) + P for r in rec], device=dev)
        idx = idx * N[a] + node
    count = int(math.ceil(float(np.float32(np.float32(2.0) / np.float32(F0[m])) / np.float32(DT[m]))))
    tau = (np.arange(count) * dt - 1.0 / F0[m]) * math.pi * F0[m]
    stf = (1.0 - 2.0 * tau ** 2) * np.exp(-tau ** 2)
    stf = np.concatenate([stf / np.abs(stf).max() * dt, np.zeros(nt + 1)])

    def segment(i0, i1, bk_, *rest):
        bv_, st = rest[:dim], list(rest[dim:])
        p, vel, mp, mv = st[0], st[1:1 + dim], st[1 + dim:1 + 2 * dim], st[1 + 2 * dim:]
        seis = []
        for i in range(i0, i1):
            seis.append(p.reshape(S, -1)[:, idx])
            g = 0.0
            for q in range(dim):
                h = along(ops[q][0], vel[q], q)
                mp[q] = pml_p[q][0] * h + pml_p[q][1] * mp[q]
                g = g + h + mp[q]
            if live_p is not None:
                g = g * live_p
            p = p - bk_ * g
            if mirror is not None:
                p = along(mirror, p, 0)
            for q in range(dim):
                h = along(ops[q][1], p, q)
                mv[q] = pml_v[q][0] * h + pml_v[q][1] * mv[q]
                h = h + mv[q]
                vel[q] = vel[q] - bv_[q] * (h if live_v[q] is None else h * live_v[q])
            if stf[i] != 0.0:
                p = p + stf[i] * inj
        return (torch.stack(seis, dim=-1), p, *vel, *mp, *mv)

    step = max(5, int(math.sqrt(nt)) // 2)
    state = [torch.zeros([S] + N, **f64) for _ in range(1 + 3 * dim)]
    parts = []
    with torch.set_grad_enabled(case["task"] == "gradient"):
        for i0 in range(0, nt, step):
            args = (i0, min(nt, i0 + step), bk, *bv, *state)
            if case["task"] == "gradient":
                out = checkpoint(segment, *args, use_reentrant=False)
            else:
                out = segment(*args)
            parts.append(out[0])
            state = list(out[1:])
        syn = torch.cat(parts, dim=-1)
        if case["task"] == "forward":
            return syn.reshape(-1).cpu().numpy()
        obs = torch.from_numpy(_observed(case, seed)).to(**f64).reshape(syn.shape)
        misfit = ((obs - syn) ** 2).sum(dim=(1, 2))
        gvp, grho = torch.autograd.grad(0.5 * misfit.sum(), (vp, rho))
    flat = [g.permute(*reversed(range(dim))).reshape(-1).cpu().numpy() for g in (gvp, grho)]
    return {"misfit": misfit.detach().cpu().numpy(), "grad": np.concatenate(flat)}
