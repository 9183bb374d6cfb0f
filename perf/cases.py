"""The work this framework is timed on: its operators, its steppers and its
drivers, each through the public call a user's program makes.

``listed()`` names the cases, ``draw`` gives more of the same ranges,
``prepare`` makes what such a program holds before the call, ``run`` is one
pass, ``work`` its unavoidable bytes and operations, and ``exact`` the same
outputs in 64-bit torch without this framework's code.
"""
from __future__ import annotations

import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "exactclosure.jl_gb300"))
from exactclosure_gb300 import burgers as GB  # noqa: E402
from exactclosure_gb300 import navierstokes as NS  # noqa: E402
from exactclosure_gb300.learned import SHAPES, VALID, Net, flatten  # noqa: E402
from exactclosure_gb300.serving import Server  # noqa: E402

DTYPES = {"f64": torch.float64, "f32": torch.float32}
L = 1.0
CFL = 0.3
F64 = torch.float64


def listed():
    return [
        # the projected right-hand side of one field, two operator calls of a host program's own time loop: on an
        # LES grid (the smallest call) and on the reference driver's default DNS grid
        {"name": "stage_32_f64", "kind": "stage", "n": 32, "prec": "f64"},
        {"name": "stage_500_f64", "kind": "stage", "n": 500, "prec": "f64"},
        # the convection-diffusion right-hand side alone, FP32, a grid that is no multiple of the tiles
        {"name": "rhs_180_f32", "kind": "rhs", "n": 180, "prec": "f32"},
        # the reference's small case: 90^3 with LES 18^3 and 30^3 (odd ratios), ten steps between two outputs
        {"name": "step_90_f64", "kind": "step", "n": 90, "prec": "f64", "les": "5v,3v", "steps": 10},
        # DNS 128^3 with one LES grid 32^3, the plain method's configuration
        {"name": "step_128_f64", "kind": "step", "n": 128, "prec": "f64", "les": "4v", "steps": 10},
        # DNS 512^3 with LES 64^3 and 128^3, the benchmark's configuration: the largest
        {"name": "step_512_f64", "kind": "step", "n": 512, "prec": "f64", "les": "8v,4v", "steps": 2},
        # the precision form with volume and face filters, the form of the large snapshot-pair runs
        {"name": "step_512_f32", "kind": "step", "n": 512, "prec": "f32", "les": "8v,4v,8f,4f", "steps": 4},
        # the reference's own Euler driver with its five LES (ratio 5, Gaussian filter of width 2H)
        {"name": "euler_250_f64", "kind": "euler", "n": 250, "ratio": 5, "gauss": True, "steps": 4},
        # served FP32 solves of mixed sizes, submitted together and drained
        {"name": "serve_mixed_f32", "kind": "serve", "sizes": "64,96,64,96,128,64", "steps": 100},
        # the learned closure inside an LES: one 64^3 field per call
        {"name": "net_forward_64_b1", "kind": "net", "n": 64, "batch": 1, "mode": "forward"},
        # its training pass: loss and gradients of eight 64^3 snapshots
        {"name": "net_gradients_64_b8", "kind": "net", "n": 64, "batch": 8, "mode": "gradients"},
        # the Burgers DNS-aided LES of 152 samples at the reference's DNS size
        {"name": "burgers_13500_s152", "kind": "burgers", "nh": 13500, "nH": 900, "samples": 152, "delta": 2.0,
         "filter": "gaussian", "tstop": 0.02},
    ]


def _supported(n: int) -> bool:
    if n < 4 or n % 2:
        return False
    for p in (2, 3, 5, 7, 11, 13, 17):
        while n % p == 0:
            n //= p
    return n == 1


def _grid(rng, lo: int, hi: int, mult: int = 1) -> int:
    """A supported grid size, log-uniform over [lo, hi], a multiple of `mult`
    with a supported quotient."""
    while True:
        n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / mult)) * mult
        if lo <= n <= hi and _supported(n) and _supported(n // mult):
            return n


def draw(rng):
    kind = rng.choice(("stage", "stage", "rhs", "step", "step", "step", "euler", "serve", "net", "burgers"))
    if kind in ("stage", "rhs"):
        return {"kind": kind, "n": _grid(rng, 24, 512), "prec": rng.choice(("f64", "f32"))}
    if kind == "step":
        ratio = rng.choice((2, 3, 4, 5, 8))
        prec = rng.choice(("f64", "f32"))
        n = _grid(rng, 48, 320 if prec == "f64" else 448, ratio)
        les = f"{ratio}{rng.choice('vf')}"
        if ratio in (2, 4) and _supported(n // (2 * ratio)) and n % (2 * ratio) == 0:
            les = f"{2 * ratio}v," + les
        return {"kind": kind, "n": n, "prec": prec, "les": les, "steps": 10 if n <= 160 else 4}
    if kind == "euler":
        ratio = rng.choice((3, 5))
        return {"kind": kind, "n": _grid(rng, 60, 300, ratio), "ratio": ratio, "gauss": rng.random() < 0.5, "steps": 4}
    if kind == "serve":
        sizes = [rng.choice((48, 64, 96, 128)) for _ in range(rng.randint(3, 6))]
        return {"kind": kind, "sizes": ",".join(map(str, sizes)), "steps": rng.randint(30, 100)}
    if kind == "net":
        return {"kind": kind, "n": rng.choice((32, 48, 64, 64)), "batch": rng.randint(1, 8),
                "mode": rng.choice(("forward", "gradients"))}
    nH = rng.choice((100, 300, 500, 900))
    comp = rng.choice([c for c in range(5, 46, 2) if 1500 <= nH * c <= 13800])
    return {"kind": kind, "nh": nH * comp, "nH": nH, "samples": rng.randint(16, 200), "delta": float(rng.randint(1, 3)),
            "filter": rng.choice(("gaussian", "tophat")), "tstop": 0.01}


# --------------------------------------------------------------------------
# Inputs
# --------------------------------------------------------------------------
def _gen(seed: int) -> torch.Generator:
    return torch.Generator(device="cuda").manual_seed(seed)


def _velocity(n: int, seed: int, kpeak: float = 6.0, energy: float = 1.0):
    """A solenoidal random-phase field with E(k) ~ k^4 exp(-2 (k/kpeak)^2),
    float64 ``(3, n, n, n)`` on the GPU."""
    g = _gen(seed)
    k = torch.fft.fftfreq(n, 1 / n, dtype=F64, device="cuda")
    kx = k[: n // 2 + 1].abs()
    k2 = k[:, None, None] ** 2 + k[None, :, None] ** 2 + kx[None, None, :] ** 2
    amp = k2.sqrt() * torch.exp(-k2 / kpeak**2)
    u = torch.empty((3, n, n, n), dtype=F64, device="cuda")
    for c in range(3):
        w = torch.randn((n, n, n), generator=g, dtype=F64, device="cuda")
        u[c] = torch.fft.irfftn(torch.fft.rfftn(w) * amp, s=(n, n, n))
    u = _project(u, L / n)[0]
    return u * math.sqrt(2 * energy * n**3 / float((u * u).sum()))


def _visc(n: int) -> float:
    return 1 / 2000 if n >= 128 else 1 / 500


def _les(spec: str):
    return [(int(s[:-1]), {"v": "volume", "f": "face"}[s[-1]]) for s in spec.split(",")]


def _gaussian(case):
    """The Gaussian of width 2H and 2 sigmas of the reference's default setup."""
    return NS.gaussian(L / case["n"], 2 * L * case["ratio"] / case["n"], 2) if case["gauss"] else None


def _gaussian_exact(case):
    if not case["gauss"]:
        return None
    s = 2 * case["ratio"] / math.sqrt(12)
    x = np.arange(-round(2 * s), round(2 * s) + 1)
    w = np.exp(-(x**2) / (2 * s * s))
    return w / w.sum()


def _burgers_start(case, seed: int) -> np.ndarray:
    g = np.random.default_rng(seed)
    nh, ns, k0 = case["nh"], case["samples"], 10
    k = np.arange(nh // 2 + 1)
    amp = (k / k0) ** 4 * np.exp(-2 * (k / k0) ** 2)
    a = np.fft.irfft(amp * np.exp(2j * np.pi * g.random((ns, nh // 2 + 1))) * nh, nh, axis=1)
    return a * np.sqrt(2.0 / ((a * a).sum(axis=1, keepdims=True) / 2 * (2 * np.pi / nh)))


def _net_inputs(case, seed: int):
    """Filtered-velocity-like inputs, closure-like targets, He-initialised weights."""
    n, b = case["n"], case["batch"]
    g = _gen(seed)
    k = torch.fft.fftfreq(n, 1 / n, device="cuda")
    k2 = k[:, None, None] ** 2 + k[None, :, None] ** 2 + k[None, None, : n // 2 + 1] ** 2
    out = []
    for slope in (-1.8, -0.8):
        w = torch.fft.rfftn(torch.randn((b, 3, n, n, n), generator=g, device="cuda"), dim=(2, 3, 4))
        f = torch.fft.irfftn(w * (1 + k2) ** (slope / 2), s=(n, n, n), dim=(2, 3, 4))
        out.append((f / f.square().mean().sqrt()).contiguous())
    r = np.random.default_rng(seed)
    params = [(r.normal(0, math.sqrt(2 / (27 * ci)), (27, ci, co)).astype(np.float32),
               r.normal(0, 0.05, co).astype(np.float32)) for ci, co in VALID]
    return out[0], out[1], params


_stream = None


def _case_stream():
    """One stream for every case of the program, as a host program has."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream.cuda_stream


class _Device:
    """The case's device velocity for ``torch.as_tensor`` (no copy); keeps the case."""

    def __init__(self, case, dtype):
        n = case.n
        self.case = case
        self.__cuda_array_interface__ = {"shape": (3, n, n, n), "typestr": "<f8" if dtype == F64 else "<f4",
                                         "data": (case.device_ptr(), False), "version": 2}


def _view(cs, dtype):
    return torch.as_tensor(_Device(cs, dtype), device="cuda")


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind in ("stage", "rhs"):
        n, dt = case["n"], DTYPES[case["prec"]]
        s["grid"] = NS.Grid(L, n)
        s["u"] = _velocity(n, seed).to(dt)
        s["out"] = torch.empty_like(s["u"])
        if kind == "stage":
            s["p"] = torch.empty_like(s["u"][0])
            s["poisson"] = NS.poissonsolver(s["grid"], 0 if case["prec"] == "f64" else 1)
    elif kind == "step":
        n, dt = case["n"], DTYPES[case["prec"]]
        cs = NS.Case(n, L, _visc(n), CFL, precision=0 if dt == F64 else 1, les=_les(case["les"]), stream=_case_stream())
        _view(cs, dt).copy_(_velocity(n, seed))
        torch.cuda.synchronize()
        cs.reset_les()
        s["cs"], s["dtype"] = cs, dt
        s["pairs"] = [torch.empty((2, 3) + (n // c,) * 3, dtype=dt, device="cuda") for c, _ in cs.les_list]
    elif kind == "euler":
        n = case["n"]
        d = NS.DnsAid(n, L, 2e-4, case["ratio"], _gaussian(case))
        d.set_velocity(_velocity(n, seed).cpu().numpy())
        d.start()
        s["d"] = d
    elif kind == "serve":
        s["server"], s["seed"] = Server(), seed
    elif kind == "net":
        s["u"], s["m"], params = _net_inputs(case, seed)
        s["net"] = Net(0)
        s["net"].set_params(flatten(params))
        s["out"] = torch.empty_like(s["u"])
    else:
        s["batch"] = GB.Batch(GB.Grid(2 * math.pi, case["nh"]), case["samples"], 5e-4)
        s["batch"].set_velocity(_burgers_start(case, seed))
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind in ("stage", "rhs"):
        NS.tensordivergence(s["out"], s["u"], _visc(case["n"]), s["grid"])
        if kind == "rhs":
            return s["out"]
        NS.project(s["out"], s["poisson"], s["p"])
        return {"k": s["out"], "p": s["p"]}
    if kind == "step":
        cs = s["cs"]
        cs.step(case["steps"])
        for i, pair in enumerate(s["pairs"]):
            cs.snapshot(i, pair[0], pair[1])
        # the LES states come as float64 arrays; an FP32 case's hold FP32 values
        word = np.float64 if s["dtype"] == F64 else np.float32
        les = [cs.les(0, w).astype(word, copy=False) for w in ("exact", "nomodel")]
        return {"u": _view(cs, s["dtype"]), "pairs": s["pairs"], "les": les}
    if kind == "euler":
        s["d"].step(math.inf, CFL, max_steps=case["steps"])
        return {k: s["d"].get(k) for k in NS.DNSAID_FIELDS}
    if kind == "serve":
        sv = s["server"]
        for i, n in enumerate(_sizes(case)):
            sv.submit(n, _visc(n), case["steps"], seed=s["seed"] + i, keep_field=True)
        sv.drain()
        got = sorted(sv.poll(), key=lambda r: r["id"])
        # served FP32: the float64 host buffers hold FP32 values
        return {"field": [r["field"].astype(np.float32) for r in got],
                "energy": np.array([r["energy"] for r in got], dtype=np.float32),
                "time": np.array([r["sim_time"] for r in got], dtype=np.float32)}
    if kind == "net":
        if case["mode"] == "forward":
            return s["net"].forward(s["u"], s["out"])
        loss, grad = s["net"].gradients(s["u"], s["m"])
        return {"loss": loss, "grad": grad}
    gH = GB.Grid(2 * math.pi, case["nH"])
    return GB.dns_aided_les(s["batch"], gH, case["delta"] * gH.spacing, case["tstop"], CFL, case["filter"])


def _sizes(case):
    return [int(x) for x in case["sizes"].split(",")]


# --------------------------------------------------------------------------
# What a pass cannot do without
# --------------------------------------------------------------------------
def _solve_flops(n: int) -> float:
    """A real transform and its inverse, the divide, divergence and gradient."""
    return n**3 * (2 * 2.5 * math.log2(n**3) + 1 + 6 + 6)


def _rk4_flops(n: int) -> float:
    """Four stages: 63 operations of the right-hand side, a projection, the combination."""
    return 4 * (n**3 * (63 + 12) + _solve_flops(n))


def work(case):
    kind = case["kind"]
    if kind in ("stage", "rhs"):
        n3, w = case["n"] ** 3, 8 if case["prec"] == "f64" else 4
        if kind == "rhs":
            return {"bytes": 6 * n3 * w, "flops": 63 * n3}
        return {"bytes": 7 * n3 * w, "flops": 63 * n3 + _solve_flops(case["n"])}
    if kind == "step":
        n, w, k = case["n"], 8 if case["prec"] == "f64" else 4, case["steps"]
        les = [n // c for c, _ in _les(case["les"])]
        # the state in and out once a step; three solves a stage on each LES grid
        b = 6 * n**3 * w + sum(12 * m**3 * w for m in les)
        f = _rk4_flops(n) + sum(2 * _rk4_flops(m) + 4 * (_solve_flops(m) + 6 * n**3) for m in les)
        return {"bytes": k * b, "flops": k * f}
    if kind == "euler":
        n, m = case["n"], case["n"] // case["ratio"]
        f = n**3 * (63 + 6 + 2 * 48) + _solve_flops(n) + 6 * (_solve_flops(m) + 63 * m**3)
        return {"bytes": case["steps"] * 8 * (6 * n**3 + 30 * m**3), "flops": case["steps"] * f}
    if kind == "serve":
        z = _sizes(case)
        return {"bytes": case["steps"] * sum(24 * n**3 for n in z) + sum(24 * n**3 for n in z),
                "flops": case["steps"] * sum(_rk4_flops(n) for n in z)}
    if kind == "net":
        v = case["batch"] * case["n"] ** 3
        f = 2 * 27 * v * sum(ci * co for ci, co in VALID)
        if case["mode"] == "forward":
            return {"bytes": 24 * v, "flops": f}
        return {"bytes": 24 * v, "flops": 3 * f - 2 * 27 * v * 3 * 32}
    nh, nH, ns = case["nh"], case["nH"], case["samples"]
    # initial peak speed about 1.6 sets the step; taps of the coarse filters per step
    steps = case["tstop"] / (CFL * min(2 * math.pi / nh / 1.6, (2 * math.pi / nh) ** 2 / 5e-4))
    return {"bytes": 8 * ns * (3 * nh + 5 * nH), "flops": ns * steps * (nh * 12 + nH * 5 * 2 * 4 * nh / nH)}


# --------------------------------------------------------------------------
# The same outputs in 64 bits
# --------------------------------------------------------------------------
SYM6 = ((0, 0), (1, 1), (2, 2), (0, 1), (1, 2), (2, 0))


def _at(a, d: int, k: int):
    """a[I + k e_d] of fields laid out [..., z, y, x]."""
    return a if k == 0 else torch.roll(a, -k, dims=-1 - d)


def _stress(u, visc, h):
    s = {}
    for i, j in SYM6:
        o = int(i != j)
        a, b, c, d = _at(u[i], j, o), _at(u[i], j, o - 1), _at(u[j], i, o), _at(u[j], i, o - 1)
        s[i, j] = s[j, i] = (a + b) * (c + d) / 4 - visc * ((a - b) + (c - d)) / h
    return s


def _tensordiv(s, h, du=None):
    out = torch.zeros((3,) + s[0, 0].shape, dtype=F64, device="cuda") if du is None else du.clone()
    for i in range(3):
        for j in range(3):
            t = s[i, j]
            out[i] -= ((_at(t, j, 1) - t) if i == j else (t - _at(t, j, -1))) / h
    return out


def _rhs(u, visc, h):
    return _tensordiv(_stress(u, visc, h), h)


def _project(u, h):
    n = u.shape[-1]
    d = sum(u[i] - _at(u[i], i, -1) for i in range(3)) / h
    s = torch.sin(math.pi * torch.arange(n, dtype=F64, device="cuda") / n) ** 2
    lam = -4 / h**2 * (s[:, None, None] + s[None, :, None] + s[None, None, : n // 2 + 1])
    lam[0, 0, 0] = 1
    q = torch.fft.rfftn(d) / lam
    q[0, 0, 0] = 0
    p = torch.fft.irfftn(q, s=(n, n, n))
    return torch.stack([u[i] - (_at(p, i, 1) - p) / h for i in range(3)]), p


def _taps(c: int, stag: bool, mode: str, fd):
    """Offsets and weights of the coarse sample along one axis: the box over the
    coarse cell or the point sample, at a face (stag) or a centre, convolved
    with the Gaussian where there is one."""
    a = c // 2
    if mode == "point":
        o, w = ([c - 1], [1.0]) if stag else ([a], [1.0]) if c % 2 else ([a - 1, a], [0.5, 0.5])
    elif not stag:
        o, w = list(range(c)), [1 / c] * c
    else:
        o = list(range(c - 1 - a, c + a))
        w = [1 / c] * len(o)
        if c % 2 == 0:
            w[0] = w[-1] = 0.5 / c
    if fd is not None:
        w = np.convolve(w, fd)
        o = range(o[0] - len(fd) // 2, o[0] - len(fd) // 2 + len(w))
    return list(zip(o, w))


def _coarse(f, c: int, stags, modes, fd=None):
    n = f.shape[-1]
    base = c * torch.arange(n // c, device="cuda")
    for d in range(3):
        f = sum(w * torch.index_select(f, 2 - d, (base + o) % n) for o, w in _taps(c, stags[d], modes[d], fd))
    return f


def _filter(u, c: int, kind: str, fd=None):
    return torch.stack([_coarse(u[i], c, [d == i for d in range(3)],
                                ["box" if kind == "volume" or d != i else "point" for d in range(3)], fd)
                        for i in range(3)])


def _edge(i: int, j: int):
    return [i != j and d in (i, j) for d in range(3)]


def _dt(u, visc, cfl, h):
    return min(cfl * h / float(u.abs().max()), cfl * h * h / visc / 6)


def _rk4(u, visc, h, les, steps, cfl=CFL):
    """RK4 with the exact closure at every stage; `les`: [ratio, kind, exact, no-model] lists, updated."""
    n = u.shape[-1]
    last = []
    for _ in range(steps):
        dt = _dt(u, visc, cfl, h)
        us, acc = u, torch.zeros_like(u)
        st = [[g[2], g[3], torch.zeros_like(g[2]), torch.zeros_like(g[3])] for g in les]
        last = []
        for s in range(4):
            k = _project(_rhs(us, visc, h), h)[0]
            wt, nx = (1, 2, 2, 1)[s], (0.5, 0.5, 1, 0)[s]
            for g, x in zip(les, st):
                H = L * g[0] / n
                ub = _filter(us, g[0], g[1])
                if g[1] == "volume":
                    ub = _project(ub, H)[0]
                m = _project(_filter(k, g[0], g[1]), H)[0] - _project(_rhs(ub, visc, H), H)[0]
                if s == 0:
                    last.append(torch.stack([ub, m]))
                for q, extra in ((0, m), (1, 0)):
                    kv = _project(_rhs(x[q], visc, H), H)[0] + extra
                    x[2 + q] += wt * kv
                    x[q] = g[2 + q] + nx * dt * kv
            acc += wt * k
            us = u + nx * dt * k
        u = u + dt / 6 * acc
        for g, x in zip(les, st):
            g[2], g[3] = g[2] + dt / 6 * x[2], g[3] + dt / 6 * x[3]
    return u, last


def _exact_step(case, seed):
    n, dt = case["n"], DTYPES[case["prec"]]
    u = _velocity(n, seed).to(dt).double()
    les = []
    for c, kind in _les(case["les"]):
        v = _filter(u, c, kind)
        v = _project(v, L * c / n)[0] if kind == "volume" else v
        les.append([c, kind, v, v])
    u, last = _rk4(u, _visc(n), L / n, les, case["steps"])
    return {"u": u, "pairs": last, "les": [les[0][2], les[0][3]]}


def _exact_euler(case, seed):
    n, c, visc = case["n"], case["ratio"], 2e-4
    h, H = L / n, L * c / n
    fd = _gaussian_exact(case)
    u = _velocity(n, seed)
    box = ["box"] * 3
    target = lambda w: _project(_filter(w, c, "volume", fd), H)[0]  # noqa: E731
    ub = target(u)
    v = {k: ub for k in NS.DNSAID_FIELDS[1:]}
    fine = _taps(c, False, "box", fd)
    for _ in range(case["steps"]):
        dt = _dt(u, visc, CFL, h)
        sig = _stress(u, visc, h)
        du, p = _project(_tensordiv(sig, h), h)
        r = {k: sig[k] + p if k[0] == k[1] else sig[k] for k in sig}
        r9 = {(i, j): _coarse(r[i, j], c, _edge(i, j), ["point" if d == j else "box" for d in range(3)], fd)
              for i in range(3) for j in range(3)}
        sdh = {k: _coarse(sig[k], c, _edge(*k), box, fd) for k in SYM6}
        uf = u
        for d in range(3):
            uf = sum(w * _at(uf, d, o - c // 2) for o, w in fine)
        s2 = {k: _coarse(t, c, _edge(*k), ["point"] * 3) for k, t in _stress(uf, visc, h).items() if k in SYM6}
        ub = target(u)
        sub = _stress(ub, visc, H)
        sl = {k: _stress(v[k], visc, H) for k in v}
        sym = {(i, j): (r9[i, j] + r9[j, i]) / 2 for i, j in r9}
        both = lambda a: {(i, j): a[i, j] if (i, j) in a else a[j, i] for i, j in r9}  # noqa: E731
        sdh, s2 = both(sdh), both(s2)
        v["u_nomo"] = _project(v["u_nomo"] + dt * _tensordiv(sl["u_nomo"], H), H)[0]
        for k, extra in (("u_c", {q: sdh[q] - s2[q] for q in r9}), ("u_cf", {q: sdh[q] - sub[q] for q in r9}),
                         ("u_cfd", {q: r9[q] - sub[q] for q in r9}), ("u_cfd_symm", {q: sym[q] - sub[q] for q in r9})):
            v[k] = v[k] + dt * _project(_tensordiv({q: sl[k][q] + extra[q] for q in r9}, H), H)[0]
        u = u + dt * du
    return {"u_les": target(u), **v}


def _hash(z):
    """splitmix64's output function on wrapping int64."""
    for sh, m in ((30, -0x40A7B892E31B1A47), (27, -0x6B2FB644ECCEEE15)):
        z = (z ^ ((z >> sh) & ((1 << (64 - sh)) - 1))) * m
    return z ^ ((z >> 31) & ((1 << 33) - 1))


def _served_start(n: int, seed: int, kpeak: float, energy: float):
    """The server's seeded initial field: counter-based normals, projected, shells scaled to the peak profile."""
    mul = 0x9E3779B97F4A7C15
    base = (seed * mul) % (1 << 64)
    base -= (1 << 64) if base >= 1 << 63 else 0
    m = torch.arange(3 * n**3, device="cuda", dtype=torch.int64)
    f = [(((_hash(base + 2 * m + q) >> 11) & ((1 << 53) - 1)).double() + 0.5) * 2.0**-53 for q in (0, 1)]
    u = (torch.sqrt(-2 * torch.log(f[0])) * torch.cos(2 * math.pi * f[1])).reshape(3, n, n, n)
    u = _project(u, L / n)[0]
    w = [torch.fft.rfftn(u[c]) / n**3 for c in range(3)]
    k = torch.fft.fftfreq(n, 1 / n, dtype=F64, device="cuda")
    k2 = k[:, None, None] ** 2 + k[None, :, None] ** 2 + k[: n // 2 + 1].abs()[None, None, :] ** 2
    shell = torch.floor(torch.sqrt(k2) + 1e-9).long()
    two = torch.full((n // 2 + 1,), 2.0, dtype=F64, device="cuda")
    two[0] = two[-1] = 1
    nsh = int(math.sqrt(3) * (n // 2)) + 1
    es = torch.zeros(nsh + 1, dtype=F64, device="cuda")
    es.index_add_(0, shell.reshape(-1), (sum(x.abs() ** 2 for x in w) / 2 * two).reshape(-1))
    q = torch.arange(nsh, dtype=F64, device="cuda")
    prof = q**4 * torch.exp(-2 * (q / kpeak) ** 2)
    fac = torch.ones_like(es)
    fac[:nsh] = torch.where(es[:nsh] > 0, torch.sqrt(energy * prof / prof.sum() / es[:nsh]), fac[:nsh])
    u = torch.stack([torch.fft.irfftn(x * fac[shell], s=(n, n, n)) * n**3 for x in w])
    return _project(u, L / n)[0]


def _exact_serve(case, seed):
    out = {"field": [], "energy": [], "time": []}
    for i, n in enumerate(_sizes(case)):
        u, t, h, visc = _served_start(n, seed + i, 4.0, 1.0), 0.0, L / n, _visc(n)
        for _ in range(case["steps"]):
            t += _dt(u, visc, CFL, h)
            u = _rk4(u, visc, h, [], 1)[0]
        out["field"].append(u)
        out["energy"].append(float((u * u).sum()) / 2 / n**3)
        out["time"].append(t)
    return {"field": out["field"], "energy": np.array(out["energy"]), "time": np.array(out["time"])}


def _conv(x, W):
    """[b, z, y, x, ci] with W [tap, ci, co], periodic."""
    out = 0
    for t in range(27):
        s = (1 - t // 9, 1 - t // 3 % 3, 1 - t % 3)
        out = out + torch.roll(x, s, dims=(1, 2, 3)) @ W[t]
    return out


def _exact_net(case, seed):
    u, m, params = _net_inputs(case, seed)
    P = [tuple(torch.from_numpy(a).cuda().double() for a in p) for p in params]
    # the input as the network holds it: its rounding is the format's, not an error of the computation
    x = u.permute(0, 2, 3, 4, 1).to(torch.bfloat16).double()
    hs, pres = [x], []
    for i, (W, b) in enumerate(P):
        pre = _conv(hs[-1], W) + b
        pres.append(pre)
        hs.append(torch.nn.functional.gelu(pre) if i < 2 else pre)
    if case["mode"] == "forward":
        return hs[-1].permute(0, 4, 1, 2, 3).contiguous()
    d = hs[-1] - m.permute(0, 2, 3, 4, 1).double()
    loss, g = float(d.square().mean()), 2 * d / d.numel()
    grads = []
    for i in (2, 1, 0):
        W, _ = P[i]
        if i < 2:
            q = pres[i]
            g = g * (0.5 * (1 + torch.erf(q / math.sqrt(2))) + q * torch.exp(-q * q / 2) / math.sqrt(2 * math.pi))
        gf = g.reshape(-1, g.shape[-1])
        dW = torch.stack([torch.roll(hs[i], (1 - t // 9, 1 - t // 3 % 3, 1 - t % 3), dims=(1, 2, 3))
                          .reshape(-1, W.shape[1]).T @ gf for t in range(27)])
        grads.insert(0, (dW, gf.sum(0)))
        if i:
            g = _conv(g, W.flip(0).transpose(1, 2))
    flat = []
    for (kp, np_), (W, b) in zip(SHAPES, grads):
        Wp = torch.zeros((27, kp, np_), dtype=F64, device="cuda")
        Wp[:, : W.shape[1], : W.shape[2]] = W
        bp = torch.zeros(np_, dtype=F64, device="cuda")
        bp[: b.shape[0]] = b
        flat += [Wp.reshape(-1), bp]
    return {"loss": loss, "grad": torch.cat(flat)}


def _exact_burgers(case, seed):
    nh, nH = case["nh"], case["nH"]
    Lb, visc, c = 2 * math.pi, 5e-4, nh // nH
    h, H = Lb / nh, Lb / nH
    u = torch.from_numpy(_burgers_start(case, seed)).cuda()
    if case["filter"] == "gaussian":
        s2 = (case["delta"] * c) ** 2 / 12
        R = round(3 * math.sqrt(s2))
        les = np.exp(-(np.arange(-R, R + 1.0) ** 2) / (2 * s2))
        les /= les.sum()
    else:
        R = round(case["delta"] * c) // 2
        les = np.full(2 * R + 1, 1 / (2 * R + 1))
    dbl = np.convolve(np.full(c, 1 / c), les)
    face = c * torch.arange(1, nH + 1, device="cuda") - 1
    cen = face - c // 2

    def at(f, w, pos):
        r = torch.arange(-(len(w) // 2), len(w) // 2 + 1, device="cuda")
        return f[:, (pos[:, None] + r) % nh] @ torch.from_numpy(w).cuda()

    def stress(f, d):
        a = torch.roll(f, 1, 1)
        return -((a + f) ** 2) / 8 + visc * (f - a) / d

    def dcoll(p, d):
        return (torch.roll(p, -1, 1) - p) / d

    v0 = at(u, dbl, face)
    V = {k: v0 for k in ("nomodel", "class_m", "class_p", "swapfil")}
    t = torch.zeros(u.shape[0], dtype=F64, device="cuda")
    while bool((act := t < case["tstop"]).any()):
        dt = torch.minimum(CFL * torch.minimum(h / u.abs().amax(1), torch.full_like(t, h * h / visc)), case["tstop"] - t)
        dt = torch.where(act, dt, torch.zeros_like(dt))
        d = dt[:, None]
        su = stress(u, h)
        fsu, vsu, vu = at(su, les, cen), at(su, dbl, cen), at(u, dbl, face)
        a, b = at(u, dbl, cen - 1), at(u, dbl, cen)
        svu, sVU = stress(vu, H), -((a + b) ** 2) / 8 + visc * (b - a) / h
        for k, e in (("nomodel", 0), ("class_m", vsu - sVU), ("class_p", vsu - svu), ("swapfil", fsu - svu)):
            V[k] = V[k] + d * dcoll(stress(V[k], H) + e, H)
        u = u + d * dcoll(su, h)
        t = torch.where(act, t + dt, t)
    full = torch.cat([at(u, dbl, q) for q in torch.arange(nh, device="cuda").split(512)], 1)
    return {"dns_ref": u, "dns_ref_fil": full, "dns_fil": full[:, face], **V}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("stage", "rhs"):
        n, dt = case["n"], DTYPES[case["prec"]]
        du = _rhs(_velocity(n, seed).to(dt).double(), _visc(n), L / n)
        if kind == "rhs":
            return du
        k, p = _project(du, L / n)
        return {"k": k, "p": p}
    return {"step": _exact_step, "euler": _exact_euler, "serve": _exact_serve, "net": _exact_net,
            "burgers": _exact_burgers}[kind](case, seed)
