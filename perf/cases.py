"""Performance cases of the solver: what its users run, through the public Python mirror of the
C ABI (``cushg_b200.shg``), with a 64-bit restatement of the model to check the results.

A case names one kind of call and its sizes:

  single    one plain run (``shg.solve_device``, or ``shg.solve`` with host buffers)
  sweep     a mixed batch of plain runs, ``params.config_sweep`` (``shg.solve_batch_device``)
  batch     a batch of equal plain runs (``shg.solve_batch_device``)
  grad      adjoint gradients with a poling vector (``shg.grad`` / ``shg.grad_batch``)
  thermal   thermal runs (``shg.solve_device`` / ``shg.thermal_batch``), Jacobi or direct
  sweeps    Jacobi sweeps of the heat equation in place (``shg.heat_sweeps_device``)
  steady    the steady temperature of a heat source (``shg.heat_steady_device``)

Beams, powers and oven temperatures are drawn from the seed around the values of the standard
workloads in ``cushg_b200/params.py``.  Results that are scalars (powers, derivatives) are
returned in the precision of the run they belong to.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from cushg_b200 import params as P
from cushg_b200 import shg

CDT = {32: torch.complex64, 64: torch.complex128}
RDT = {32: torch.float32, 64: torch.float64}
PLAIN_SIDES = (32, 48, 64, 96, 128, 192, 256, 512)
THERMAL_SIDES = (32, 64, 128, 256, 512)


# ------------------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest run: one 64 x 64 point of a study, where launches and latency count
        {"name": "single_64_f64", "kind": "single", "n": 64, "nz": 100, "precision": 64, "host": False},
        # the reference's compiled-in configuration (128 x 128 x 100, FP32) into host arrays
        {"name": "single_128_f32_host", "kind": "single", "n": 128, "nz": 100, "precision": 32, "host": True},
        # one run at full transverse resolution in FP64
        {"name": "single_256_f64", "kind": "single", "n": 256, "nz": 400, "precision": 64, "host": False},
        # the parameter sweep of the reference's shell script, 256 points as one guarded batch
        {"name": "sweep_256_f32", "kind": "sweep", "count": 256, "precision": 32, "guard": 1e-5},
        # runs whose planes exceed a cluster's shared memory
        {"name": "batch_512_f32", "kind": "batch", "n": 512, "nz": 200, "count": 8, "precision": 32},
        # one optimiser step: gradient of the SH power by waist, focus, oven and 399 poling phases
        {"name": "grad_256_f32", "kind": "grad", "n": 256, "nz": 400, "count": 1, "precision": 32},
        # gradients of many starting points at once, in FP64
        {"name": "grad_batch_256_f64", "kind": "grad", "n": 256, "nz": 400, "count": 18, "precision": 64},
        # the reference's thermal run: Jacobi to max|dT| < 1e-6 K in each outer iteration
        {"name": "thermal_128_jacobi_f64", "kind": "thermal", "n": 128, "nz": 200, "count": 1, "precision": 64,
         "direct": False, "outer": 2, "sweeps": 0, "grad": False, "boundary": 0},
        # a temperature study at high resolution: ovens side by side, solved directly, with dJ/dT
        {"name": "thermal_512_direct_grad_f32", "kind": "thermal", "n": 512, "nz": 200, "count": 4, "precision": 32,
         "direct": True, "outer": 2, "sweeps": 0, "grad": True, "boundary": 0},
        # the heat equation alone: sweeps on a grid far larger than L2
        {"name": "sweeps_512_f32", "kind": "sweeps", "n": 512, "nz": 250, "count": 100, "precision": 32, "boundary": 0},
        # and its steady state, large and small with odd slice counts and both boundary models
        {"name": "steady_512_f32", "kind": "steady", "n": 512, "nz": 501, "precision": 32, "boundary": 0},
        {"name": "steady_96_oven_f64", "kind": "steady", "n": 96, "nz": 37, "precision": 64, "boundary": 1},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["single", "single", "sweep", "batch", "grad", "thermal", "thermal", "sweeps", "steady"])
    prec = rng.choice([32, 64])
    if kind == "single":
        n = rng.choice(PLAIN_SIDES)
        return {"kind": kind, "n": n, "nz": _log_int(rng, 30, 400), "precision": prec, "host": rng.random() < 0.3}
    if kind == "sweep":
        return {"kind": kind, "count": _log_int(rng, 3, 200), "precision": 32, "guard": rng.choice([0.0, 1e-5])}
    if kind == "batch":
        n = rng.choice(PLAIN_SIDES)
        most = 8 if n == 512 else 32 if n >= 192 else 128
        return {"kind": kind, "n": n, "nz": _log_int(rng, 30, 250), "count": _log_int(rng, 2, most), "precision": prec}
    if kind == "grad":
        return {"kind": kind, "n": rng.choice([64, 128, 256]), "nz": _log_int(rng, 30, 300),
                "count": _log_int(rng, 1, 16), "precision": prec}
    if kind == "thermal":
        n = rng.choice(THERMAL_SIDES)
        direct = rng.random() < 0.5
        grad = direct and n >= 256 and rng.random() < 0.5
        return {"kind": kind, "n": n, "nz": _log_int(rng, 21, 120 if n == 512 else 300),
                "count": _log_int(rng, 1, 3 if n == 512 else 6), "precision": prec, "direct": direct,
                "outer": rng.randint(1, 3), "sweeps": 0 if direct else _log_int(rng, 100, 3000 if n < 256 else 300),
                "grad": grad, "boundary": rng.choice([0, 0, 1])}
    n = rng.choice([48, 64, 96, 128, 192, 256, 512])
    nz = _log_int(rng, 15, 400)
    if kind == "sweeps":
        return {"kind": kind, "n": n, "nz": nz, "count": _log_int(rng, 20, 2000 if n <= 128 else 300 if n <= 256 else 60),
                "precision": prec, "boundary": rng.choice([0, 1])}
    return {"kind": kind, "n": n, "nz": nz, "precision": prec, "boundary": rng.choice([0, 1])}


# ------------------------------------------------------------------------------ inputs
def _beam(rng, n, nz, prec, thermal=0):
    """One run near phase matching (27 C): the values a user tunes around."""
    lz = float(rng.choice([10000.0, 20000.0]))
    p = P.workload(n, nz, lz, float(math.exp(rng.uniform(math.log(2.0), math.log(40.0)))), float(rng.uniform(25.0, 50.0)),
                   float(rng.uniform(0.3, 0.7)) * lz, float(rng.uniform(25.0, 30.0)), precision=prec, thermal=thermal)
    if thermal:  # studies of beams and ovens in one crystal: its window and length stay
        p.lx = p.ly = 12.0 * 40.0
        p.lz, p.focus = 20000.0, p.focus / lz * 20000.0
    return p


def _params(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "sweep":
        # the grids of the standard sweep with the beams, ovens and crystals of this seed
        grids = P.config_sweep(case["count"], seed=0, precision=case["precision"])
        ps = [P.workload(g.nx, g.nz, b.lz, b.power, b.waist, b.focus, b.temp, precision=case["precision"])
              for g, b in zip(grids, P.config_sweep(case["count"], seed=seed))]
        for p in ps:
            p.fp32_guard = case["guard"]
        return ps
    if kind == "single" and case["host"]:
        # the reference's own crystal and rectangular window, its beam varied
        p = P.reference_defaults()
        p.nx = p.ny = case["n"]
        p.nz, p.precision = case["nz"], case["precision"]
        p.power, p.waist = float(rng.uniform(20.0, 40.0)), float(rng.uniform(25.0, 35.0))
        p.temp = p.t_peltier = float(rng.uniform(55.0, 56.5))
        return [p]
    if kind in ("sweeps", "steady"):
        p = P.workload(case["n"], case["nz"], 20000.0, 30.0, 40.0, 10000.0, float(rng.uniform(30.0, 65.0)),
                       precision=case["precision"], thermal=1)
        p.boundary = case["boundary"]
        return [p]
    ps = [_beam(rng, case["n"], case["nz"], case["precision"], 1 if kind == "thermal" else 0)
          for _ in range(case.get("count", 1))]
    if kind == "thermal":
        for p in ps:
            p.boundary = case["boundary"]
            p.max_outer = case["outer"]
            p.jacobi_tol = 1e-6
            p.check_every = 1000
            p.conv_rule = P.SHG_CONV_FIXED if case["sweeps"] else P.SHG_CONV_MAXABS
            p.max_sweeps = case["sweeps"]
            p.heat_solver = P.SHG_HEAT_DIRECT if case["direct"] else P.SHG_HEAT_JACOBI
            # absorption strong enough to heat the crystal by a fraction of a kelvin
            p.alpha_p, p.alpha_s = 2e-7, 4e-6
    return ps


def _polings(ps, seed):
    rng = np.random.default_rng(seed + 1)
    return [rng.normal(0.0, 0.1, p.nz - 1) for p in ps]


def _heat_fields(case, p, seed):
    """A temperature field on its way to the steady state and a focused beam's heat source."""
    dt = RDT[case["precision"]]
    n, nz = p.nx, p.nz
    g = torch.Generator(device="cuda").manual_seed(seed)
    T = torch.full((nz, n, n), p.temp, dtype=dt, device="cuda")
    x = torch.linspace(-6.0, 6.0, n, dtype=torch.float64, device="cuda")
    w2 = 1.0 + torch.linspace(-1.0, 1.0, nz, dtype=torch.float64, device="cuda") ** 2
    r2 = x[None, None, :] ** 2 + x[None, :, None] ** 2
    peak = 4.0 * p.kappa / p.waist ** 2  # about a kelvin across the beam
    Q = (peak * torch.exp(-2.0 * r2 / w2[:, None, None]) / w2[:, None, None])
    Q = (Q * (1.0 + 0.1 * torch.rand((nz, 1, 1), dtype=torch.float64, device="cuda", generator=g))).to(dt)
    if case["kind"] == "sweeps":
        T += 0.1 * torch.rand((nz, n, n), dtype=dt, device="cuda", generator=g)
        oven = _dirichlet(n, case["boundary"])
        T[:, oven] = p.temp
    return T, Q


def _dirichlet(n, boundary):
    m = torch.zeros((n, n), dtype=torch.bool, device="cuda")
    m[0] = True
    if boundary:
        m[-1] = m[:, 0] = m[:, -1] = True
    return m


def prepare(case, seed):
    ps = _params(case, seed)
    st = {"case": case, "ps": ps, "prec": case["precision"]}
    kind = case["kind"]
    if kind == "grad":
        st["pol"] = _polings(ps, seed)
    elif kind in ("sweeps", "steady"):
        st["T"], st["Q"] = _heat_fields(case, ps[0], seed)
    elif not (kind == "single" and case["host"]):
        # one buffer for all output fields, an instance's pump and SH plane after each other
        total = sum(2 * p.nx * p.nx for p in ps)
        st["out"] = torch.empty(total, dtype=CDT[st["prec"]], device="cuda")
        st["pump"], st["sig"], o = [], [], 0
        for p in ps:
            k = p.nx * p.nx
            st["pump"].append(st["out"][o:o + k].view(p.nx, p.nx))
            st["sig"].append(st["out"][o + k:o + 2 * k].view(p.nx, p.nx))
            o += 2 * k
        if kind == "thermal":
            st["T"] = [torch.empty((p.nz, p.nx, p.nx), dtype=RDT[st["prec"]], device="cuda") for p in ps]
    return st


def _scalars(v, prec):
    return np.asarray(v, dtype=np.float64 if prec == 64 else np.float32)


def run(st):
    case, ps, prec = st["case"], st["ps"], st["prec"]
    kind = case["kind"]
    if kind == "single":
        if case["host"]:
            r = shg.solve(ps[0])
            return {"pump": r.pump, "signal": r.signal, "power": _scalars([r.stats.sh_power, r.stats.pump_power], prec)}
        s = shg.solve_device(ps[0], st["pump"][0], st["sig"][0])
        return {"pump": st["pump"][0], "signal": st["sig"][0], "power": _scalars([s.sh_power, s.pump_power], prec)}
    if kind in ("sweep", "batch"):
        power = shg.solve_batch_device(ps, st["pump"], st["sig"])
        return {"fields": st["out"], "power": _scalars(power, prec)}
    if kind == "grad":
        g = [shg.grad(ps[0], st["pol"][0])] if len(ps) == 1 else shg.grad_batch(ps, st["pol"])
        return {k: _scalars(np.concatenate([np.atleast_1d(d[k]) for d in g]), prec)
                for k in ("sh_power", "d_waist", "d_focus", "d_temp", "d_poling")}
    if kind == "thermal":
        if len(ps) == 1 and not case["grad"]:
            s = [shg.solve_device(ps[0], st["pump"][0], st["sig"][0], temperature_out=st["T"][0])]
            d = None
        else:
            s, d = shg.thermal_batch(ps, st["pump"], st["sig"], st["T"], grad=case["grad"])
        out = {"fields": st["out"], "T": st["T"], "power": _scalars([x.sh_power for x in s], prec),
               "outer": [int(x.outer_iterations) for x in s], "sweeps": [int(x.jacobi_sweeps) for x in s]}
        if d is not None:
            out["d_temp"] = _scalars(d, prec)
        return out
    if kind == "sweeps":
        shg.heat_sweeps_device(ps[0], st["T"], st["Q"], case["count"])
        return st["T"]
    # (the residual that heat_steady_device returns is rounding noise, not a result)
    shg.heat_steady_device(ps[0], st["T"], st["Q"])
    return st["T"]


# ------------------------------------------------------------------------------ work
def _march_flops(n, steps):
    """Four 2D transforms, two propagator products and two RK4 applications per point and step."""
    return n * n * steps * (4 * 5 * math.log2(n * n) + 2 * 6 + 2 * 192)


def _heat_flops(n, nz):
    """The steady solve as separable dense transforms (the x one folded) and a tridiagonal solve."""
    return n * n * nz * (2.0 * (2 * n + n) + 30.0)


def work(case):
    kind = case["kind"]
    c = 2 * case["precision"] // 8
    if kind == "sweep":
        ps = _params(case, 0)
        return {"bytes": float(sum(2 * c * p.nx * p.nx for p in ps)),
                "flops": float(sum(_march_flops(p.nx, p.nz - 1) for p in ps))}
    n, nz, k = case["n"], case["nz"], case.get("count", 1)
    vox = float(n * n * nz)
    if kind in ("single", "batch"):
        return {"bytes": float(2 * c * n * n * k), "flops": float(k * _march_flops(n, nz - 1))}
    if kind == "grad":  # the forward march and its vector-Jacobian product
        return {"bytes": float(16 * nz * k), "flops": float(3 * k * _march_flops(n, nz - 1))}
    if kind == "thermal":
        # Jacobi to a tolerance: about 16500 sweeps an outer iteration (66004 in four at 128 x 128 x 200)
        heat = _heat_flops(n, nz) if case["direct"] else 11.0 * vox * (case["sweeps"] or 16500)
        march = _march_flops(n, nz) + 60.0 * vox
        if case["grad"]:
            heat, march = 2 * heat, 3 * march
        return {"bytes": float(k * (2 * c * n * n + c / 2 * vox)), "flops": float(k * case["outer"] * (heat + march))}
    if kind == "sweeps":  # T read and written once, Q read once
        return {"bytes": 3 * c / 2 * vox, "flops": 11.0 * vox * case["count"]}
    return {"bytes": 3 * c / 2 * vox, "flops": _heat_flops(n, nz)}


# ------------------------------------------------------------------------------ 64-bit restatement
# The reference's model (src/headers/Crystal.h, PhaseMatching.h, Efields.h, Solver.h, Tfield.h)
# in torch complex128 / float64.
PI = math.pi
CL = 299792458 * 1e6 / 1e12
EPS0 = 8.8541878128e-12 * 1e12 / 1e6


def _n(L, T):
    A, B, C, D = 4.502483, 0.007294, 0.185087, -0.02357
    E, F, G, H = 0.073423, 0.199595, 0.001, 7.99724
    tk = T + 273.15
    b, c, l2 = 3.483933e-8 * tk * tk, 1.607839e-8 * tk * tk, L * L
    return torch.sqrt(A + (B + b) / (l2 - (C + c) ** 2) + E / (l2 - F * F) + G / (l2 - H * H) + D * l2)


def _dk(lp, period, T):
    ls, d = 0.5 * lp, T - 25.0
    return 2 * PI * (2 * _n(lp, T) / lp - _n(ls, T) / ls + 1 / (period * (1 + 2.2e-6 * d - 5.9e-9 * d * d)))


def _col(ps, name):
    return torch.tensor([getattr(p, name) for p in ps], dtype=torch.float64, device="cuda").view(-1, 1, 1)


def _optics(ps, Tc, waist=None, focus=None):
    """Pump at z = 0, the propagators and the constants of one optical pass, B instances of one side."""
    n = ps[0].nx
    lp = ps[0].lambda_p
    ls = 0.5 * lp
    o = {"lp": lp, "ls": ls}
    waist = _col(ps, "waist") if waist is None else waist
    focus = _col(ps, "focus") if focus is None else focus
    o["np"], o["ns"] = _n(lp, Tc), _n(ls, Tc)
    o["dx"], o["dy"] = _col(ps, "lx") / (n - 1), _col(ps, "ly") / (n - 1)
    o["dz"] = _col(ps, "lz") / torch.tensor([p.nz - 1 for p in ps], dtype=torch.float64, device="cuda").view(-1, 1, 1)
    o["dQ"] = 2.0 * _col(ps, "deff") / PI
    w2 = waist * waist
    zr = PI * o["np"] * w2 / lp
    amp = torch.sqrt(4 * _col(ps, "power") / (EPS0 * CL * PI * o["np"] * w2))
    M = torch.complex(torch.ones_like(zr), -focus / zr)
    i = torch.arange(n, dtype=torch.float64, device="cuda")
    ax, ay = (i.view(1, 1, -1) - 0.5 * n) * o["dx"], (i.view(1, -1, 1) - 0.5 * n) * o["dy"]
    o["pump"] = amp / M * torch.exp(-(ax * ax + ay * ay) / (w2 * M))
    s = torch.where(i < n // 2, i, i - n)
    fx, fy = s.view(1, 1, -1) / (n * o["dx"]), s.view(1, -1, 1) / (n * o["dy"])
    for f, nn, lam, rho in (("p", o["np"], lp, "rho_p"), ("s", o["ns"], ls, "rho_s")):
        k = 2 * PI * nn / lam
        th = -o["dz"] * (2 * PI * PI / k * (fx * fx + fy * fy) + 2 * PI * torch.tan(_col(ps, rho)) * fx)
        o["prop_" + f] = torch.polar(torch.ones_like(th), th)
    o["hap"], o["has"] = 0.5 * _col(ps, "alpha_p"), 0.5 * _col(ps, "alpha_s")
    return o


def _rk4(A, S, cps, css, hap, has, qs, dz):
    """The reference's RK4: stages without dz, phases at z, z + dz/4 (twice), z + dz/2."""
    def f(a, s, j):
        return (cps[j] * s * a.conj() - hap * a,
                css[j] * a * a - (has + qs * (s.real ** 2 + s.imag ** 2)) * s)
    k1 = f(A, S, 0)
    k2 = f(A + 0.5 * k1[0], S + 0.5 * k1[1], 1)
    k3 = f(A + 0.5 * k2[0], S + 0.5 * k2[1], 1)
    k4 = f(A + k3[0], S + k3[1], 2)
    return tuple(v + (a + 2 * b + 2 * c + d) * (dz / 6) for v, a, b, c, d in zip((A, S), k1, k2, k3, k4))


def _phases(kp, ks, phis):
    one = [torch.polar(torch.ones_like(p), p) for p in phis]
    return [1j * kp * e.conj() for e in one], [1j * ks * e for e in one]


def _plain_setup(ps, temp, waist=None, focus=None):
    o = _optics(ps, temp, waist, focus)
    o["dk"] = _dk(o["lp"], _col(ps, "period"), temp)
    o["kp"], o["ks"] = PI * o["dQ"] / (o["np"] * o["lp"]), 0.5 * PI * o["dQ"] / (o["ns"] * o["ls"])
    o["qs"] = 0.5 * _col(ps, "beta_s") * 0.5 * CL * EPS0 * o["ns"]
    return o


def _plain_step(o, A, S, z, pol):
    c = _phases(o["kp"], o["ks"], [(z + o["dz"] * t) * o["dk"] + pol for t in (0.0, 0.25, 0.5)])
    A, S = _rk4(A, S, *c, o["hap"], o["has"], o["qs"], o["dz"])
    A = torch.fft.ifft2(torch.fft.fft2(A) * o["prop_p"])
    S = torch.fft.ifft2(torch.fft.fft2(S) * o["prop_s"])
    return _rk4(A, S, *c, o["hap"], o["has"], o["qs"], o["dz"])


def _plain_exact(ps):
    """Fields and [SH, pump] powers of plain runs, in the order of ps."""
    res = [None] * len(ps)
    for n in sorted({p.nx for p in ps}):
        idx = sorted((i for i in range(len(ps)) if ps[i].nx == n), key=lambda i: -ps[i].nz)
        for lo in range(0, len(idx), 64):
            part = idx[lo:lo + 64]
            sub = [ps[i] for i in part]
            o = _plain_setup(sub, _col(sub, "temp"))
            A = o["pump"].clone()
            S = torch.zeros_like(A)
            live = len(sub)
            for s in range(sub[0].nz - 1):
                while sub[live - 1].nz - 1 <= s:
                    live -= 1  # the shortest marches come last
                q = {k: v[:live] if torch.is_tensor(v) else v for k, v in o.items()}
                A[:live], S[:live] = _plain_step(q, A[:live], S[:live], s * q["dz"], 0.0)
            w = 0.5 * EPS0 * CL * o["dx"] * o["dy"]
            for k, i in enumerate(part):
                res[i] = (A[k], S[k], float((w * o["ns"])[k] * S[k].abs().square().sum()),
                          float((w * o["np"])[k] * A[k].abs().square().sum()))
    return res


def _grad_exact(ps, pols):
    """SH power and its derivatives by automatic differentiation, one checkpoint per step."""
    from torch.utils.checkpoint import checkpoint

    v = {k: _col(ps, k).requires_grad_() for k in ("waist", "focus", "temp")}
    pol = torch.tensor(np.stack(pols), device="cuda").requires_grad_()
    o = _plain_setup(ps, v["temp"], v["waist"], v["focus"])
    keys = ("dz", "dk", "kp", "ks", "qs", "hap", "has", "prop_p", "prop_s")

    def step(A, S, z, ph, *vals):
        return _plain_step(dict(zip(keys, vals)), A, S, z, ph)

    A = o["pump"]
    S = torch.zeros_like(A)
    for s in range(ps[0].nz - 1):
        A, S = checkpoint(step, A, S, s * o["dz"], pol[:, s].view(-1, 1, 1), *[o[k] for k in keys], use_reentrant=False)
    J = (0.5 * EPS0 * CL * o["ns"] * o["dx"] * o["dy"] * (S.real ** 2 + S.imag ** 2)).sum(dim=(1, 2))
    g = torch.autograd.grad(J.sum(), [v["waist"], v["focus"], v["temp"], pol])
    return {"sh_power": J.detach(), "d_waist": g[0].flatten(), "d_focus": g[1].flatten(), "d_temp": g[2].flatten(),
            "d_poling": g[3].flatten()}


def _heat_geometry(p):
    d = [p.lx / (p.nx - 1), p.ly / (p.ny - 1), p.lz / (p.nz - 1)]
    return d, [p.h_conv * h / p.kappa for h in d]


def _sweep_exact(p, T, Q, count):
    """Jacobi sweeps as updates of whole blocks: the inner points, and each face, edge and vertex
    by the sum of its three directions' one-dimensional rows (scaled to a common form)."""
    (dx, dy, dz), bi = _heat_geometry(p)
    n, nz = p.nx, p.nz
    dev = T.device
    ones = [torch.ones(m, dtype=torch.float64, device=dev) for m in (n, n, nz)]
    diag, rhs = [], []
    for m, h, b, one in zip((n, n, nz), (dx, dy, dz), bi, ones):
        a = one * (2.0 / h ** 2)
        r = one * 0.0
        a[0] = a[-1] = 2.0 * (1.0 + b) / h ** 2
        r[0] = r[-1] = 2.0 * b * p.t_inf / h ** 2
        diag.append(a)
        rhs.append(r)
    D = diag[2].view(-1, 1, 1) + diag[1].view(1, -1, 1) + diag[0].view(1, 1, -1)
    R = rhs[2].view(-1, 1, 1) + rhs[1].view(1, -1, 1) + rhs[0].view(1, 1, -1)
    R[1:-1, 1:-1, 1:-1] += Q[1:-1, 1:-1, 1:-1] / p.kappa
    fixed = _dirichlet(n, p.boundary)
    T = T.clone()
    keep = T[:, fixed].clone()
    for _ in range(count):
        acc = R.clone()
        for ax, h in ((2, dx), (1, dy), (0, dz)):
            m = T.shape[ax]
            acc.narrow(ax, 1, m - 2).add_((T.narrow(ax, 0, m - 2) + T.narrow(ax, 2, m - 2)) / h ** 2)
            acc.select(ax, 0).add_(T.select(ax, 1) * (2.0 / h ** 2))
            acc.select(ax, m - 1).add_(T.select(ax, m - 2) * (2.0 / h ** 2))
        T = acc.div_(D)
        T[:, fixed] = keep
    return T


def _steady_exact(p, T, Q):
    """The sweeps' fixed point by separable eigenvectors in x and y and along z."""
    (dx, dy, dz), bi = _heat_geometry(p)
    n, nz = p.nx, p.nz
    top = p.boundary == 0
    ranges = [(0, n, True, True) if top else (1, n - 1, False, False),
              (1, n, False, True) if top else (1, n - 1, False, False), (0, nz, True, True)]
    modes = []
    for (lo, hi, rl, rh), h, b in zip(ranges, (dx, dy, dz), bi):
        m = hi - lo
        M = torch.diag(torch.full((m,), 2.0)) - torch.diag(torch.ones(m - 1), 1) - torch.diag(torch.ones(m - 1), -1)
        M = M.to(torch.float64)
        s = torch.ones(m, dtype=torch.float64)
        if rl:  # the end rows, made symmetric by the diagonal scaling s
            M[0, 0], M[0, 1], M[1, 0] = 2.0 * (1.0 + b), -math.sqrt(2.0), -math.sqrt(2.0)
            s[0] = math.sqrt(0.5)
        if rh:
            M[-1, -1], M[-1, -2], M[-2, -1] = 2.0 * (1.0 + b), -math.sqrt(2.0), -math.sqrt(2.0)
            s[-1] = math.sqrt(0.5)
        lam, V = torch.linalg.eigh((M / h ** 2).to("cuda"))
        s = s.to("cuda")
        modes.append((lam, V.T * s, V / s[:, None]))  # forward (mode, point), inverse (point, mode)
    xs, ys = slice(ranges[0][0], ranges[0][1]), slice(ranges[1][0], ranges[1][1])
    R = torch.zeros_like(T)
    R[1:-1, 1:-1, 1:-1] = Q[1:-1, 1:-1, 1:-1] / p.kappa
    R[0] += 2 * bi[2] * p.t_inf / dz ** 2
    R[-1] += 2 * bi[2] * p.t_inf / dz ** 2
    if top:
        R[:, :, 0] += 2 * bi[0] * p.t_inf / dx ** 2
        R[:, :, -1] += 2 * bi[0] * p.t_inf / dx ** 2
        R[:, -1] += 2 * bi[1] * p.t_inf / dy ** 2
        R[:, 1] += T[:, 0] / dy ** 2
    else:
        R[:, 1] += T[:, 0] / dy ** 2
        R[:, -2] += T[:, -1] / dy ** 2
        R[:, :, 1] += T[:, :, 0] / dx ** 2
        R[:, :, -2] += T[:, :, -1] / dx ** 2
    b = R[:, ys, xs]
    for axis, (_, F, _) in zip((2, 1, 0), modes):
        b = torch.movedim(torch.tensordot(b, F, dims=([axis], [1])), -1, axis)
    b = b / (modes[2][0].view(-1, 1, 1) + modes[1][0].view(1, -1, 1) + modes[0][0].view(1, 1, -1))
    for axis, (_, _, G) in zip((2, 1, 0), modes):
        b = torch.movedim(torch.tensordot(b, G, dims=([axis], [1])), -1, axis)
    out = T.clone()
    out[:, ys, xs] = b
    return out


def _thermal_exact(p, direct, sweeps, outers):
    """One thermal run with `outers` outer iterations: fields, temperature and SH power."""
    n, nz = p.nx, p.nz
    lp, ls = p.lambda_p, 0.5 * p.lambda_p
    T = torch.full((nz, n, n), p.temp, dtype=torch.float64, device="cuda")
    T[:, _dirichlet(n, p.boundary)] = p.t_peltier
    Q = torch.zeros_like(T)
    for _ in range(outers):
        T = _steady_exact(p, T, Q) if direct else _sweep_exact(p, T, Q, sweeps)
        o = _optics([p], T[0, n // 2, n // 2].view(1, 1, 1))
        dz, q = o["dz"], 0.5 * CL * EPS0
        A = o["pump"].clone()
        S = torch.zeros_like(A)
        run_dk = torch.zeros((1, n, n), dtype=torch.float64, device="cuda")
        for s in range(nz):
            npv, nsv = _n(lp, T[s:s + 1]), _n(ls, T[s:s + 1])
            run_dk = run_dk + _dk(lp, p.period, T[s:s + 1])
            c = _phases(PI * o["dQ"] / lp / npv, 0.5 * PI * o["dQ"] / ls / nsv,
                        [run_dk * (dz * t + s * dz) / (s + 1) for t in (0.0, 0.25, 0.5)])
            qs = 0.5 * p.beta_s * q * nsv
            if s == nz - 1:
                fields = (A, S)
                power = float((q * o["dx"] * o["dy"] * nsv * S.abs().square()).sum())
            A, S = _rk4(A, S, *c, o["hap"], o["has"], qs, dz)
            A = torch.fft.ifft2(torch.fft.fft2(A) * o["prop_p"])
            S = torch.fft.ifft2(torch.fft.fft2(S) * o["prop_s"])
            A, S = _rk4(A, S, *c, o["hap"], o["has"], qs, dz)
            a2, s2 = A.abs().square(), S.abs().square()
            Q[s] = (p.alpha_p * q * npv * a2 + p.alpha_s * q * nsv * s2 + p.beta_s * (q * nsv * s2) ** 2)[0]
    return fields[0][0], fields[1][0], T, power


def exact(case, seed):
    ps = _params(case, seed)
    kind = case["kind"]
    with torch.no_grad():
        if kind in ("single", "sweep", "batch"):
            r = _plain_exact(ps)
            if kind == "single":
                return {"pump": r[0][0], "signal": r[0][1], "power": np.asarray(r[0][2:])}
            return {"fields": torch.cat([f.flatten() for x in r for f in x[:2]]), "power": np.asarray([x[2] for x in r])}
        if kind == "thermal":
            if not case["direct"] and not case["sweeps"]:
                return None  # tens of thousands of sweeps to a tolerance
            # a direct solve in FP64 may settle before its last outer iteration; within three it does not
            r = [_thermal_exact(p, case["direct"], case["sweeps"], case["outer"]) for p in ps]
            out = {"fields": torch.cat([f.flatten() for x in r for f in x[:2]]), "T": [x[2] for x in r],
                   "power": np.asarray([x[3] for x in r]), "outer": None, "sweeps": None}
            if case["grad"]:
                out["d_temp"] = None  # through the whole coupled run
            return out
        if kind in ("sweeps", "steady"):
            T, Q = _heat_fields(case, ps[0], seed)
            T, Q = T.double(), Q.double()
            return _sweep_exact(ps[0], T, Q, case["count"]) if kind == "sweeps" else _steady_exact(ps[0], T, Q)
    return _grad_exact(ps, _polings(ps, seed))
