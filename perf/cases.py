"""Timed cases of the framework: what a user's program has it do, through its public entry
points, from one small solve to the 512-solve sweep and the full THERMAL run.

``listed()`` gives the cases, ``draw(rng)`` one more of the same ranges, ``prepare`` the inputs
and handles a program holds before the call, ``run`` one pass, ``work`` the least bytes and
operations of a pass, and ``exact`` the same outputs from plain torch in 64 bits. ``exact``
keeps the scalars that the method itself defines in float (refractive indices, phase mismatch,
slice positions, grid spacings: the phase mismatch is a difference of nearly equal floats, so
another rounding of it is another crystal) and does everything per point in double.
"""
import ctypes
import math
import random

import numpy as np
import torch
import torch.utils.checkpoint

from shg_focused_gaussian_beams_gb300 import _lib
from shg_focused_gaussian_beams_gb300 import workloads as W
from shg_focused_gaussian_beams_gb300.solver import Solver, Sweep, ThermalGradBatch

F = np.float32
DEV = "cuda"
CRYSTALS = {"reference": W.CRYSTAL_REFERENCE, "qpm50": W.CRYSTAL_QPM50, "ppln": W.CRYSTAL_PPLN_QPM50}


# ---------------------------------------------------------------------------------------
# Cases

def listed():
    return [
        # a quick look at a beam on a coarse grid: launches and host calls are all of it
        {"name": "solve_32x48", "kind": "solve", "n": 32, "nz": 48, "crystal": "qpm50"},
        # the stock command line's grid and crystal (64 x 64 x 200), one solve
        {"name": "solve_64x200", "kind": "solve", "n": 64, "nz": 200, "crystal": "reference"},
        # the plain 128 x 128 x 200 benchmark solve
        {"name": "solve_128x200", "kind": "solve", "n": 128, "nz": 200, "crystal": "qpm50"},
        # a full-size solve of a field the caller holds on the device, with an SH seed
        {"name": "field_256x400", "kind": "field", "n": 256, "nz": 400, "crystal": "qpm50"},
        # a parameter scan as the sweep script makes it: a few powers, waists and temperatures
        {"name": "sweep_24", "kind": "sweep", "count": 24, "mixed": False, "n": 64, "nz": 200, "crystal": "reference"},
        # the 512-solve benchmark sweep of mixed grids and lengths
        {"name": "sweep_512", "kind": "sweep", "count": 512, "mixed": True, "n": 256, "nz": 400, "crystal": "qpm50"},
        # the gradient of the converted power in pump field and run parameters, 20 checkpoints
        {"name": "gradient_256x400", "kind": "gradient", "n": 256, "nz": 400, "crystal": "qpm50", "checkpoints": 20},
        # the stock THERMAL run (open top, the reference's stop rule)
        {"name": "thermal_64x200", "kind": "thermal", "n": 64, "nz": 200, "crystal": "reference", "bc": 0,
         "rule": "reference"},
        # the THERMAL benchmark run: 256 x 256 x 400, oven-surrounded
        {"name": "thermal_256x400", "kind": "thermal", "n": 256, "nz": 400, "crystal": "qpm50", "bc": 1,
         "rule": "reference"},
        # heat sweeps alone, on a cross-section that is no power of two
        {"name": "heat_100x75", "kind": "heat", "n": 100, "nz": 75, "bc": 0, "sweeps": 64},
        # one step of the input-beam design loop: batched THERMAL gradient
        {"name": "thermal_gradient_16", "kind": "thermal_gradient", "count": 16, "n": 256, "nz": 100,
         "checkpoints": 20},
        # a batched THERMAL forward pass with the output fields, odd slice count
        {"name": "thermal_forward_64", "kind": "thermal_forward", "count": 64, "n": 64, "nz": 133},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "field", "sweep", "sweep", "gradient", "thermal", "heat", "thermal_gradient",
                       "thermal_forward"])
    c = {"kind": kind}
    if kind in ("solve", "field"):
        c.update(n=rng.choice([16, 32, 64, 128, 256]), nz=_log_int(rng, 24, 400),
                 crystal=rng.choice(["reference", "qpm50", "ppln"]))
    elif kind == "sweep":
        mixed = rng.random() < 0.5
        c.update(count=_log_int(rng, 2, 400), mixed=mixed, n=256 if mixed else rng.choice([32, 64, 128]),
                 nz=400 if mixed else _log_int(rng, 40, 300), crystal=rng.choice(["reference", "qpm50"]))
    elif kind == "gradient":
        nz = _log_int(rng, 30, 400)
        c.update(n=rng.choice([32, 64, 128, 256]), nz=nz, crystal=rng.choice(["reference", "qpm50", "ppln"]),
                 checkpoints=rng.choice([5, 20, nz]))
    elif kind == "thermal":
        c.update(n=rng.choice([32, 64, 128]), nz=_log_int(rng, 40, 200), crystal=rng.choice(["reference", "qpm50"]),
                 bc=rng.choice([0, 1]), rule=rng.choice(["reference", "relative"]))
    elif kind == "heat":
        c.update(n=rng.choice([rng.randrange(24, 257), 4 * rng.randrange(6, 65)]), nz=_log_int(rng, 12, 400),
                 bc=rng.choice([0, 1]), sweeps=_log_int(rng, 5, 200))
    elif kind == "thermal_gradient":
        nz = _log_int(rng, 24, 120)
        c.update(count=_log_int(rng, 2, 16), n=rng.choice([64, 128, 256]), nz=nz, checkpoints=rng.choice([10, 20, nz]))
    else:
        c.update(count=_log_int(rng, 2, 64), n=rng.choice([64, 128]), nz=_log_int(rng, 24, 200))
    return c


# ---------------------------------------------------------------------------------------
# Inputs: seeded values of the benchmark's distributions

def _f(x):
    return float(F(x))


def _beam(rng, crystal):
    """(power, waist, temperature) of one run: P log-U(1, 50) W, xi U(0.5, 5), T = 50 C + U(-2, 2) K."""
    p = _f(math.exp(rng.uniform(0.0, math.log(50.0))))
    t = _f(50.0 + rng.uniform(-2.0, 2.0))
    return p, W.waist_for_xi(rng.uniform(0.5, 5.0), t, crystal=CRYSTALS[crystal].crystal), t


def _instances(case, seed):
    rng = random.Random(1000 + seed)
    out, shape = [], random.Random(17 * case["count"] + case["nz"])  # the grids belong to the case, not to the seed
    for _ in range(case["count"]):
        p, w, t = _beam(rng, case["crystal"])
        n, nz = (shape.choice([64, 128, 256]), shape.choice([100, 200, 400])) if case["mixed"] else (case["n"], case["nz"])
        win = _f(16.0 * w)
        out.append(W.Instance(nx=n, ny=n, nz=nz, lx=win, ly=win, power=p, waist=w, temp=t))
    return out


def _field(n, lx, beam, seed, sh):
    """Input fields a program holds on the device: the focused beam with a smooth seeded
    perturbation, and a weak SH seed of a tenth of its amplitude."""
    p, w, t = beam
    g = torch.Generator().manual_seed(seed)
    dx = lx / (n - 1)
    x = ((torch.arange(n, dtype=torch.float64) - 0.5 * n) * dx)
    r2 = x[:, None] ** 2 + x[None, :] ** 2
    n_p = float(W.sellmeier_n(1.064, t))
    M = complex(1.0, -15000.0 / (math.pi * n_p * w * w / 1.064))
    a0 = math.sqrt(4 * p / (_EPS0 * _C * math.pi * n_p * w * w))
    k = torch.randn(4, generator=g, dtype=torch.float64) * 2 * math.pi / lx
    ripple = 1 + 0.05 * torch.cos(k[0] * x[None, :] + k[1] * x[:, None]) + 0.05j * torch.sin(k[2] * x[None, :] + k[3] * x[:, None])
    pump = (a0 / M) * torch.exp(-r2 / (w * w * M)) * ripple
    s = (0.1 * pump * torch.exp(1j * k[1] * x[None, :])) if sh else torch.zeros_like(pump)
    return pump.to(torch.complex64).to(DEV), s.to(torch.complex64).to(DEV)


def _thermal_args(case, seed):
    """Peltier and ambient temperatures, power and waist of a THERMAL run."""
    rng = random.Random(2000 + seed)
    t = _f(rng.uniform(45.0, 55.0))
    return {"power": _f(rng.uniform(20.0, 30.0)), "waist": W.waist_for_xi(2.84, 50.0), "temp": t}


def _temperature(n, nz, lx, ly, i, seed):
    """A heated crystal: oven temperature at the faces, a few tenths of a kelvin on the beam's axis."""
    rng = random.Random(3000 + 97 * seed + i)
    t0, dt = 50.0 + rng.uniform(-1, 1), rng.uniform(0.05, 0.4)
    x = np.linspace(-1, 1, n)
    cross = (1 - x[None, :] ** 2) * (1 - x[:, None] ** 2)
    z = np.linspace(0, 1, nz)
    return (t0 + dt * (0.5 + z)[:, None, None] * cross[None]).astype(np.float32)


def _thermal_batch(case, seed):
    rng = random.Random(4000 + seed)
    w = W.waist_for_xi(2.84, 50.0)
    win = _f(16.0 * w)
    return [(_f(rng.uniform(5.0, 40.0)), w, 15000.0) for _ in range(case["count"])], win


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case = case
    kind = case["kind"]
    if kind in ("solve", "field", "gradient"):
        rng = random.Random(seed)
        s.beam = _beam(rng, case["crystal"])
        s.win = _f(16.0 * s.beam[1])
        s.solver = Solver(crystal=CRYSTALS[case["crystal"]], nx=case["n"], ny=case["n"], nz=case["nz"], lx=s.win, ly=s.win)
        if kind == "field":
            s.pump, s.sh = _field(case["n"], s.win, s.beam, seed, True)
        if kind == "gradient":
            g = torch.Generator().manual_seed(seed)
            r = torch.randn(2, 1, generator=g, dtype=torch.float64).expand(2, case["n"]) * 0.02
            x = torch.linspace(0, 2 * math.pi, case["n"], dtype=torch.float64)
            s.factor = (1 + r[0] * torch.cos(x)[:, None] + 1j * r[1] * torch.sin(x)[None, :]).to(torch.complex64).to(DEV).contiguous()
    elif kind == "sweep":
        s.sweep = Sweep(_instances(case, seed), crystal=CRYSTALS[case["crystal"]])
        points = int(s.sweep.field_offsets()[-1])
        s.pinned = torch.empty(points, dtype=torch.complex64, pin_memory=True)
        s.eta = torch.empty(case["count"], dtype=torch.float64, pin_memory=True)
    elif kind == "thermal":
        s.args = _thermal_args(case, seed)
        s.solver = Solver(crystal=CRYSTALS[case["crystal"]], nx=case["n"], ny=case["n"], nz=case["nz"], thermal=True,
                          bc=case["bc"])
        if case["rule"] == "relative":
            s.solver.set_jacobi_rule(1e-6, 100, 400)
    elif kind == "heat":
        s.cfg, s.T0, s.qk = _heat_inputs(case, seed)
        s.a, s.b = torch.empty_like(s.T0), torch.empty_like(s.T0)
    else:
        solves, win = _thermal_batch(case, seed)
        s.batch = ThermalGradBatch(case["count"], crystal=W.CRYSTAL_QPM50, nx=case["n"], ny=case["n"], nz=case["nz"],
                                   lx=win, ly=win, bc=1)
        for i, (p, w, f) in enumerate(solves):
            s.batch.set_temperature(i, _temperature(case["n"], case["nz"], win, win, i, seed), p, w, f)
        s.pump = s.batch.gaussian_pumps()
    return s


def _heat_inputs(case, seed):
    n, nz = case["n"], case["nz"]
    cfg = _lib.default_config()
    cfg.nx, cfg.ny, cfg.nz = n, n, nz
    g = torch.Generator().manual_seed(seed)
    x = torch.linspace(-1, 1, n, dtype=torch.float64)
    beam = torch.exp(-40 * (x[:, None] ** 2 + x[None, :] ** 2))
    z = torch.linspace(0, 1, nz, dtype=torch.float64)
    T = 50 + 3 * torch.rand(1, generator=g, dtype=torch.float64) + (z[:, None, None] + 0.2) * beam + \
        0.01 * torch.rand(nz, n, n, generator=g, dtype=torch.float64)
    qk = (1e-6 * (1 + torch.rand(1, generator=g, dtype=torch.float64)) * (0.3 + z)[:, None, None] * beam)
    return cfg, T.to(torch.float32).to(DEV).contiguous(), qk.to(torch.float32).to(DEV).contiguous()


def run(s):
    case = s.case
    kind = case["kind"]
    if kind == "solve":
        p, w, t = s.beam
        s.solver.run(p, w, 15000.0, t)
        pump, sh = s.solver.fields()
        return {"pump": pump, "sh": sh, "efficiency": s.solver.efficiency()}
    if kind == "field":
        pump, sh = s.solver.cwes_device(s.beam[2], s.pump, s.sh)
        return {"pump": pump, "sh": sh}
    if kind == "sweep":
        s.sweep.run(eta_out=s.eta.numpy(), sh_out_all=s.pinned.numpy())
        # a ratio of sums of 32-bit fields: it is as accurate as they are
        return {"efficiency": s.eta.to(torch.float32), "sh": s.pinned}
    if kind == "gradient":
        p, w, t = s.beam
        r = s.solver.grad_run(p, w, 15000.0, t, pump_factor=s.factor, checkpoints=case["checkpoints"])
        return {"grad_pump": r["grad_pump"], **{k: float(r[k]) for k in ("loss", "dT", "dLambda", "dfocal", "dwaist", "dpower")}}
    if kind == "thermal":
        a = s.args
        s.solver.run(a["power"], a["waist"], 15000.0, a["temp"])
        pump, sh = s.solver.fields()
        return {"pump": pump, "sh": sh, "efficiency": s.solver.efficiency(), "temperature": s.solver.temperature(),
                "counts": np.array(s.solver.jacobi_counts(), np.int64)}
    if kind == "heat":
        s.a.copy_(s.T0)
        s.b.copy_(s.T0)
        _lib.check(_lib.lib().shg_heat_sweeps_device(ctypes.byref(s.cfg), s.a.data_ptr(), s.b.data_ptr(), s.qk.data_ptr(),
                                                     25.0, case["sweeps"], case["bc"],
                                                     torch.cuda.current_stream().cuda_stream), "shg_heat_sweeps_device")
        return s.b if case["sweeps"] % 2 else s.a
    if kind == "thermal_gradient":
        r = s.batch.gradient(s.pump, checkpoints=case["checkpoints"])
        return {"grad": r["grad"], "p_sh": r["p_sh"].astype(np.float32), "p_in": r["p_in"].astype(np.float32)}
    r = s.batch.forward(s.pump, with_fields=True)
    return {"pump": r["pump_out"], "sh": r["sh_out"], "p_sh": r["p_sh"].astype(np.float32)}


# ---------------------------------------------------------------------------------------
# The least a pass can do

def _march_flops(n, nz):
    # two fields' transform pairs and two RK4 calls per point and step
    return n * n * nz * (20.0 * math.log2(n * n) + 456.0)


def _sweep_count(case):
    # Jacobi sweeps the stop rule asks for at the least: one heating solve of 5001
    return {"relative": 100, "reference": 5003}[case["rule"]]


def work(case):
    kind, n, nz = case["kind"], case["n"], case["nz"]
    pts = n * n
    if kind == "solve":
        return {"bytes": 16.0 * pts, "flops": _march_flops(n, nz)}
    if kind == "field":
        return {"bytes": 32.0 * pts, "flops": _march_flops(n, nz)}
    if kind == "sweep":
        it = _instances(case, 0)
        return {"bytes": sum(8.0 * i.nx * i.ny for i in it), "flops": sum(_march_flops(i.nx, i.nz) for i in it)}
    if kind == "gradient":
        return {"bytes": 16.0 * pts, "flops": 2.5 * _march_flops(n, nz)}
    if kind == "thermal":
        vox = float(pts * nz)
        return {"bytes": 4.0 * vox + 16.0 * pts, "flops": 13.0 * vox * _sweep_count(case) + 2 * _march_flops(n, nz)}
    if kind == "heat":
        vox = float(pts * nz)
        return {"bytes": 12.0 * vox, "flops": 13.0 * vox * case["sweeps"]}
    b = float(case["count"] * pts)
    if kind == "thermal_gradient":
        return {"bytes": 16.0 * b + 16.0 * b * nz, "flops": 2.5 * case["count"] * _march_flops(n, nz)}
    return {"bytes": 24.0 * b + 16.0 * b * nz, "flops": case["count"] * _march_flops(n, nz)}


# ---------------------------------------------------------------------------------------
# The same outputs in 64 bits, from torch alone

_PI = F(3.14159265358979323846)
_C = float(F(299792458 * 1e6 / 1e12))
_EPS0 = float(F(8.8541878128e-12 * 1e12 / 1e6))
_LP, _LS = F(1.064), F(0.5 * float(F(1.064)))


def _index_terms(L, crystal):
    """The Sellmeier coefficients at wavelength L and the double evaluation n^2(T) and its derivative."""
    L2 = float(L) * float(L)
    if crystal == 1:
        def n2(T, lib):
            f = (T - 24.5) * (T + 570.82)
            c3 = 0.20692 + -0.89e-8 * f
            return (5.35583 + 4.629e-7 * f + (0.100473 + 3.862e-8 * f) / (L2 - c3 * c3)
                    + (100.0 + 2.657e-5 * f) / (L2 - 11.34927 * 11.34927) - 1.5334e-2 * L2)
        return n2
    A, B, C, D, E, G, H, J = (float(F(v)) for v in (4.502483, 0.007294, 0.185087, -0.02357, 0.073423, 0.199595, 0.001, 7.99724))

    def n2(T, lib):
        tk = T + 273.15
        tk2 = tk * tk
        if lib == "smooth":
            b, c = 3.483933e-8 * tk2, 1.607839e-8 * tk2
            Bb, Cc = B + b, C + c
        else:  # float coefficients, as the method rounds them
            b, c = _r32(3.483933e-8 * tk2), _r32(1.607839e-8 * tk2)
            Bb, Cc = _r32(B + b), _r32(C + c)
        return A + Bb / (L2 - Cc * Cc) + E / (L2 - G * G) + H / (L2 - J * J) + D * L2
    return n2


def _r32(v):
    return v.to(torch.float32).to(torch.float64) if isinstance(v, torch.Tensor) else float(F(v))


def _index(L, T, crystal):
    """n(L, T) rounded to float, of a number or a tensor of float temperatures."""
    v = _index_terms(L, crystal)(T.to(torch.float64) if isinstance(T, torch.Tensor) else float(F(T)), "float")
    return _r32(torch.sqrt(v)) if isinstance(v, torch.Tensor) else F(math.sqrt(v))


def _index_dT(L, T, crystal):
    n2 = _index_terms(L, crystal)
    t = torch.tensor(float(F(T)), dtype=torch.float64, requires_grad=True)
    return float(torch.autograd.grad(torch.sqrt(n2(t, "smooth")), t)[0])


class _Medium:
    """Scalars of one solve: float where the method defines them so, double products of them."""

    def __init__(self, crystal, n, nz, lx, ly, temp, tprop=None):
        cr = crystal
        tprop = temp if tprop is None else tprop
        self.n, self.nz, self.cr, self.temp = n, nz, cr, temp
        self.dx, self.dy, self.dz = F(lx) / F(n - 1), F(ly) / F(n - 1), F(cr.lz) / F(nz - 1)
        n_p, n_s = _index(_LP, temp, cr.crystal), _index(_LS, temp, cr.crystal)
        self.np_, self.ns_ = float(n_p), float(n_s)
        self.dk = float(F(2) * _PI * (F(2) * n_p / _LP - n_s / _LS + F(1) / F(cr.lambda_qpm)))
        z, zs = F(0), []
        for _ in range(nz):
            zs.append(z)
            z = z + self.dz
        self.z = zs
        self.dQ = 2.0 / math.pi * float(F(cr.deff))
        self.kp = math.pi * self.dQ / (self.np_ * float(_LP))
        self.ks = 0.5 * math.pi * self.dQ / (self.ns_ * float(_LS))
        self.hp, self.hs = 0.5 * float(F(cr.alpha_p)), 0.5 * float(F(cr.alpha_s))
        self.tpa = 0.25 * float(F(cr.beta_s)) * _C * _EPS0 * self.ns_
        self.npr, self.nsr = float(_index(_LP, tprop, cr.crystal)), float(_index(_LS, tprop, cr.crystal))

    def q2(self):
        n = self.n
        t = (torch.arange(n, device=DEV, dtype=torch.float64) + n // 2) % n - 0.5 * n
        return (t[None, :] / (float(self.dx) * n)) ** 2 + (t[:, None] / (float(self.dy) * n)) ** 2

    def propagators(self, np_=None, ns_=None):
        q2, dz = self.q2(), float(self.dz)
        kp = 2 * math.pi * (self.npr if np_ is None else np_) / float(_LP)
        ks = 2 * math.pi * (self.nsr if ns_ is None else ns_) / float(_LS)
        return torch.exp(-1j * dz * 2 * math.pi ** 2 / kp * q2), torch.exp(-1j * dz * 2 * math.pi ** 2 / ks * q2)

    def pump(self, power, waist, focal, n_p=None):
        n, w = self.n, waist
        n_p = self.npr if n_p is None else n_p
        x = (torch.arange(n, device=DEV, dtype=torch.float64) - 0.5 * n)
        r2 = (x[:, None] * float(self.dy)) ** 2 + (x[None, :] * float(self.dx)) ** 2
        M = 1 - 1j * (focal / (math.pi * n_p * w * w / float(_LP)))
        a0 = (4 * power / (_EPS0 * _C * math.pi * n_p * w * w)) ** 0.5
        return a0 / M * torch.exp(-r2 / (w * w * M))

    def power(self, a, index):
        return 0.5 * _EPS0 * _C * index * (a.real ** 2 + a.imag ** 2).sum(dim=(-2, -1)) * float(self.dx) * float(self.dy)


def _rk4(P, S, stages, hp, hs, tpa, dz):
    """One RK4 call: stage offsets 1/2, 1/2, 1 without dz, one pair of coupling factors per stage."""
    def f(P, S, c):
        return c[0] * S * P.conj() - hp * P, c[1] * P * P - (hs + tpa * (S.real ** 2 + S.imag ** 2)) * S
    k1 = f(P, S, stages[0])
    k2 = f(P + 0.5 * k1[0], S + 0.5 * k1[1], stages[1])
    k3 = f(P + 0.5 * k2[0], S + 0.5 * k2[1], stages[2])
    k4 = f(P + k3[0], S + k3[1], stages[3])
    w = dz / 6
    return P + w * (k1[0] + 2 * k2[0] + 2 * k3[0] + k4[0]), S + w * (k1[1] + 2 * k2[1] + 2 * k3[1] + k4[1])


def _diffract(A, H):
    return torch.fft.fft2(torch.fft.ifft2(A) * H)


def _march_plain(m, P, S, H):
    """The plain march of fields (..., n, n) with one medium or, batched, tensors of shape (b, 1, 1) in it."""
    dz = float(m.dz)
    for s in range(m.nz - 1):
        arg = m.arg(s) if hasattr(m, "arg") else float(F(m.z[s] * F(m.dk)))
        if isinstance(arg, torch.Tensor):
            e = torch.exp(-1j * arg)
            c = (1j * m.kp * e, 1j * m.ks * e.conj())
        else:
            e = complex(math.cos(arg), -math.sin(arg))
            c = (1j * m.kp * e, 1j * m.ks * e.conjugate())
        st = (c, c, c, c)
        P, S = _rk4(P, S, st, m.hp, m.hs, m.tpa, dz)
        P, S = _diffract(P, H[0]), _diffract(S, H[1])
        P, S = _rk4(P, S, st, m.hp, m.hs, m.tpa, dz)
    return P, S


class _Stack:
    """Several media of one grid and length as tensors over a leading axis."""

    def __init__(self, ms):
        def t(v):
            return torch.tensor([float(x) for x in v], dtype=torch.float64, device=DEV)[:, None, None]
        self.nz, self.dz = ms[0].nz, ms[0].dz
        for k in ("kp", "ks", "tpa"):
            setattr(self, k, t([getattr(m, k) for m in ms]))
        self.hp, self.hs = ms[0].hp, ms[0].hs
        self._args = [[float(F(z * F(m.dk))) for z in m.z] for m in ms]
        self._t = t

    def arg(self, s):
        return self._t([a[s] for a in self._args])


def _exact_sweep(case, seed):
    cr, it = CRYSTALS[case["crystal"]], _instances(case, seed)
    if sum(i.nx * i.ny * i.nz for i in it) > 6e8:
        return None
    groups = {}
    for k, i in enumerate(it):
        groups.setdefault((i.nx, i.nz), []).append(k)
    sh, eta = [None] * len(it), [0.0] * len(it)
    for (n, nz), ks in groups.items():
        ms = [_Medium(cr, n, nz, it[k].lx, it[k].ly, it[k].temp) for k in ks]
        P0 = torch.stack([m.pump(it[k].power, it[k].waist, it[k].focal) for m, k in zip(ms, ks)])
        H = [torch.stack(h) for h in zip(*(m.propagators() for m in ms))]
        P, S = _march_plain(_Stack(ms), P0, torch.zeros_like(P0), H)
        for j, k in enumerate(ks):
            sh[k] = S[j].reshape(-1).cpu()
            eta[k] = float(ms[j].power(S[j], ms[j].ns_) / ms[j].power(P0[j], ms[j].np_))
    return {"efficiency": torch.tensor(eta, dtype=torch.float64), "sh": torch.cat(sh)}


def _exact_gradient(case, seed):
    s_rng = random.Random(seed)
    p, w, t = _beam(s_rng, case["crystal"])
    cr, n, nz = CRYSTALS[case["crystal"]], case["n"], case["nz"]
    win = _f(16.0 * w)
    m = _Medium(cr, n, nz, win, win, t)
    g = torch.Generator().manual_seed(seed)
    r = torch.randn(2, 1, generator=g, dtype=torch.float64).expand(2, n) * 0.02
    x = torch.linspace(0, 2 * math.pi, n, dtype=torch.float64)
    factor = (1 + r[0] * torch.cos(x)[:, None] + 1j * r[1] * torch.sin(x)[None, :]).to(torch.complex64).to(DEV)
    v = {k: torch.tensor(float(x0), dtype=torch.float64, device=DEV, requires_grad=True)
         for k, x0 in (("dfocal", 15000.0), ("dwaist", w), ("dpower", p), ("dT", 0.0), ("dLambda", 0.0))}
    A = m.pump(v["dpower"], v["dwaist"], v["dfocal"]) * factor.to(torch.complex128)
    A0 = A.detach().clone().requires_grad_(True)
    dnp, dns = _index_dT(_LP, t, cr.crystal), _index_dT(_LS, t, cr.crystal)
    n_p, n_s = m.np_ + dnp * v["dT"], m.ns_ + dns * v["dT"]
    lam = float(F(cr.lambda_qpm))
    m.ddk = 2 * math.pi * (2 * dnp / float(_LP) - dns / float(_LS)) * v["dT"] - 2 * math.pi / lam ** 2 * v["dLambda"]
    m.kp, m.ks = math.pi * m.dQ / (n_p * float(_LP)), 0.5 * math.pi * m.dQ / (n_s * float(_LS))
    m.tpa = 0.25 * float(F(cr.beta_s)) * _C * _EPS0 * n_s
    dz = float(m.dz)

    def segment(P, S, kp, ks, tpa, ddk, np_, ns_, s0, s1):
        H = m.propagators(np_, ns_)
        for s in range(s0, s1):
            e = torch.exp(-1j * (float(F(m.z[s] * F(m.dk))) + float(m.z[s]) * ddk))
            st = ((1j * kp * e, 1j * ks * e.conj()),) * 4
            P, S = _rk4(P, S, st, m.hp, m.hs, tpa, dz)
            P, S = _diffract(P, H[0]), _diffract(S, H[1])
            P, S = _rk4(P, S, st, m.hp, m.hs, tpa, dz)
        return P, S

    P, S = A0, torch.zeros_like(A0)
    for s0 in range(0, nz - 1, 16):
        P, S = torch.utils.checkpoint.checkpoint(segment, P, S, m.kp, m.ks, m.tpa, m.ddk, n_p, n_s, s0,
                                                 min(nz - 1, s0 + 16), use_reentrant=False)
    loss = m.power(S, n_s)
    names = ["dT", "dLambda"]
    gA, *gs = torch.autograd.grad(loss, [A0] + [v[k] for k in names])
    out = {"grad_pump": gA, "loss": float(loss.detach()), "dT": float(gs[0]), "dLambda": float(gs[1])}
    rest = ["dfocal", "dwaist", "dpower"]
    for k, x in zip(rest, torch.autograd.grad(A, [v[k] for k in rest], grad_outputs=gA)):
        out[k] = float(x)
    return out


class _Heat:
    """Jacobi sweeps of the steady heat equation in double (both boundary modes)."""

    def __init__(self, cr, n, nz, lx, ly, t_inf, bc):
        dx, dy, dz = F(lx) / F(n - 1), F(ly) / F(n - 1), F(cr.lz) / F(nz - 1)
        dx, dy, dz, k, h = float(dx), float(dy), float(dz), float(F(cr.kth)), float(F(cr.htc))
        self.bc, self.ti = bc, t_inf
        self.inv = (1 / dx ** 2, 1 / dy ** 2, 1 / dz ** 2)
        self.L2 = 1 / (2 / dx ** 2 + 2 / dy ** 2 + 2 / dz ** 2)
        self.Bi = Bix, Biy, Biz = h * dx / k, h * dy / k, h * dz / k
        self.face = {"x": (dx * dx / (2 * dy * dy), dx * dx / (2 * dz * dz), Bix),
                     "y": (dy * dy / (2 * dx * dx), dy * dy / (2 * dz * dz), Biy),
                     "z": (dz * dz / (2 * dx * dx), dz * dz / (2 * dy * dy), Biz)}
        self.v = (dz / (2 * dx), dx / (2 * dz), dx * dz / (4 * dy * dy), 0.5 * (Bix + Biz))
        self.hh = (dz / (2 * dy), dy / (2 * dz), dy * dz / (4 * dx * dx), 0.5 * (Biy + Biz))
        self.d = (dx / (2 * dy), dy / (2 * dx), dx * dy / (4 * dz * dz), 0.5 * (Bix + Biy))
        self.c = (dy * dz / dx, dx * dz / dy, dx * dy / dz, Bix * dy + Biy * dz + Biz * dx)

    def sweep(self, T, N, qk):
        """N <- one sweep of T (arrays [z, y, x]); what the method never writes is left alone in N."""
        I, ti = slice(1, -1), self.ti
        i = self.inv
        N[I, I, I] = self.L2 * ((T[I, I, 2:] + T[I, I, :-2]) * i[0] + (T[I, 2:, I] + T[I, :-2, I]) * i[1]
                                + (T[2:, I, I] + T[:-2, I, I]) * i[2] + qk[I, I, I])
        a, b, Bi = self.face["z"]
        for z, zn in ((0, 1), (-1, -2)):
            N[z, I, I] = (T[zn, I, I] + a * (T[z, I, 2:] + T[z, I, :-2]) + b * (T[z, 2:, I] + T[z, :-2, I]) + Bi * ti) / (1 + 2 * a + 2 * b + Bi)
        if self.bc:
            return
        a, b, Bi = self.face["x"]
        for x, xn in ((0, 1), (-1, -2)):
            N[I, I, x] = (T[I, I, xn] + a * (T[I, 2:, x] + T[I, :-2, x]) + b * (T[2:, I, x] + T[:-2, I, x]) + Bi * ti) / (1 + 2 * a + 2 * b + Bi)
        a, b, Bi = self.face["y"]
        N[I, -1, I] = (T[I, -2, I] + a * (T[I, -1, 2:] + T[I, -1, :-2]) + b * (T[2:, -1, I] + T[:-2, -1, I]) + Bi * ti) / (1 + 2 * a + 2 * b + Bi)
        a, b, c, B = self.v
        V = 1 / (a + b + 2 * c + B)
        for x, xn in ((0, 1), (-1, -2)):
            for z, zn in ((0, 1), (-1, -2)):
                N[z, I, x] = (a * T[z, I, xn] + b * T[zn, I, x] + c * (T[z, 2:, x] + T[z, :-2, x]) + B * ti) * V
        a, b, c, B = self.hh
        V = 1 / (a + b + 2 * c + B)
        for z, zn in ((0, 1), (-1, -2)):
            N[z, -1, I] = (a * T[z, -2, I] + b * T[zn, -1, I] + c * (T[z, -1, 2:] + T[z, -1, :-2]) + B * ti) * V
        a, b, c, B = self.d
        V = 1 / (a + b + 2 * c + B)
        for x, xn in ((0, 1), (-1, -2)):
            N[I, -1, x] = (a * T[I, -2, x] + b * T[I, -1, xn] + c * (T[2:, -1, x] + T[:-2, -1, x]) + B * ti) * V
        a, b, c, B = self.c
        for x, xn in ((0, 1), (-1, -2)):
            for z, zn in ((0, 1), (-1, -2)):
                N[z, -1, x] = (a * T[z, -1, xn] + b * T[z, -2, x] + c * T[zn, -1, x] + ti * B) / (a + b + c + B)

    def run(self, T, qk, count):
        """T after `count` sweeps and the state before the last one."""
        A, B = T.clone(), T.clone()
        if count > 40:  # two sweeps as one graph, replayed
            side = torch.cuda.Stream()
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):
                self.sweep(A, B, qk)
                self.sweep(B, A, qk)
            torch.cuda.current_stream().wait_stream(side)
            count -= 2
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g):
                self.sweep(A, B, qk)
                self.sweep(B, A, qk)
            for _ in range(count // 2 - 1):
                g.replay()
            count -= 2 * (count // 2 - 1)
        for _ in range(count):
            self.sweep(A, B, qk)
            A, B = B, A
        return A, B


def _thermal_tables(cr, T, lx, ly):
    """Per-voxel coupling (kp, ks, TPA factor) and the float phase mismatch of a temperature field."""
    n_p, n_s = _index(_LP, T, cr.crystal), _index(_LS, T, cr.crystal)
    f = [v.to(torch.float32) for v in (n_p, n_s)]
    two_pi = float(F(2) * _PI)
    lp, ls = (torch.tensor(float(v), dtype=torch.float32, device=T.device) for v in (_LP, _LS))  # IEEE float division
    dk = (two_pi * ((2.0 * f[0] / lp - f[1] / ls) + float(F(1) / F(cr.lambda_qpm)))).to(torch.float64)
    dQ = 2.0 / math.pi * float(F(cr.deff))
    return n_p, n_s, dk, math.pi * dQ / (n_p * float(_LP)), 0.5 * math.pi * dQ / (n_s * float(_LS))


def _march_thermal(m, P, S, H, tabs, steps, heat=None):
    """The THERMAL march of `steps` steps; tabs = per-slice (kp, ks, tpa, running dk sum) by index.
    Returns the state after nz-1 steps; `heat(s, P, S)` sees the state after each step."""
    dz, out = float(m.dz), None
    for s in range(steps):
        kp, ks, tpa, dki = tabs(s)
        st = []
        for inc in (0.0, 0.25, 0.25, 0.5):
            e = torch.exp(-1j * (dki * ((s + 1 + inc) * dz) / (s + 1)))
            st.append((1j * kp * e, 1j * ks * e.conj()))
        P, S = _rk4(P, S, st, m.hp, m.hs, tpa, dz)
        P, S = _diffract(P, H[0]), _diffract(S, H[1])
        P, S = _rk4(P, S, st, m.hp, m.hs, tpa, dz)
        if heat is not None:
            heat(s, P, S)
        if s == m.nz - 2:
            out = (P, S)
    return out


def _exact_thermal(case, seed):
    n, nz, bc = case["n"], case["nz"], case["bc"]
    if n * n * nz > (3.5e6 if case["rule"] == "relative" else 9e5):
        return None
    cr, a = CRYSTALS[case["crystal"]], _thermal_args(case, seed)
    lx, ly, t = cr.lx, cr.ly, a["temp"]
    h = _Heat(cr, n, nz, lx, ly, 25.0, bc)
    T = torch.full((nz, n, n), t, dtype=torch.float64, device=DEV)  # Peltiers and oven at the run temperature
    qk = torch.zeros_like(T)
    qc, kth = 0.5 * _C * _EPS0, float(F(cr.kth))
    ap, as_, bs = (float(F(v)) for v in (cr.alpha_p, cr.alpha_s, cr.beta_s))
    tol, k, it = 5e-4 / T.numel(), 0, 5
    while k < it:
        count, last, res = 0, -1.0, 1.0
        if case["rule"] == "relative":
            while True:
                T, prev = h.run(T, qk, 100)
                count += 100
                if float((T - prev).norm() / T.norm()) < 1e-6 or count >= 400:
                    break
        else:
            T, prev = h.run(T, qk, 1)
            count, res = 1, float(((T - prev) ** 2).sum()) / T.numel()
            while res >= tol and res != last:
                T, prev = h.run(T, qk, 5000)
                count, last, res = count + 5000, res, float(((T - prev) ** 2).sum()) / T.numel()
        T32 = T.to(torch.float32)
        n_p, n_s, dk, kp, ks = _thermal_tables(cr, T32, lx, ly)
        tc = float(T32[0, n // 2, n // 2])
        m = _Medium(cr, n, nz, lx, ly, tc)
        run_dk = torch.cumsum(dk, 0)
        tpa_c = 0.25 * bs * _EPS0 * _C
        P0 = m.pump(a["power"], a["waist"], 15000.0)

        def heat(s, P, S):
            Ip, Is = qc * n_p[s] * (P.real ** 2 + P.imag ** 2), qc * n_s[s] * (S.real ** 2 + S.imag ** 2)
            qk[s] = (ap * Ip + as_ * Is + bs * Is * Is) / kth

        P, S = _march_thermal(m, P0, torch.zeros_like(P0), m.propagators(),
                              lambda s: (kp[s], ks[s], tpa_c * n_s[s], run_dk[s]), nz, heat)
        if count == 1 and k != 0:
            k = it
        k += 1
    eta = float(m.power(S, m.ns_) / m.power(P0, m.np_))
    return {"pump": P, "sh": S, "efficiency": eta, "temperature": T, "counts": None}


def _exact_thermal_batch(case, seed):
    n, nz, cr = case["n"], case["nz"], W.CRYSTAL_QPM50
    solves, win = _thermal_batch(case, seed)
    grad = case["kind"] == "thermal_gradient"
    if case["count"] * n * n * nz > (1.2e8 if grad else 4e8):
        return None
    T = torch.stack([torch.from_numpy(_temperature(n, nz, win, win, i, seed)) for i in range(case["count"])]).to(DEV)
    ms = [_Medium(cr, n, nz, win, win, float(T[i, 0, n // 2, n // 2])) for i in range(case["count"])]
    A = torch.stack([m.pump(*s) for m, s in zip(ms, solves)]).to(torch.complex64)  # the batch's own pumps are 32-bit
    A = A.to(torch.complex128)
    H = [torch.stack(x) for x in zip(*(m.propagators() for m in ms))]
    n_p, n_s, dk, kp, ks = _thermal_tables(cr, T.transpose(0, 1), win, win)
    run_dk = torch.cumsum(dk, 0)
    tpa_c = 0.25 * float(F(cr.beta_s)) * _EPS0 * _C
    m = ms[0]
    tabs = lambda s: (kp[s], ks[s], tpa_c * n_s[s], run_dk[s])  # noqa: E731
    ns = torch.tensor([x.ns_ for x in ms], dtype=torch.float64, device=DEV)
    npv = torch.tensor([x.np_ for x in ms], dtype=torch.float64, device=DEV)
    if not grad:
        P, S = _march_thermal(m, A, torch.zeros_like(A), H, tabs, nz - 1)
        return {"pump": P, "sh": S, "p_sh": m.power(S, ns)}
    A.requires_grad_(True)

    def segment(P, S, s0, s1):
        dz = float(m.dz)
        for s in range(s0, s1):
            kp_, ks_, tpa, dki = tabs(s)
            st = []
            for inc in (0.0, 0.25, 0.25, 0.5):
                e = torch.exp(-1j * (dki * ((s + 1 + inc) * dz) / (s + 1)))
                st.append((1j * kp_ * e, 1j * ks_ * e.conj()))
            P, S = _rk4(P, S, st, m.hp, m.hs, tpa, dz)
            P, S = _diffract(P, H[0]), _diffract(S, H[1])
            P, S = _rk4(P, S, st, m.hp, m.hs, tpa, dz)
        return P, S

    P, S = A, torch.zeros_like(A)
    for s0 in range(0, nz - 1, 4):
        P, S = torch.utils.checkpoint.checkpoint(segment, P, S, s0, min(nz - 1, s0 + 4), use_reentrant=False)
    p = m.power(S, ns)
    (g,) = torch.autograd.grad(p.sum(), A)
    return {"grad": g, "p_sh": p.detach(), "p_in": m.power(A.detach(), npv)}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("solve", "field"):
        p, w, t = _beam(random.Random(seed), case["crystal"])
        win = _f(16.0 * w)
        m = _Medium(CRYSTALS[case["crystal"]], case["n"], case["nz"], win, win, t)
        if kind == "field":
            P0, S0 = (v.to(torch.complex128) for v in _field(case["n"], win, (p, w, t), seed, True))
            P, S = _march_plain(m, P0, S0, m.propagators())
            return {"pump": P, "sh": S}
        P0 = m.pump(p, w, 15000.0)
        P, S = _march_plain(m, P0, torch.zeros_like(P0), m.propagators())
        return {"pump": P, "sh": S, "efficiency": float(m.power(S, m.ns_) / m.power(P0, m.np_))}
    if kind == "sweep":
        return _exact_sweep(case, seed)
    if kind == "gradient":
        return _exact_gradient(case, seed)
    if kind == "thermal":
        return _exact_thermal(case, seed)
    if kind == "heat":
        cfg, T0, qk = _heat_inputs(case, seed)
        cr = W.CRYSTAL_REFERENCE
        return _Heat(cr, case["n"], case["nz"], cr.lx, cr.ly, 25.0, case["bc"]).run(T0.double(), qk.double(), case["sweeps"])[0]
    return _exact_thermal_batch(case, seed)
