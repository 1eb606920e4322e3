"""The work that users have this framework do, as measurable cases.

``listed()`` names the cases, ``draw(rng)`` gives more of the same ranges, ``prepare`` makes what a
program has in hand before the call (solver, network, loaded state), ``run`` is one pass through
the public entry points, ``work`` the bytes and flops the pass cannot do without, and ``exact``
the same pass in 64-bit torch arithmetic.

Kinds of case:

* ``flow``: one run of a single flow (2D vorticity or 3D velocity), advanced by a few steps and
  read back.  ``drive`` says how the program steps it: ``fixed`` (``advance`` with one dt),
  ``cfl`` (``simulate.run_steps``: CFL dt from the host every ten steps) or ``device``
  (``run_to``: CFL and constant-power forcing evaluated on the device).
* ``ensemble``: many independent 2D runs of uneven sizes advanced together.
* ``les``: a coarse 2D run with the learned closure in its nonlinear term.
* ``train``: optimiser steps of the closure network on a bank of snapshots.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from pyspectral_b200 import Config, registry, simulate
from pyspectral_b200.closure import ClosureNet, ClosureSolver
from pyspectral_b200.ensemble import Ensemble

FUSED, GENERAL = "b200/fused-fft-graph", "b200/fused-inplace-graph"
POWER, KLO, KHI, ALPHA, ALPHA_KMAX = 1e-3, 10.0, 12.0, 0.1, 2.0  # constant-power band forcing
CFL, DT_MAX, CFL_EVERY = 0.5, 0.05, 10


def _flow(name, n, dim, dtype, form, drive, steps, variant=FUSED, forced=False, records=False):
    return {"name": name, "kind": "flow", "n": n, "dim": dim, "dtype": dtype, "form": form,
            "drive": drive, "steps": steps, "variant": variant, "forced": forced,
            "records": records}


def listed():
    return [
        # convergence and regression studies: small double-precision grids, launches count
        _flow("conv2d-64-fp64", 64, 2, "float64", "basdevant", "fixed", 10),
        # the plain 2D validation workload (256^2, fp64, dt = 1e-3)
        _flow("vortex2d-256-fp64", 256, 2, "float64", "basdevant", "fixed", 10),
        # forced turbulence with drag at a spin-up size, loop control on the device
        _flow("forced2d-512-fp32", 512, 2, "float32", "basdevant", "device", 50, forced=True),
        # the fine DNS that feeds and judges the closure
        _flow("dns2d-2048-fp32", 2048, 2, "float32", "basdevant", "device", 20, forced=True),
        # the headline 2D decaying-turbulence run
        _flow("decay2d-8192-fp32", 8192, 2, "float32", "basdevant", "cfl", 10),
        # a grid that is no power of two, on the general engine, with its records
        _flow("ragged2d-1536-fp32", 1536, 2, "float32", "basdevant", "cfl", 10, GENERAL,
              records=True),
        # the Re = 1600 validation grid in double precision
        _flow("box3d-128-fp64-rot", 128, 3, "float64", "rotational", "cfl", 5),
        # an ordinary 3D run in the rotational form
        _flow("box3d-256-fp32-rot", 256, 3, "float32", "rotational", "cfl", 5),
        # the headline 3D run
        _flow("box3d-512-fp32-bas", 512, 3, "float32", "basdevant", "cfl", 2),
        # the data engine: 256 forced runs of four sizes
        {"name": "ensemble-4x64-fp32", "kind": "ensemble", "dtype": "float32", "n128": 64,
         "n256": 64, "n512": 64, "n1024": 64, "steps": 5},
        # the coarse run that the closure makes possible, network held over a step's stages
        {"name": "les-256", "kind": "les", "n": 256, "steps": 50, "every_stage": False},
        # closure training at the study's batch (65536 points)
        {"name": "train-256x512", "kind": "train", "n": 256, "entries": 64, "tiles": 512,
         "steps": 50},
    ]


def draw(rng):
    kind = rng.choice(["flow2", "flow2", "flow2", "flow3", "flow3", "general", "ensemble", "les",
                       "train"])
    if kind == "flow2":
        dtype = rng.choice(["float32", "float64"])
        n = 2 ** rng.randint(5, 13 if dtype == "float32" else 12)
        drive = rng.choice(["fixed", "cfl", "device"])
        forced = n >= 64 and rng.random() < 0.5
        steps = rng.randint(1, 10) if n >= 4096 else rng.randint(2, 40)
        return {"kind": "flow", "n": n, "dim": 2, "dtype": dtype, "form": "basdevant",
                "drive": drive, "steps": steps, "variant": FUSED, "forced": forced,
                "records": rng.random() < 0.25}
    if kind == "flow3":
        dtype = rng.choice(["float32", "float64"])
        n = 2 ** rng.randint(4, 9 if dtype == "float32" else 8)
        steps = 1 if n >= 512 else rng.randint(1, 2) if n >= 256 else rng.randint(2, 12)
        return {"kind": "flow", "n": n, "dim": 3, "dtype": dtype,
                "form": rng.choice(["basdevant", "rotational"]),
                "drive": rng.choice(["fixed", "cfl", "device"]), "steps": steps, "variant": FUSED,
                "forced": False, "records": rng.random() < 0.25}
    if kind == "general":
        dim = rng.choice([2, 2, 3])
        lo, hi = (48, 3072) if dim == 2 else (24, 288)
        n = 2 * int(round(math.exp(rng.uniform(math.log(lo / 2), math.log(hi / 2)))))
        return {"kind": "flow", "n": n, "dim": dim, "dtype": rng.choice(["float32", "float64"]),
                "form": "basdevant" if dim == 2 else rng.choice(["basdevant", "rotational"]),
                "drive": rng.choice(["fixed", "cfl", "device"]),
                "steps": rng.randint(1, 4) if dim == 3 else rng.randint(1, 10),
                "variant": GENERAL, "forced": dim == 2 and n >= 64 and rng.random() < 0.5,
                "records": rng.random() < 0.25}
    if kind == "ensemble":
        c = {"kind": "ensemble", "dtype": rng.choice(["float32", "float32", "float64"])}
        top = 64 if c["dtype"] == "float32" else 24
        for n in (128, 256, 512, 1024):
            c[f"n{n}"] = int(round(math.exp(rng.uniform(0.0, math.log(top)))))
        return {**c, "steps": rng.randint(1, 5)}
    if kind == "les":
        return {"kind": "les", "n": rng.choice([128, 256, 512]), "steps": rng.randint(10, 60),
                "every_stage": rng.random() < 0.3}
    return {"kind": "train", "n": rng.choice([128, 256, 512]), "entries": rng.randint(4, 48),
            "tiles": rng.randint(64, 1024), "steps": rng.randint(5, 60)}


# ---------------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFF)


def _wave(n, dim):
    """Broadcastable float64 wavenumbers of the r2c grid, on the GPU."""
    full = torch.cat([torch.arange(0, n // 2), torch.arange(-(n // 2), 0)]).double().cuda()
    half = torch.arange(n // 2 + 1, device="cuda").double()
    axes = [full] * (dim - 1) + [half]
    return [a.reshape([-1 if i == d else 1 for i in range(dim)]) for d, a in enumerate(axes)]


def _mask(n, dim):
    m = None
    for k in _wave(n, dim):
        keep = 3.0 * k.abs() < n
        m = keep if m is None else m & keep
    return m


def _vorticity(n, k0, energy, gen, batch=()):
    """Random-phase spectral vorticity, E(k) ~ k^4 exp(-2 (k/k0)^2), dealiased, complex128."""
    kx, ky = _wave(n, 2)
    k2 = kx * kx + ky * ky
    kk = k2.sqrt()
    amp = kk**2.5 * torch.exp(-((kk / k0) ** 2)) * _mask(n, 2)
    phase = torch.rand((*batch, n, n // 2 + 1), generator=gen, device="cuda",
                       dtype=torch.float64) * (2.0 * math.pi)
    spec = torch.polar(amp.expand_as(phase).contiguous(), phase)
    half = n // 2  # the ky = 0 column of a real field is Hermitian
    spec[..., n - half + 1:, 0] = spec[..., 1:half, 0].flip(-1).conj()
    spec[..., 0, 0] = 0.0
    spec[..., half, 0] = 0.0
    w = torch.full((n // 2 + 1,), 2.0, device="cuda", dtype=torch.float64)
    w[0] = w[-1] = 1.0
    dens = torch.where(k2 > 0, w / torch.where(k2 > 0, k2, 1.0), 0.0)
    e = 0.5 * (spec.abs().square() * dens).sum(dim=(-2, -1), keepdim=True) / float(n) ** 4
    return spec * (energy / e).sqrt()


def _velocity(n, gen):
    """The Taylor-Green velocity with a random solenoidal perturbation of 2 % of its energy."""
    ks = _wave(n, 3)
    k2 = sum(k * k for k in ks)
    kk = k2.sqrt()
    shape = torch.where(kk > 0, kk * torch.exp(-((kk / 4.0) ** 2)), 0.0) * _mask(n, 3)
    out = []
    for _ in range(3):
        noise = torch.randn((n, n, n), generator=gen, device="cuda", dtype=torch.float64)
        out.append(torch.fft.rfftn(noise) * shape)
        del noise
    div = sum(k * c for k, c in zip(ks, out)) / torch.where(k2 > 0, k2, 1.0)
    out = torch.stack([c - k * div for c, k in zip(out, ks)])
    w = torch.full((n // 2 + 1,), 2.0, device="cuda", dtype=torch.float64)
    w[0] = w[-1] = 1.0
    e = 0.5 * sum(float((c.abs().square() * w).sum()) for c in out) / float(n) ** 6
    out *= math.sqrt(0.02 * 0.125 / e)
    a = float(n) ** 3 / 8.0  # sin x cos y cos z and -cos x sin y cos z on the modes (+-1, +-1, 1)
    for sx in (1, -1):
        for sy in (1, -1):
            out[0, sx, sy, 1] += -1j * sx * a
            out[1, sx, sy, 1] += 1j * sy * a
    return out


def _nu(case):
    n = case["n"]
    if case["dim"] == 3:
        return (512.0 / n) ** (4.0 / 3.0) / 1600.0
    if case["forced"]:
        return _nu_forced(n)
    return 2e-6 * (8192.0 / n) ** 2


def _nu_forced(n):
    """k_max eta = 1 for the band forcing's enstrophy injection."""
    kf = 0.5 * (KLO + KHI)
    return (kf * kf * POWER) ** (1.0 / 3.0) * (3.0 / n) ** 2


def _config(case):
    forcing = dict(alpha=ALPHA, alpha_kmax=ALPHA_KMAX, force_klo=KLO, force_khi=KHI)
    return Config(n=case["n"], dim=case["dim"], nu=_nu(case), dtype=case["dtype"],
                  form=case["form"], **(forcing if case["forced"] else {}))


def _dt(case):
    return 1e-3 if case["dim"] == 2 and case["n"] <= 256 else 0.5 / case["n"]


def _flow_state(case, seed):
    g = _gen(seed)
    if case["dim"] == 3:
        return _velocity(case["n"], g)
    return _vorticity(case["n"], min(12.0, case["n"] / 10.0), 0.05 if case["forced"] else 0.5, g)


def _members(case):
    return [n for n in (128, 256, 512, 1024) for _ in range(case[f"n{n}"])]


def _ensemble_states(case, seed):
    g = _gen(seed)
    return {n: _vorticity(n, 8.0, 0.05, g, (case[f"n{n}"],))
            for n in (128, 256, 512, 1024) if case[f"n{n}"]}


def _fields(n, count, gen):
    """(count, 4, n, n) snapshots: vorticity, its gradient and a term made from them."""
    w = _vorticity(n, 12.0, 5e-3, gen, (count,))
    kx, ky = _wave(n, 2)
    om, ox, oy = (torch.fft.irfft2(w * f, s=(n, n)) for f in (1.0, 1j * kx, 1j * ky))
    k2 = (kx * kx + ky * ky) / (n / 6.0) ** 2
    s = torch.fft.irfft2(-w * k2, s=(n, n)) + 0.2 * om * ox / om.std() + 0.1 * oy
    return torch.stack([om, ox, oy, s], dim=1).float()


def _params(seed):
    """Network parameters as a trained network has them: LeCun-sized weights, small biases."""
    rng = np.random.default_rng(seed)
    p = np.zeros(15440, np.float32)
    for layer, fan in enumerate((75, 64, 64)):
        w = np.zeros((64, 80), np.float32)
        w[:, :fan] = rng.normal(0.0, 1.0 / math.sqrt(fan), (64, fan))
        w[:, 75 if layer == 0 else 64] = rng.normal(0.0, 0.05, 64)
        p[layer * 5120: (layer + 1) * 5120] = w.ravel()
    p[15360: 15424] = rng.normal(0.0, 0.1 / 8.0, 64)
    return p


# the scales of the closure's inputs and output: vorticity of order one at k ~ 8
LES_INSCALE, LES_OUTSCALE = (1.0, 0.12, 0.12), 0.05
LES_NU = 5e-6


def _les_state(case, seed):
    return _vorticity(case["n"], 8.0, 5e-3, _gen(seed))


def prepare(case, seed):
    if case["kind"] == "flow":
        solver = registry.get(case["variant"]).make(_config(case))
        solver.set_state(_flow_state(case, seed))
        return {"case": case, "solver": solver}
    if case["kind"] == "ensemble":
        cfgs = [Config(n=n, dim=2, nu=_nu_forced(n), alpha=ALPHA, alpha_kmax=ALPHA_KMAX,
                       force_klo=KLO, force_khi=KHI, dtype=case["dtype"]) for n in _members(case)]
        ens = Ensemble(cfgs)
        states = _ensemble_states(case, seed)
        ens.set_states([a for n in sorted(states) for a in states[n].cpu().numpy()])
        return {"case": case, "ens": ens}
    if case["kind"] == "les":
        net = ClosureNet(n=case["n"], capacity=1)
        net.set_params(_params(seed))
        net.set_scales(LES_INSCALE, LES_OUTSCALE)
        cfg = Config(n=case["n"], dim=2, nu=LES_NU, alpha=ALPHA, alpha_kmax=ALPHA_KMAX,
                     force_klo=KLO, force_khi=KHI)
        solver = ClosureSolver(cfg, net, every_stage=case["every_stage"])
        solver.set_state(_les_state(case, seed))
        return {"case": case, "solver": solver, "net": net}
    bank = _fields(case["n"], case["entries"], _gen(seed))
    std = bank.double().square().mean(dim=(0, 2, 3)).sqrt().cpu().numpy()
    net = ClosureNet(n=case["n"], capacity=case["entries"])
    net.load_bank(bank.cpu().numpy())
    net.set_params(_params(seed))
    net.set_scales(1.0 / std[:3], float(std[3]))
    net.set_adam(lr=1e-3, total_steps=20000, warmup=200)
    return {"case": case, "net": net, "seed": int(seed) % 1000}


# ---------------------------------------------------------------------- one pass
def run(state):
    case = state["case"]
    if case["kind"] == "flow":
        s = state["solver"]
        if case["drive"] == "fixed":
            s.advance(case["steps"], _dt(case))
        elif case["drive"] == "cfl":
            simulate.run_steps(s, case["steps"], cfl=CFL, dt_max=DT_MAX, cfl_every=CFL_EVERY,
                               target_power=POWER if case["forced"] else None)
        else:
            s.run_to(s.t + 1e3, cfl=CFL, dt_max=DT_MAX, cfl_every=min(CFL_EVERY, case["steps"]),
                     target_power=POWER if case["forced"] else None, max_steps=case["steps"])
        out = {"state": s.state_native(), "t": s.t}
        if case["records"]:
            st = s.state_native()
            sums = s.diag.all(st)
            out["sums"] = np.array([sums["energy"], sums["enstrophy"]])
            out["spectrum"] = s.diag.spectrum(st)[1]
        return out
    if case["kind"] == "ensemble":
        ens = state["ens"]
        ens.run_steps(case["steps"], cfl=CFL, dt_max=DT_MAX, cfl_every=CFL_EVERY,
                      target_power=POWER)
        out = {"t": ens.t.copy()}
        for ci, c in enumerate(ens.classes):  # reading one member refreshes its class
            ens.state_native(ens.index[ci][0])
            out[f"n{c.n:04d}"] = c.u0
        return out
    if case["kind"] == "les":
        s = state["solver"]
        s.run_to(s.t + 1e3, cfl=CFL, dt_max=DT_MAX, cfl_every=CFL_EVERY, target_power=POWER,
                 max_steps=case["steps"])
        return {"state": s.state_native(), "t": s.t}
    net = state["net"]
    losses = net.train(case["steps"], batch_tiles=case["tiles"], seed=state["seed"])
    return {"losses": losses, "params": net.params()}


# ---------------------------------------------------------------------- what a pass needs
def _chunked(steps):
    return -(-steps // CFL_EVERY) * CFL_EVERY  # run_to takes whole chunks of steps


def _steps(case):
    """Steps that a pass takes."""
    if case.get("drive") == "device":
        every = min(CFL_EVERY, case["steps"])
        return -(-case["steps"] // every) * every
    return _chunked(case["steps"]) if case["kind"] == "les" else case["steps"]


def _step_flops(n, dim, form):
    ffts = {(2, "basdevant"): 4, (3, "basdevant"): 8, (3, "rotational"): 9}[(dim, form)]
    pts = float(n) ** dim
    return 4 * (ffts * 2.5 * pts * math.log2(pts) + 30 * pts)


def work(case):
    if case["kind"] == "flow":
        real = 4 if case["dtype"] == "float32" else 8
        n, dim = case["n"], case["dim"]
        state = (1 if dim == 2 else 3) * float(n) ** (dim - 1) * (n // 2 + 1) * 2 * real
        return {"bytes": 2 * state, "flops": _steps(case) * _step_flops(n, dim, case["form"])}
    if case["kind"] == "ensemble":
        real = 4 if case["dtype"] == "float32" else 8
        return {"bytes": sum(4.0 * real * n * (n // 2 + 1) for n in _members(case)),
                "flops": case["steps"] * sum(_step_flops(n, 2, "basdevant")
                                             for n in _members(case))}
    net = 2.0 * (75 * 64 + 64 * 64 + 64 * 64 + 64)
    if case["kind"] == "les":
        n = case["n"]
        per = (4 if case["every_stage"] else 1) * net * n * n
        return {"bytes": 16.0 * n * (n // 2 + 1),
                "flops": _steps(case) * (per + _step_flops(n, 2, "basdevant"))}
    points = case["tiles"] * 128.0
    return {"bytes": case["steps"] * points * 16.0, "flops": case["steps"] * points * 68.6e3}


# ---------------------------------------------------------------------- the same in 64 bits
class _Exact2D:
    """Lawson IF-RK4 of the 2D vorticity equation in complex128; leading axes are members."""

    def __init__(self, w, nu, forced, extra=None, every_stage=False):
        self.w, self.n = w, w.shape[-2]
        self.nu, self.forced, self.extra, self.every = nu, forced, extra, every_stage
        self.kx, self.ky = _wave(self.n, 2)
        self.k2 = self.kx * self.kx + self.ky * self.ky
        self.mask = _mask(self.n, 2)
        self.ik2 = torch.where(self.k2 > 0, 1.0 / torch.where(self.k2 > 0, self.k2, 1.0), 0.0)
        self.w = self.w * self.mask
        self.amp = torch.zeros(w.shape[:-2], device="cuda", dtype=torch.float64)
        wt = torch.full((self.n // 2 + 1,), 2.0, device="cuda", dtype=torch.float64)
        wt[0] = wt[-1] = 1.0
        self.wt = wt / float(self.n) ** 4
        self.t = torch.zeros(w.shape[:-2], device="cuda", dtype=torch.float64)

    def phys(self, spec):
        return torch.fft.irfft2(spec, s=(self.n, self.n))

    def uv(self, w):
        psi = w * self.ik2
        return self.phys(1j * self.ky * psi), self.phys(-1j * self.kx * psi)

    def nonlinear(self, w, stage):
        u, v = self.uv(w)
        nl = self.kx * self.ky * torch.fft.rfft2(v * v - u * u)
        nl += (self.kx * self.kx - self.ky * self.ky) * torch.fft.rfft2(u * v)
        if self.extra is not None:
            if stage == 0 or self.every:
                self.held = self.extra(self, w)
            nl = nl + self.held
        return nl * self.mask

    def cfl(self):
        u, v = self.uv(self.w)
        umax = u.abs().amax(dim=(-2, -1)) + v.abs().amax(dim=(-2, -1))
        return torch.clamp(CFL * (2.0 * math.pi / self.n) / umax, max=DT_MAX)

    def density(self):
        return self.w.abs().square() * self.wt

    def set_power(self):
        band = (self.k2 >= KLO**2) & (self.k2 <= KHI**2)
        eb = 0.5 * (self.density() * self.ik2 * band).sum(dim=(-2, -1))
        self.amp = POWER / (2.0 * eb)

    def step(self, dt):
        self.t = self.t + dt
        h = dt[..., None, None]
        lin = -(self.nu * self.k2)
        if self.forced:
            lin = lin - ALPHA * (self.k2 <= ALPHA_KMAX**2)
            lin = lin + self.amp[..., None, None] * ((self.k2 >= KLO**2) & (self.k2 <= KHI**2))
        e, eh = torch.exp(lin * h), torch.exp(lin * (0.5 * h))
        w = self.w
        k = self.nonlinear(w, 0)
        acc = e * (w + h / 6.0 * k)
        k = self.nonlinear(eh * (w + 0.5 * h * k), 1)
        acc += h / 3.0 * eh * k
        k = self.nonlinear(eh * w + 0.5 * h * k, 2)
        acc += h / 3.0 * eh * k
        k = self.nonlinear(e * w + h * eh * k, 3)
        self.w = acc + h / 6.0 * k

    def steps(self, count, every, dt=None):
        h = None
        for i in range(count):
            if i % every == 0:
                h = self.cfl() if dt is None else torch.full_like(self.t, dt)
                if self.forced and dt is None:
                    self.set_power()
            self.step(h)

    def sums(self):
        d = self.density()
        return np.array([0.5 * float((d * self.ik2).sum()), 0.5 * float(d.sum())])

    def spectrum(self):
        shell = torch.floor(self.k2.sqrt() + 0.5).long()
        out = torch.zeros(int(math.sqrt(2.0) * (self.n // 2) + 0.5) + 1, device="cuda",
                          dtype=torch.float64)
        return out.index_add_(0, shell.reshape(-1),
                              (0.5 * self.density() * self.ik2).reshape(-1)).cpu().numpy()


class _Exact3D:
    """The 3D rotational / Basdevant equations, unforced, in complex128."""

    def __init__(self, u, nu, rot):
        self.n, self.nu, self.rot = u.shape[-2], nu, rot
        self.k = _wave(self.n, 3)
        self.k2 = sum(k * k for k in self.k)
        self.ik2 = torch.where(self.k2 > 0, 1.0 / torch.where(self.k2 > 0, self.k2, 1.0), 0.0)
        self.mask = _mask(self.n, 3)
        self.u = u * self.mask
        self.t = 0.0

    def phys(self, f):
        return torch.fft.irfftn(f, s=(self.n,) * 3, dim=(-3, -2, -1))

    def spec(self, f):
        return torch.fft.rfftn(f, dim=(-3, -2, -1))

    def nonlinear(self, s):
        kx, ky, kz = self.k
        u = [self.phys(c) for c in s]
        if self.rot:
            w = [self.phys(1j * (ky * s[2] - kz * s[1])), self.phys(1j * (kz * s[0] - kx * s[2])),
                 self.phys(1j * (kx * s[1] - ky * s[0]))]
            nl = [self.spec(u[1] * w[2] - u[2] * w[1]), self.spec(u[2] * w[0] - u[0] * w[2]),
                  self.spec(u[0] * w[1] - u[1] * w[0])]
        else:
            q = (u[0] * u[0] + u[1] * u[1] + u[2] * u[2]) / 3.0
            t11, t22 = self.spec(u[0] * u[0] - q), self.spec(u[1] * u[1] - q)
            t12, t13, t23 = (self.spec(u[0] * u[1]), self.spec(u[0] * u[2]),
                             self.spec(u[1] * u[2]))
            nl = [-1j * (kx * t11 + ky * t12 + kz * t13), -1j * (kx * t12 + ky * t22 + kz * t23),
                  -1j * (kx * t13 + ky * t23 - kz * (t11 + t22))]
        div = (kx * nl[0] + ky * nl[1] + kz * nl[2]) * self.ik2
        return torch.stack([(c - k * div) * self.mask for c, k in zip(nl, self.k)])

    def cfl(self):
        umax = sum(float(self.phys(c).abs().max()) for c in self.u)
        return min(DT_MAX, CFL * (2.0 * math.pi / self.n) / umax)

    def step(self, h):
        self.t += h
        e, eh = torch.exp(-self.nu * self.k2 * h), torch.exp(-self.nu * self.k2 * (0.5 * h))
        u = self.u
        k = self.nonlinear(u)
        acc = e * (u + h / 6.0 * k)
        k = self.nonlinear(eh * (u + 0.5 * h * k))
        acc += h / 3.0 * eh * k
        k = self.nonlinear(eh * u + 0.5 * h * k)
        acc += h / 3.0 * eh * k
        k = self.nonlinear(e * u + h * eh * k)
        self.u = acc + h / 6.0 * k

    def steps(self, count, every, dt=None):
        h = dt
        for i in range(count):
            if i % every == 0 and dt is None:
                h = self.cfl()
            self.step(h)

    def density(self):
        w = torch.full((self.n // 2 + 1,), 2.0, device="cuda", dtype=torch.float64)
        w[0] = w[-1] = 1.0
        return sum(c.abs().square() for c in self.u) * (w / float(self.n) ** 6)

    def sums(self):
        d = self.density()
        return np.array([0.5 * float(d.sum()), 0.5 * float((d * self.k2).sum())])

    def spectrum(self):
        shell = torch.floor(self.k2.sqrt() + 0.5).long()
        out = torch.zeros(int(math.sqrt(3.0) * (self.n // 2) + 0.5) + 1, device="cuda",
                          dtype=torch.float64)
        return out.index_add_(0, shell.reshape(-1), (0.5 * self.density()).reshape(-1)).cpu().numpy()


def _gelu(z):
    return 0.5 * z * (1.0 + torch.tanh(0.7978845608028654 * (z + 0.044715 * z**3)))


def _net(p, x):
    """The network on (points, 75) inputs; p: 15440 float64 parameters."""
    for layer, fan in enumerate((75, 64, 64)):
        w = p[layer * 5120: (layer + 1) * 5120].reshape(64, 80)
        x = _gelu(x @ w[:, :fan].T + w[:, fan])
    return x @ p[15360: 15424] + p[15424]


def _stencils(f, rows, cols):
    """(points, 75) 5 x 5 stencils of the three fields f (3, n, n) at the given points."""
    n = f.shape[-1]
    d = torch.arange(-2, 3, device="cuda")
    r = (rows[:, None, None] + d[None, :, None]) % n
    c = (cols[:, None, None] + d[None, None, :]) % n
    return f[:, r, c].permute(1, 0, 2, 3).reshape(rows.numel(), 75)


def _les_term(p):
    scale = torch.tensor(LES_INSCALE, dtype=torch.float32, device="cuda").double()[:, None, None]

    def term(flow, w):
        n = flow.n
        f = torch.stack([flow.phys(w * g) for g in (1.0, 1j * flow.kx, 1j * flow.ky)]) * scale
        i = torch.arange(n * n, device="cuda")
        s = float(np.float32(LES_OUTSCALE)) * _net(p, _stencils(f, i // n, i % n))
        out = torch.fft.rfft2(s.reshape(n, n))
        out[0, 0] = 0.0  # the mean of the term is not applied
        return out

    return term


def _mix64(x):
    m = (1 << 64) - 1
    x = (x + 0x9E3779B97F4A7C15) & m
    x = ((x ^ (x >> 30)) * 0xBF58476D1CE4E5B9) & m
    x = ((x ^ (x >> 27)) * 0x94D049BB133111EB) & m
    return x ^ (x >> 31)


def _exact_train(case, seed):
    """Adam on the mean squared error of the drawn tiles: the documented counter hash picks
    (snapshot, row, 128-point segment) of each tile of a step."""
    n, count = case["n"], case["entries"]
    bank = _fields(n, count, _gen(seed)).double()
    std = bank.square().mean(dim=(0, 2, 3)).sqrt().cpu().numpy()
    scale = torch.tensor((1.0 / std[:3]).astype(np.float32), device="cuda").double()
    outscale = float(np.float32(std[3]))
    p = torch.tensor(_params(seed), device="cuda").double().requires_grad_()
    used = torch.zeros(15440, dtype=torch.float64, device="cuda")
    for layer, fan in enumerate((75, 64, 64)):
        used[layer * 5120: (layer + 1) * 5120].reshape(64, 80)[:, : fan + 1] = 1.0
    used[15360: 15425] = 1.0
    m, v, losses, lane = torch.zeros_like(used), torch.zeros_like(used), [], torch.arange(
        128, device="cuda")
    for step in range(case["steps"]):
        snap, rows, cols = [], [], []
        for i in range(case["tiles"]):
            h = _mix64((int(seed) % 1000 + _mix64((step << 32) | i)) & ((1 << 64) - 1))
            lo = h & 0xFFFFFFFF
            snap.append((h >> 32) % count)
            rows.append(lo % n)
            cols.append((lo // n) % (n // 128) * 128)
        s, r, c = (torch.tensor(a, device="cuda").repeat_interleave(128)
                   for a in (snap, rows, cols))
        c = c + lane.repeat(case["tiles"])
        d = torch.arange(-2, 3, device="cuda")
        x = torch.stack([bank[s[:, None, None], f, (r[:, None, None] + d[:, None]) % n,
                              (c[:, None, None] + d) % n] * scale[f] for f in range(3)], dim=1)
        loss = (_net(p, x.reshape(-1, 75)) - bank[s, 3, r, c] / outscale).square().mean()
        (g,) = torch.autograd.grad(loss, p)
        g = g * used
        losses.append(float(loss.detach()))
        with torch.no_grad():
            t = step + 1
            lr = 1e-3 * t / 200 if t <= 200 else 1e-5 + 0.5 * (1e-3 - 1e-5) * (
                1.0 + math.cos(math.pi * min((t - 200) / 19800.0, 1.0)))
            m = 0.9 * m + 0.1 * g
            v = 0.999 * v + 0.001 * g * g
            p -= lr * (m / (1.0 - 0.9**t)) / ((v / (1.0 - 0.999**t)).sqrt() + 1e-8)
    return {"losses": np.array(losses), "params": p.detach().cpu().numpy()}


def exact(case, seed):
    every = min(CFL_EVERY, case["steps"])
    if case["kind"] == "flow":
        a = _flow_state(case, seed)
        if case["dtype"] == "float32":  # the state as the solver is given it
            a = a.to(torch.complex64).to(torch.complex128)
        dt = _dt(case) if case["drive"] == "fixed" else None
        flow = (_Exact2D(a, _nu(case), case["forced"]) if case["dim"] == 2
                else _Exact3D(a, _nu(case), case["form"] == "rotational"))
        flow.steps(_steps(case), every, dt)
        out = {"state": flow.w if case["dim"] == 2 else flow.u, "t": float(flow.t)}
        if case["records"]:
            out["sums"], out["spectrum"] = flow.sums(), flow.spectrum()
        return out
    if case["kind"] == "ensemble":
        out, t = {}, []
        for n, w in sorted(_ensemble_states(case, seed).items()):
            if case["dtype"] == "float32":
                w = w.to(torch.complex64).to(torch.complex128)
            flow = _Exact2D(w, _nu_forced(n), True)
            flow.steps(case["steps"], CFL_EVERY)
            out[f"n{n:04d}"] = flow.w
            t.append(flow.t.cpu().numpy())
        return {**out, "t": np.concatenate(t)}
    if case["kind"] == "les":
        w = _les_state(case, seed).to(torch.complex64).to(torch.complex128)
        p = torch.tensor(_params(seed), device="cuda").double()
        flow = _Exact2D(w, LES_NU, True, _les_term(p), case["every_stage"])
        flow.steps(_steps(case), CFL_EVERY)
        return {"state": flow.w, "t": float(flow.t)}
    return _exact_train(case, seed)
