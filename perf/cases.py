"""The work a user has this framework do, as cases that can be timed and checked.

Every case goes through the public binding (cfb200.Context, Ensemble, Adjoint):

* evolve    RK4 steps of one lattice, optionally followed by the spectra an observer
            saves; `calls` x `steps`: a run between two observer saves is one call of
            many steps, an application that hands the stepper one step at a time makes
            many calls of one.
* observe   what an observer saves of a state: density and mode spectra, shells, slices.
* odeint    an application's own RK4 loop over the right-hand side and the linear
            combinations, one call each.
* ensemble  lattices of uneven size advanced together, spectra after each interval.
* gradient  one gradient of a spectrum loss with respect to shell amplitudes and mass.

Units follow the repository's configurations: L = N, radiation-dominated background
a = t^(1/2) from t = 1, dt = 0.05 (flat space and ensembles 0.1), unit-variance Gaussian
random fields; a curvature field k^-3 with rms Psi = 1e-2, either cut at k = 0.5 ("cut")
or with every mode of the lattice ("full", as the reference driver's initializer makes it).

`exact` restates the equations in plain torch FP64.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), os.pardir, "cosmic-fields-lite_b200"))

import cfb200  # noqa: E402

EQUATION = {"flat": cfb200.EQ_KG, "frw": cfb200.EQ_KG_FRW, "comoving": cfb200.EQ_COMOVING_FRW,
            "lambda": cfb200.EQ_LAMBDA_FRW, "sqrt": cfb200.EQ_SQRT_FRW, "fixed": cfb200.EQ_FIXED_CURVATURE_FRW,
            "approx": cfb200.EQ_APPROX_COMOVING_FRW}
PRECISION = {"fp64": cfb200.FP64, "fp32comp": cfb200.FP32_COMP}
A1, H1, T1 = 1.0, 0.5, 1.0  # a = t^(1/2)
LAM, F_A = 0.8, 0.7
MASS = 1.0
K_STAR, K_MAX, PSI_RMS = 0.25, 0.5, 1e-2
GROUPS, FLOOR, TARGET_MASS = 32, 1e-12, 1.1


def listed():
    return [
        # flat space at 64^3, an observer interval of 10 steps and both spectra
        evolve("flat_fp64_n64_interval", "flat", "fp64", 64, steps=10, spectra="both"),
        # the smallest call: one step of a small lattice, where launches are all there is
        evolve("frw_fp64_n48_one_step", "frw", "fp64", 48),
        # an observer interval (100 steps) of the 256^3 radiation-era run, compensated FP32
        evolve("frw_fp32comp_n256_interval", "frw", "fp32comp", 256, steps=100, spectra="density"),
        # a stepper object that is handed one step at a time, a self-interacting field, a ragged size
        evolve("lambda_fp64_n200_stepper", "lambda", "fp64", 200, calls=10),
        # the fourth-order stencil in FP64
        evolve("frw_fp64_13pt_n256", "frw", "fp64", 256, stencil=13, steps=20),
        # the curvature-coupled benchmark run
        evolve("comoving_fp32comp_n512", "comoving", "fp32comp", 512, steps=20, band="cut"),
        # the same with the fourth-order stencil
        evolve("comoving_fp32comp_13pt_n512", "comoving", "fp32comp", 512, stencil=13, steps=6, band="cut"),
        # the reference driver's own run: FP64, 384^3, a curvature field with every mode
        evolve("comoving_fp64_n384_full_band", "comoving", "fp64", 384, steps=4, band="full"),
        # everything the observer saves, at the benchmark's size
        {"name": "observe_comoving_n512", "kind": "observe", "equation": "comoving", "precision": "fp32comp",
         "n": 512, "band": "cut"},
        # an unmodified integrator that calls the right-hand side and the linear combinations
        {"name": "odeint_frw_n256", "kind": "odeint", "equation": "frw", "n": 256, "steps": 2, "band": "none"},
        # realisations of three sizes in one run, two observer intervals
        {"name": "ensemble_12", "kind": "ensemble", "precision": "fp32comp", "n0": 64, "n1": 96, "n2": 128,
         "each": 4, "steps": 25, "segments": 2},
        # one gradient of the inference loop
        {"name": "gradient_fp64_n128", "kind": "gradient", "precision": "fp64", "n": 128, "steps": 40, "every": 10},
    ]


def evolve(name, equation, precision, n, stencil=7, calls=1, steps=1, spectra="none", band="none", m=0):
    return {"name": name, "kind": "evolve", "equation": equation, "precision": precision, "n": n, "m": m,
            "stencil": stencil, "calls": calls, "steps": steps, "spectra": spectra, "band": band}


def draw(rng):
    """Another case: sizes from 32 to 512 in steps of 8 over their logarithm, a third of them
    powers of two; every equation, precision and stencil; no dearer than the benchmark run."""
    kind = rng.choices(["evolve", "observe", "odeint", "ensemble", "gradient"], [11, 3, 2, 2, 2])[0]
    precision = rng.choice(["fp64", "fp32comp"])
    if kind == "ensemble":
        n = sorted(_size(rng, 32, 128) for _ in range(3))
        return {"kind": kind, "precision": precision, "n0": n[0], "n1": n[1], "n2": n[2], "each": rng.randint(1, 4),
                "steps": rng.randint(5, 25), "segments": rng.randint(1, 2)}
    if kind == "gradient":
        n = _size(rng, 32, 128)
        every = rng.randint(2, 10)
        return {"kind": kind, "precision": precision, "n": n, "steps": every * rng.randint(1, 4), "every": every}
    equation = rng.choices(["flat", "frw", "comoving", "lambda", "sqrt", "fixed", "approx"], [2, 5, 6, 2, 1, 1, 1])[0]
    band = "none"
    if equation in ("comoving", "approx"):
        band = rng.choice(["cut", "cut", "full"])
    if kind == "odeint":
        equation = "frw" if equation == "approx" else equation
        return {"kind": kind, "equation": equation, "n": _size(rng, 32, 256), "steps": rng.randint(1, 4),
                "band": band if equation == "comoving" else "none"}
    if kind == "observe":
        equation = "frw" if equation == "approx" else equation
        return {"kind": kind, "equation": equation, "precision": precision, "n": _size(rng, 32, 512),
                "band": band if equation == "comoving" else "none"}
    n, m = _size(rng, 32, 512), 0
    if equation == "approx":
        coarse = 8 * rng.randint(2, 8)
        n, m = coarse * rng.randint(1, 512 // coarse), coarse
    stencil = rng.choices([7, 13], [3, 1])[0]
    cost = n ** 3 * (2.2 if precision == "fp64" else 1.0) * (2.8 if stencil == 13 else 1.0) * (2.5 if band == "full" else 1.0)
    most = max(1, min(100, int(20 * 512 ** 3 / cost)))
    if rng.random() < 0.25:
        calls, steps = rng.randint(1, max(1, min(10, most // 2))), 1
    else:
        calls, steps = 1, max(1, int(math.exp(rng.uniform(0.0, math.log(most)))))
    spectra = rng.choice(["none", "none", "density", "both"])
    case = evolve("", equation, precision, n, stencil, calls, steps, spectra, band, m)
    del case["name"]
    return case


def _size(rng, lo, hi):
    if rng.random() < 1 / 3:
        return 2 ** rng.randint(int(math.log2(lo)), int(math.log2(hi)))
    return 8 * int(round(math.exp(rng.uniform(math.log(lo / 8), math.log(hi / 8)))))


# ---- inputs (on the GPU, from the seed alone) ---------------------------------


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _white(n, g):
    return torch.randn((n, n, n), generator=g, device="cuda", dtype=torch.float64)


def _s2_grid(n):
    """s^2 = i^2 + j^2 + k^2 of every half-complex mode."""
    i = torch.arange(n, device="cuda")
    i = torch.minimum(i, n - i)
    k = torch.arange(n // 2 + 1, device="cuda")
    return (i * i)[:, None, None] + (i * i)[None, :, None] + (k * k)[None, None, :]


def _weights(n):
    """Modes of the full grid that a half-complex entry stands for, by k."""
    w = torch.full((n // 2 + 1,), 2.0, device="cuda", dtype=torch.float64)
    w[0] = w[n // 2] = 1.0
    return w


def _field(n, g, k_star=K_STAR):
    """Gaussian random field, P(k) ~ exp(-k^2 / 2 k*^2), zero mean, unit variance (L = N)."""
    k2 = _s2_grid(n).double() * (2 * math.pi / n) ** 2
    f = torch.fft.irfftn(torch.fft.rfftn(_white(n, g)) * torch.exp(-k2 / (4 * k_star ** 2)), s=(n, n, n))
    f = f - f.mean()
    return f / f.square().mean().sqrt()


def _curvature(n, g, band):
    """R_fft of a k^-3 curvature field, exactly zero outside its band, rms Psi(t = 1) = PSI_RMS."""
    s2 = _s2_grid(n)
    k = s2.double().sqrt() * (2 * math.pi / n)
    amp = torch.where(s2 > 0, k, torch.ones_like(k)) ** -1.5
    amp = torch.where((s2 > 0) if band == "full" else (s2 > 0) & (k <= K_MAX), amp, torch.zeros_like(amp))
    r = torch.fft.rfftn(_white(n, g)) * amp
    psi = torch.fft.irfftn(r * _transfer(n, 1.0, n, s2)[0], s=(n, n, n))
    return r * (PSI_RMS / psi.square().mean().sqrt())


def _state(case, seed):
    n, g = case["n"], _generator(seed)
    x = torch.stack([_field(n, g), 0.1 * _field(n, g)])
    extra = None
    if case["equation"] in ("comoving", "approx"):
        extra = _curvature(n, g, case["band"])
    elif case["equation"] == "fixed":
        extra = PSI_RMS * _field(n, g)
    return x, extra


def _t0(case):
    return 0.0 if case.get("equation") == "flat" else 1.0


def _dt(case):
    return 0.1 if case.get("equation") == "flat" or case["kind"] == "ensemble" else 0.05


# ---- preparation ----------------------------------------------------------------


def _context(case, precision, stencil=7):
    n = case["n"]
    ctx = cfb200.Context(n, float(n), m=MASS, equation=EQUATION[case["equation"]], precision=PRECISION[precision],
                         stencil=stencil, a1=A1, H1=H1, t1=T1, lam=LAM, f_a=F_A, M=case.get("m", 0))
    x, extra = _state(case, case["seed"])
    if extra is not None and case["equation"] == "fixed":
        ctx.set_psi(extra.reshape(-1).contiguous(), on_device=True)
    elif extra is not None:
        ctx.set_R_fft(torch.view_as_real(extra).reshape(-1).contiguous(), on_device=True)
    torch.cuda.synchronize()
    return ctx, x


def _doubles(n):
    return torch.empty(n, device="cuda", dtype=torch.float64)


def prepare(case, seed):
    return {"evolve": _prepare_lattice, "observe": _prepare_lattice, "odeint": _prepare_odeint,
            "ensemble": _prepare_ensemble, "gradient": _prepare_gradient}[case["kind"]](dict(case, seed=seed))


def _prepare_lattice(case):
    ctx, x = _context(case, case["precision"], case.get("stencil", 7))
    info = ctx.info
    s = dict(case, ctx=ctx, step=0, t0=_t0(case), dt=_dt(case), x=_doubles(info.state_bytes // 8))
    ctx.import_f64(s["x"], x)
    if case["kind"] == "observe":
        n = case["n"]
        s.update(rho=_doubles(info.s2_bins), shells=_doubles(info.shells), plus=_doubles(info.s2_bins),
                 counts=torch.empty(info.shells, device="cuda", dtype=torch.int64), slice=_doubles(n * n), mean=_doubles(n * n))
        return s
    if case["precision"] == "fp32comp":
        s["xy"] = _doubles(2 * info.field_count)
    if case["spectra"] != "none":
        s["rho"] = _doubles(info.s2_bins)
    if case["spectra"] == "both":
        s["plus"] = _doubles(info.s2_bins)
    return s


def _prepare_odeint(case):
    ctx, x = _context(case, "fp64")
    s = dict(case, ctx=ctx, step=0, t0=_t0(case), dt=_dt(case), x=x.reshape(-1).contiguous())
    s["k"] = [torch.empty_like(s["x"]) for _ in range(4)]
    s["tmp"] = torch.empty_like(s["x"])
    return s


def _members(case, seed):
    rng = np.random.default_rng(seed)
    sizes = [case[k] for k in ("n0", "n1", "n2") for _ in range(case["each"])]
    g = _generator(seed)
    out = []
    for n in sizes:
        f = _field(n, g, 0.5)
        out.append((n, float(rng.uniform(0.5, 2.0)), torch.stack([f, torch.zeros_like(f)])))
    return out


def _prepare_ensemble(case):
    members = _members(case, case["seed"])
    ens = cfb200.Ensemble([dict(N=n, L=float(n), m=m, equation=cfb200.EQ_KG_FRW, precision=PRECISION[case["precision"]],
                                stencil=7, a1=A1, H1=H1, t1=T1) for n, m, _ in members])
    stream = torch.cuda.Stream()
    for i, (_, _, x) in enumerate(members):
        ens.upload(i, x.reshape(-1).cpu().numpy(), stream=stream)
    stream.synchronize()
    return dict(case, ens=ens, stream=stream, t=1.0, spectra=_doubles(case["segments"] * ens.spectra_total))


def _amplitudes(case, seed):
    """xi, sqrt(P) by s^2, theta and the target shells (from a run at another mass)."""
    n = case["n"]
    xi = torch.fft.rfftn(_white(n, _generator(seed))) / n ** 3
    s2 = torch.arange(3 * (n // 2) ** 2 + 1, device="cuda", dtype=torch.float64)
    p = torch.exp(-s2 * (2 * math.pi / n) ** 2 / (2 * K_STAR ** 2))
    p[0] = 0.0
    total = (p[_s2_grid(n)] * _weights(n)).sum()
    sqrt_p = torch.sqrt(p * n ** 3 / total)
    theta = np.random.default_rng(seed).uniform(0.8, 1.25, GROUPS)
    phi = _initial_phi(case, xi, sqrt_p, torch.ones(GROUPS, device="cuda", dtype=torch.float64))
    target = _shells_after(case, torch.stack([phi, torch.zeros_like(phi)]), TARGET_MASS)
    return xi, sqrt_p, theta, target


def _per_group(n):
    shells = math.isqrt(3 * (n // 2) ** 2) + 1
    return -(-shells // GROUPS)


def _prepare_gradient(case):
    n = case["n"]
    xi, sqrt_p, theta, target = _amplitudes(case, case["seed"])
    ctx = cfb200.Context(n, float(n), m=MASS, equation=cfb200.EQ_KG_FRW, precision=PRECISION[case["precision"]], a1=A1,
                         H1=H1, t1=T1)
    return dict(case, ctx=ctx, adj=cfb200.Adjoint(ctx, case["steps"], case["every"]), theta=theta,
                xi=torch.view_as_real(xi).reshape(-1).contiguous(), sqrt_p=sqrt_p, target=target.cpu().numpy(),
                x=_doubles(ctx.info.state_bytes // 8), x0=torch.zeros(2 * n ** 3, device="cuda", dtype=torch.float64),
                lam=_doubles(2 * n ** 3))


# ---- one pass -------------------------------------------------------------------


def run(s):
    return {"evolve": _run_evolve, "observe": _run_observe, "odeint": _run_odeint, "ensemble": _run_ensemble,
            "gradient": _run_gradient}[s["kind"]](s)


def _run_evolve(s):
    ctx, x = s["ctx"], s["x"]
    for _ in range(s["calls"]):
        ctx.rk4_steps(x, s["t0"], s["dt"], s["steps"], step0=s["step"])
        s["step"] += s["steps"]
    out = {}
    if s["spectra"] != "none":
        t = s["t0"] + s["step"] * s["dt"]
        ctx.density_spectrum_s2(x, t, s["rho"])
        out["rho"] = s["rho"]
        if s["spectra"] == "both":
            ctx.mode_power_spectrum_s2(x, _a(s, t), s["plus"])
            out["plus"] = s["plus"]
    if "xy" in s:  # the compensated state is read out as FP64
        ctx.export_f64(s["xy"], x)
        out["x"] = s["xy"]
    else:
        out["x"] = x
    return out


def _run_observe(s):
    ctx, x, t = s["ctx"], s["x"], s["t0"]
    ctx.density_spectrum_s2(x, t, s["rho"])
    ctx.s2_to_shells(s["shells"], s["counts"])
    ctx.mode_power_spectrum_s2(x, _a(s, t), s["plus"])
    ctx.density_slices(x, t, s["slice"], s["mean"])
    return {k: s[k] for k in ("rho", "shells", "counts", "plus", "slice", "mean")}


def _run_odeint(s):
    ctx, x, k, tmp, dt = s["ctx"], s["x"], s["k"], s["tmp"], s["dt"]
    n = x.numel()
    for _ in range(s["steps"]):
        t = s["t0"] + s["step"] * dt
        ctx.rhs(x, k[0], t)
        ctx.scale_sum(tmp, [x, k[0]], [1.0, dt / 2], n)
        ctx.rhs(tmp, k[1], t + dt / 2)
        ctx.scale_sum(tmp, [x, k[1]], [1.0, dt / 2], n)
        ctx.rhs(tmp, k[2], t + dt / 2)
        ctx.scale_sum(tmp, [x, k[2]], [1.0, dt], n)
        ctx.rhs(tmp, k[3], t + dt)
        ctx.scale_sum(x, [x] + k, [1.0, dt / 6, dt / 3, dt / 3, dt / 6], n)
        s["step"] += 1
    return x


def _run_ensemble(s):
    s["ens"].run_graph(s["t"], _dt(s), s["steps"], s["segments"], s["spectra"], stream=s["stream"])
    s["t"] += s["steps"] * s["segments"] * _dt(s)
    return s["spectra"]


def _run_gradient(s):
    ctx, adj, n3 = s["ctx"], s["adj"], s["n"] ** 3
    per = _per_group(s["n"])
    cfb200.field_from_shell_amplitudes(ctx, s["xi"], s["sqrt_p"], s["theta"], per, s["x0"][:n3])
    ctx.import_f64(s["x"], s["x0"])
    adj.forward(s["x"], 1.0, _dt(s))
    loss = adj.shell_log_loss(s["x"], s["target"], FLOOR)
    dm = adj.backward(s["lam"])
    dtheta = cfb200.shell_amplitude_gradient(ctx, s["lam"][:n3], s["xi"], s["sqrt_p"], s["theta"], per)
    return {"loss": loss, "dm": dm, "dtheta": dtheta, "lam": s["lam"]}


# ---- what a pass cannot do without --------------------------------------------------


def work(case):
    """The state read and written once a step (FP64 and compensated FP32: 32 bytes a site),
    Psi and its derivative written and read at the two new stage times of a step; an
    observer's inputs read and outputs written once; flops of the stage arithmetic."""
    kind = case["kind"]
    if kind == "ensemble":
        sites = case["each"] * sum(case[k] ** 3 for k in ("n0", "n1", "n2"))
        return {"bytes": 32.0 * sites * case["steps"] * case["segments"], "flops": 120.0 * sites * case["steps"] * case["segments"]}
    sites = case["n"] ** 3
    word = 4 if case.get("precision") == "fp32comp" else 8
    if kind == "gradient":
        # forward, and the reverse sweep's adjoint state; the forward states of a segment come again
        return {"bytes": 96.0 * sites * case["steps"], "flops": 360.0 * sites * case["steps"]}
    if kind == "observe":
        psi = word if case["equation"] in ("comoving", "fixed") else 0
        return {"bytes": float((16 + psi) * sites), "flops": 3 * 2.5 * sites * math.log2(sites) + 40.0 * sites}
    steps = case["steps"] * case.get("calls", 1)
    psi = 8 * word if case["equation"] == "comoving" else (word if case["equation"] == "fixed" else 0)
    return {"bytes": float((32 + psi) * sites * steps), "flops": (120.0 if case.get("stencil", 7) == 7 else 220.0) * sites * steps}


# ---- the same in plain torch FP64 ------------------------------------------------------


def _a(case, t):
    return 1.0 if case.get("equation") == "flat" else A1 * math.sqrt(1 + 2 * H1 * (t - T1))


def _hubble(case, t):
    return 0.0 if case.get("equation") == "flat" else H1 / (1 + 2 * H1 * (t - T1))


def _transfer(n, t, length, s2):
    """Psi and dPsi/dt over R, by mode, at t."""
    eta = math.sqrt(1 + 2 * H1 * (t - T1)) / (A1 * H1)
    x = s2.double().sqrt() * (2 * math.pi / length * eta / math.sqrt(3))
    zero = s2 == 0
    x = torch.where(zero, torch.ones_like(x), x)
    common = torch.where(zero, torch.zeros_like(x), 2 / x ** 3)
    sn, cs = torch.sin(x), torch.cos(x)
    hubble = H1 / (1 + 2 * H1 * (t - T1))
    return (sn - x * cs) * common, hubble * (3 * x * cs + (x * x - 3) * sn) * common


def _psi(case, extra, t):
    """What multiplies: e^{2 Psi}, e^{4 Psi} (the approximate equation's quadratics) and dPsi/dt."""
    n = case["n"]
    if case["equation"] == "fixed":
        return torch.exp(2 * extra), torch.exp(4 * extra), 0.0
    if case["equation"] == "approx":
        m = case["m"]
        i = torch.arange(m, device="cuda")
        at = torch.where(i < m // 2, i, n - (m - i))
        cut = extra[at][:, at][:, :, : m // 2 + 1] * (m / n) ** 3
        ft, gt = _transfer(m, t, n, _s2_grid(m))
        psi, dpsi = (torch.fft.irfftn(cut * f, s=(m, m, m)) for f in (ft, gt))
        near = ((torch.arange(n, device="cuda") + n // m // 2) % n) // (n // m)
        psi, dpsi = (f[near][:, near][:, :, near] for f in (psi, dpsi))
        return 1 + 2 * psi + 2 * psi ** 2, 1 + 4 * psi + 8 * psi ** 2, dpsi
    ft, gt = _transfer(n, t, n, _s2_grid(n))
    psi, dpsi = (torch.fft.irfftn(extra * f, s=(n, n, n)) for f in (ft, gt))
    e2 = torch.exp(2 * psi)
    return e2, e2 * e2, dpsi


def _laplacian(f, stencil):
    s1 = sum(f.roll(d, axis) for axis in range(3) for d in (1, -1))
    if stencil == 7:
        return s1 - 6 * f
    s2 = sum(f.roll(d, axis) for axis in range(3) for d in (2, -2))
    return (16 * s1 - s2 - 90 * f) / 12


def _rhs(case, x, t, mass, coupling):
    f, p = x[0], x[1]
    grad = _laplacian(f, case.get("stencil", 7)) / _a(case, t) ** 2
    rub = 3 * _hubble(case, t)
    eq = case.get("equation", "frw")
    if eq in ("comoving", "fixed", "approx"):
        e2, e4, dpsi = coupling
        return torch.stack([p, (4 * dpsi - rub) * p - e2 * mass ** 2 * f + e4 * grad])
    force = mass ** 2 * f
    if eq == "lambda":
        force = force + LAM * f ** 3
    elif eq == "sqrt":
        force = force / torch.sqrt(1 + f * f / F_A ** 2)
    return torch.stack([p, grad - rub * p - force])


def _rk4(case, x, extra, t, dt, mass=MASS):
    at = [None if extra is None else _psi(case, extra, u) for u in (t, t + dt / 2, t + dt)]
    k = _rhs(case, x, t, mass, at[0])
    acc = k
    k = _rhs(case, x + dt / 2 * k, t + dt / 2, mass, at[1])
    acc = acc + 2 * k
    k = _rhs(case, x + dt / 2 * k, t + dt / 2, mass, at[1])
    acc = acc + 2 * k
    k = _rhs(case, x + dt * k, t + dt, mass, at[2])
    return x + dt / 6 * (acc + k)


def _density(case, x, extra, t, mass=MASS):
    f, p = x[0], x[1]
    grad = sum((f.roll(-1, axis) - f.roll(1, axis)).square() for axis in range(3)) / (4 * _a(case, t) ** 2)
    eq = case.get("equation", "frw")
    if eq in ("comoving", "approx", "fixed"):
        # the approximate equation reports the full comoving energy density
        e2 = _psi(dict(case, equation="comoving") if eq == "approx" else case, extra, t)[0]
        return 0.5 * (p * p / e2 + mass ** 2 * f * f + e2 * grad)
    rho = 0.5 * (p * p + grad)
    if eq == "sqrt":
        return rho + mass ** 2 * f * f / (torch.sqrt(1 + f * f / F_A ** 2) + 1)
    rho = rho + 0.5 * mass ** 2 * f * f
    return rho + 0.25 * LAM * f ** 4 if eq == "lambda" else rho


def _bins(n, v):
    """Sums of the mode values v by s^2."""
    out = torch.zeros(3 * (n // 2) ** 2 + 1, device="cuda", dtype=torch.float64)
    return out.index_add(0, _s2_grid(n).reshape(-1), (v * _weights(n)).reshape(-1))


def _power(f):
    c = torch.fft.rfftn(f)
    return c.real.square() + c.imag.square()


def _mode_bins(case, x, t):
    n = case["n"]
    w2 = MASS ** 2 + (2 * math.pi / n) ** 2 * _s2_grid(n).double() / _a(case, t) ** 2
    return _bins(n, _power(x[0]) + _power(x[1]) / w2)


def _isqrt(s2):
    r = s2.double().sqrt().long()
    r = torch.where(r * r > s2, r - 1, r)
    return torch.where((r + 1) * (r + 1) <= s2, r + 1, r)


def _shells(n, bins):
    shell = _isqrt(torch.arange(bins.numel(), device="cuda"))
    return torch.zeros(math.isqrt(3 * (n // 2) ** 2) + 1, device="cuda", dtype=bins.dtype).index_add(0, shell, bins)


def _initial_phi(case, xi, sqrt_p, theta):
    """c2r(sqrt(theta_g) sqrt(P) xi), groups of _per_group unit shells."""
    n = case["n"]
    s2 = _s2_grid(n)
    group = torch.clamp(_isqrt(s2) // _per_group(n), max=GROUPS - 1)
    return torch.fft.irfftn(torch.sqrt(theta)[group] * sqrt_p[s2] * xi, s=(n, n, n)) * n ** 3


def _shells_after(case, x, mass):
    """Density shells at the end of the run from the state x."""
    n, dt = case["n"], _dt(case)
    for j in range(case["steps"]):
        x = _rk4(case, x, None, 1.0 + j * dt, dt, mass)
    return _shells(n, _bins(n, _power(_density(case, x, None, 1.0 + case["steps"] * dt, mass))))


def exact(case, seed):
    return {"evolve": _exact_evolve, "observe": _exact_observe, "odeint": _exact_odeint,
            "ensemble": _exact_ensemble, "gradient": _exact_gradient}[case["kind"]](case, seed)


def _exact_evolve(case, seed):
    x, extra = _state(case, seed)
    t0, dt, steps = _t0(case), _dt(case), case["calls"] * case["steps"]
    for j in range(steps):
        x = _rk4(case, x, extra, t0 + j * dt, dt)
    t = t0 + steps * dt
    out = {"x": x.reshape(-1)}
    if case["spectra"] != "none":
        out["rho"] = _bins(case["n"], _power(_density(case, x, extra, t)))
    if case["spectra"] == "both":
        out["plus"] = _mode_bins(case, x, t)
    return out


def _exact_observe(case, seed):
    n, t = case["n"], _t0(case)
    x, extra = _state(case, seed)
    rho = _density(case, x, extra, t)
    bins = _bins(n, _power(rho))
    return {"rho": bins, "shells": _shells(n, bins),
            "counts": _shells(n, _bins(n, torch.ones((n, n, n // 2 + 1), device="cuda", dtype=torch.float64))).long(),
            "plus": _mode_bins(case, x, t), "slice": rho[0].reshape(-1), "mean": rho.mean(0).reshape(-1)}


def _exact_odeint(case, seed):
    x, extra = _state(case, seed)
    for j in range(case["steps"]):
        x = _rk4(case, x, extra, _t0(case) + j * _dt(case), _dt(case))
    return x.reshape(-1)


def _exact_ensemble(case, seed):
    dt, out = _dt(case), [[] for _ in range(case["segments"])]
    for n, mass, x in _members(case, seed):
        for seg in range(case["segments"]):
            for j in range(seg * case["steps"], (seg + 1) * case["steps"]):
                x = _rk4(case, x, None, 1.0 + j * dt, dt, mass)
            rho = _density(case, x, None, 1.0 + (seg + 1) * case["steps"] * dt, mass)
            out[seg].append(_bins(n, _power(rho)))
    return torch.cat([b for seg in out for b in seg])


def _exact_gradient(case, seed):
    xi, sqrt_p, theta, target = _amplitudes(case, seed)
    theta = torch.tensor(theta, device="cuda", dtype=torch.float64, requires_grad=True)
    mass = torch.tensor(MASS, device="cuda", dtype=torch.float64, requires_grad=True)
    phi = _initial_phi(case, xi, sqrt_p, theta)
    x = torch.stack([phi, torch.zeros_like(phi)])
    x.retain_grad()
    shells = _shells_after(case, x, mass)
    kept = (shells > 0) & (target > FLOOR * target.max())
    loss = (torch.log(shells[kept]) - torch.log(target[kept])).square().sum()
    loss.backward()
    return {"loss": float(loss), "dm": float(mass.grad), "dtheta": theta.grad, "lam": x.grad.reshape(-1)}
