"""Workloads of the Schroedinger-Poisson step for timing and comparison, each
through the package's public calls:

  evolve    one box: psi in, a run of fixed-mode leap-frog steps, psi and the
            scale factor out (``Simulation.set_psi`` / ``step`` / ``get_psi_into``);
  grad      the same run and the gradient of a loss with respect to the psi it
            started from (``autograd.evolve`` and its backward pass);
  batch     many small boxes of uneven sizes advanced together (``Batch``);
  fft       the 3-D transform of a caller's own field, forward and back
            (``fft3d_``);
  spectrum  P(k) and the energy means of a box (``power_spectrum``, ``energies``).

The fields are seeded Zel'dovich-like ones at z = 50 (P(k) ~ k^-2.5, rms
density contrast 0.02) in a 10 Mpc/h box, psi in the reference's units
(|psi| ~ 1e50).  The fixed-step scale is the schedule that reaches a = 0.5 in
100 steps up to 64^3 and in 1000 steps from there on, at most the reference's
own rule (1.0).
"""

import math

import numpy as np
import torch

import ifdm_code_b200 as ifdm
from ifdm_code_b200.autograd import evolve

MFDM, XMAX, A0 = 2.5e-24, 5.0, 1.0 / 51.0
SIZES = {"fp64": (16, 32, 48, 64, 96, 128, 256, 512), "fp32": (16, 32, 48, 64, 96, 128, 256, 512),
         "mixed": (16, 32, 48, 64, 96, 128, 256)}

# the reference's unit system (Mpc, Myr, solar masses, eV)
_MPC, _MYR, _H = 3.086e22, 60.0 * 60.0 * 24.0 * 365.0 * 1e6, 0.677
RHOC, OMEGA_M = 3.51059e10, 0.276
HUBBLE = _H * 100.0 * _MYR / _MPC * 1e3
HBAR = 6.58211928e-16 / _MYR
LIGHT = 2.99792458e8 / _MPC * _MYR
GRAV = 6.674e-11 * 1.989e30 / _MPC**3 * _MYR**2


def _solar(mfdm):
    return mfdm * 1.783e-36 / 1.989e30


def _unit(mfdm):
    """|psi| of the mean density: results of the FP32 and mixed paths are kept in this unit."""
    return math.sqrt(RHOC / _solar(mfdm))


def _scale(n):
    """Fixed-step scale of an n^3 run: a = 0.5 after 100 (n <= 64) or 1000 steps."""
    return min(1.0, 0.111 * (n / 64.0) ** 2 * (1.0 if n <= 64 else 0.1))


def listed():
    return [
        # the smallest grid of the golden reference runs: ten launches of a few microseconds a step
        {"name": "evolve-fp64-16", "kind": "evolve", "n": 16, "prec": "fp64", "steps": 20, "g": 0.0},
        # the plain method's configuration: 64^3, 100 steps from z = 50
        {"name": "evolve-fp64-64", "kind": "evolve", "n": 64, "prec": "fp64", "steps": 100, "g": 0.0},
        # a grid with a factor of 3, FP64 arithmetic on FP32 storage, self-interaction
        {"name": "evolve-mixed-96", "kind": "evolve", "n": 96, "prec": "mixed", "steps": 20, "g": 1e-63},
        # the differentiation configuration's grid, forward only
        {"name": "evolve-fp32-128", "kind": "evolve", "n": 128, "prec": "fp32", "steps": 20, "g": 0.0},
        # the precision configuration's grid in the mixed mode
        {"name": "evolve-mixed-256", "kind": "evolve", "n": 256, "prec": "mixed", "steps": 10, "g": 0.0},
        # the benchmark's workload: 512^3 FP32 with self-interaction
        {"name": "evolve-fp32-512", "kind": "evolve", "n": 512, "prec": "fp32", "steps": 10, "g": 1.47e-62},
        # the same grid on the drop-in FP64 path
        {"name": "evolve-fp64-512", "kind": "evolve", "n": 512, "prec": "fp64", "steps": 5, "g": 1.47e-62},
        # differentiation: checkpointed forward run and its adjoint, FP32 at 128^3
        {"name": "grad-fp32-128", "kind": "grad", "n": 128, "prec": "fp32", "steps": 20, "every": 20, "g": 0.0},
        # the finite-difference checks' run: FP64, several segments, the last one short
        {"name": "grad-fp64-64", "kind": "grad", "n": 64, "prec": "fp64", "steps": 24, "every": 7, "g": 1e-63},
        # a quarter of the 96-realisation batch: 32^3, 48^3, 64^3 and 96^3 boxes side by side
        {"name": "batch-fp32-24", "kind": "batch", "n32": 8, "n48": 8, "n64": 6, "n96": 2, "prec": "fp32", "steps": 20},
        # a caller's own complex128 field, to k space and back
        {"name": "fft-c128-256", "kind": "fft", "n": 256, "dtype": "c128", "steps": 1},
        # a run's diagnostics between steps
        {"name": "spectrum-fp64-256", "kind": "spectrum", "n": 256, "prec": "fp64", "bins": 24},
    ]


def _log(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)) - 0.2)))))


def draw(rng):
    kind = rng.choices(("evolve", "grad", "batch", "fft", "spectrum"), (50, 15, 12, 13, 10))[0]
    most = max(work(c)["bytes"] for c in listed())
    while True:
        if kind == "evolve":
            prec = rng.choices(("fp64", "fp32", "mixed"), (4, 4, 2))[0]
            case = {"kind": kind, "n": rng.choice(SIZES[prec]), "prec": prec, "steps": _log(rng, 2, 100),
                    "g": rng.choice((0.0, 1e-63))}
        elif kind == "grad":
            case = {"kind": kind, "n": rng.choice((16, 32, 48, 64, 96, 128)), "prec": rng.choice(("fp64", "fp32", "mixed")),
                    "steps": _log(rng, 3, 24), "every": rng.choice((4, 7, 20)), "g": rng.choice((0.0, 1e-63))}
        elif kind == "batch":
            case = {"kind": kind, "n32": rng.randint(1, 12), "n48": rng.randint(0, 10), "n64": rng.randint(0, 8),
                    "n96": rng.randint(0, 3), "prec": rng.choice(("fp64", "fp32", "mixed")), "steps": _log(rng, 5, 50)}
        elif kind == "fft":
            case = {"kind": kind, "n": rng.choice((16, 32, 48, 64, 96, 128, 256, 512)), "dtype": rng.choice(("c128", "c64")),
                    "steps": rng.randint(1, 3)}
        else:
            case = {"kind": kind, "n": rng.choice((32, 48, 64, 96, 128, 256, 512)), "prec": "fp64", "bins": rng.randint(8, 40)}
        if work(case)["bytes"] <= most:
            return case


def work(case):
    n3 = float(case.get("n", 0)) ** 3
    lg = 5.0 * math.log2(max(2.0, n3))  # one complex transform, operations per cell
    cell = 48.0 if case.get("prec") == "fp64" else 24.0  # psi and phi read and written once a step
    if case["kind"] == "evolve":
        return {"bytes": n3 * (32.0 + cell * case["steps"]), "flops": n3 * case["steps"] * (3.0 * lg + 40.0)}
    if case["kind"] == "grad":  # the forward run, its replay, and the sweep over (g, psi, phi) of every step
        k = case["steps"]
        return {"bytes": n3 * (64.0 + cell * k * 3.0), "flops": n3 * k * (9.0 * lg + 150.0)}
    if case["kind"] == "batch":
        t = [(case["n%d" % n], float(n) ** 3) for n in (32, 48, 64, 96)]
        return {"bytes": sum(c * m * (32.0 + cell * case["steps"]) for c, m in t),
                "flops": sum(c * m * case["steps"] * (15.0 * math.log2(m) + 40.0) for c, m in t)}
    if case["kind"] == "fft":
        b = 16.0 if case["dtype"] == "c128" else 8.0
        return {"bytes": n3 * b * (1.0 + 2.0 * case["steps"]), "flops": n3 * lg * 2.0 * case["steps"]}
    return {"bytes": n3 * 24.0, "flops": n3 * (1.5 * lg + 60.0)}


def _field(n, seed, mfdm=MFDM):
    """psi of a seeded Gaussian random field at z = 50: complex128 (n, n, n) on the GPU."""
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev)
    gen.manual_seed(int(seed))
    wk = torch.fft.rfftn(torch.randn((n, n, n), generator=gen, device=dev, dtype=torch.float64))
    step = 2.0 * XMAX * 1e3 / n  # kpc/h
    kf = 2.0 * math.pi * torch.fft.fftfreq(n, d=step, device=dev, dtype=torch.float64)
    kr = 2.0 * math.pi * torch.fft.rfftfreq(n, d=step, device=dev, dtype=torch.float64)
    k2 = kf[:, None, None] ** 2 + kf[None, :, None] ** 2 + kr[None, None, :] ** 2
    k2[0, 0, 0] = 1.0
    wk *= k2 ** (-2.5 / 4.0)
    wk[0, 0, 0] = 0.0
    delta = torch.fft.irfftn(wk, s=(n, n, n))
    norm = 0.02 / float(delta.std())
    pot = torch.fft.irfftn(wk * (-norm / k2), s=(n, n, n))
    e = math.sqrt(OMEGA_M / A0**3 + 1.0 - OMEGA_M)
    vel = math.sqrt(A0) * 0.1 * e * (OMEGA_M / A0**3 / e**2) ** 0.55
    pot *= mfdm / LIGHT**2 / HBAR * A0**1.5 * (1e3 / _MPC * _MYR) * vel / (1e3 * _H)
    return torch.polar((1.0 + norm * delta).clamp_(min=0.0).sqrt_().mul_(1.225 * _unit(mfdm)), pot)


def _cotangent(n, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed) + 77)
    return torch.randn((n, n, n), generator=gen, device="cuda", dtype=torch.complex128) / _unit(MFDM)


def _boxes(case):
    sizes = [n for n in (32, 48, 64, 96) for _ in range(case["n%d" % n])]
    return [(n, 1e-24 * (1.0 + 4.0 * ((7 * i + 3) % 11) / 10.0)) for i, n in enumerate(sizes)]


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "evolve":
        n = case["n"]
        s["psi"] = _field(n, seed)
        s["out"] = torch.empty_like(s["psi"])
        s["sim"] = ifdm.Simulation(MFDM, case["g"], XMAX, n, precision=case["prec"])
    elif kind == "grad":
        n = case["n"]
        s["psi"] = _field(n, seed).requires_grad_(True)
        s["cot"] = _cotangent(n, seed)
        s["sim"] = ifdm.Simulation(MFDM, case["g"], XMAX, n, precision=case["prec"])
    elif kind == "batch":
        boxes = _boxes(case)
        s["psi"] = [_field(n, 100 * seed + i, m) for i, (n, m) in enumerate(boxes)]
        s["out"] = [torch.empty_like(p) for p in s["psi"]]
        s["sims"] = [ifdm.Simulation(m, 0.0, XMAX, n, precision=case["prec"]) for n, m in boxes]
        s["dts"] = [0.5 * _scale(n) for n, _ in boxes]
        for sim, p in zip(s["sims"], s["psi"]):
            sim.set_psi(p, A0)
        s["batch"] = ifdm.Batch(s["sims"])
    elif kind == "fft":
        gen = torch.Generator(device="cuda")
        gen.manual_seed(int(seed))
        n = case["n"]
        s["x"] = torch.randn((n, n, n), generator=gen, device="cuda",
                             dtype=torch.complex128 if case["dtype"] == "c128" else torch.complex64)
        s["k"], s["y"] = torch.empty_like(s["x"]), torch.empty_like(s["x"])
    else:
        s["sim"] = ifdm.Simulation(MFDM, 0.0, XMAX, case["n"], precision=case["prec"])
        s["sim"].set_psi(_field(case["n"], seed), A0)
    torch.cuda.synchronize()
    return s


def _kept(psi, prec, mfdm=MFDM):
    """psi as a program keeps it: complex128 as it comes, or complex64 in the
    unit of the mean density where the path stores 32 bits."""
    if prec == "fp64":
        return psi
    return torch.mul(psi, 1.0 / _unit(mfdm), out=torch.empty(psi.shape, dtype=torch.complex64, device=psi.device))


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "evolve":
        sim = s["sim"]
        if case["prec"] != "fp64":
            torch.cuda.current_stream().synchronize()  # the last result is read on torch's stream
        sim.set_psi(s["psi"], A0)
        sim.step(case["steps"], _scale(case["n"]))
        sim.get_psi_into(s["out"])
        return {"psi": _kept(s["out"], case["prec"]), "a": np.float32(sim.state()["a"])}
    if kind == "grad":
        out = evolve(s["psi"], s["sim"], A0, case["steps"], 0.5 * _scale(case["n"]), case["every"])
        (g,) = torch.autograd.grad(out, s["psi"], s["cot"])
        if case["prec"] == "fp64":
            return {"psi": out.detach(), "grad": g}
        return {"psi": _kept(out.detach(), case["prec"]), "grad": (g * _unit(MFDM)).to(torch.complex64)}
    if kind == "batch":
        if case["prec"] != "fp64":
            torch.cuda.current_stream().synchronize()
        for sim, p in zip(s["sims"], s["psi"]):
            sim.set_psi(p, A0)
        s["batch"].step(case["steps"], s["dts"])
        s["batch"].synchronize()
        for sim, o in zip(s["sims"], s["out"]):
            sim.get_psi_into(o)
        return [_kept(o, case["prec"], m) for o, (_, m) in zip(s["out"], _boxes(case))]
    if kind == "fft":
        k, y = s["k"], s["y"]
        k.copy_(s["x"])
        for i in range(case["steps"]):
            ifdm.fft3d_(k, -1)
            y.copy_(k)
            ifdm.fft3d_(y, +1)
            if i + 1 < case["steps"]:
                torch.mul(y, 1.0 / y.numel(), out=k)
        return [k, y]
    p = s["sim"].power_spectrum(case["bins"])
    return {"k": p["k"], "pk": p["pk"], "modes": p["modes"], "mean": p["mean_rho"], "energies": s["sim"].energies()}


# ------------------------------------------------- the same in plain 64 bits --
def _kappa(n):
    k = torch.arange(n, device="cuda", dtype=torch.float64)
    return torch.where(k < n // 2, k, k - n)


def _kappa2(n):
    k2 = _kappa(n) ** 2
    return k2[:, None, None] + k2[None, :, None] + k2[None, None, :]


_NODES, _WEIGHTS = np.polynomial.legendre.leggauss(24)


def _integral(a, da, power):
    """int da' / (H(a') a'^power) over the step."""
    x = a + 0.5 * da * (1.0 + _NODES)
    return float(np.sum(_WEIGHTS / (HUBBLE * np.sqrt(OMEGA_M / x**3 + 1.0 - OMEGA_M) * x**power)) * 0.5 * da)


def _phi(psi, k2, unit):
    """The potential of |psi|^2 (k = 0 removed); the density in units of unit^2."""
    rho = torch.fft.fftn((psi / unit).abs() ** 2)
    inv = torch.where(k2 == 0, torch.zeros_like(k2), -1.0 / k2)
    return torch.fft.ifftn(rho * inv).real


def _evolved(psi, n, g, steps, scale, mfdm=MFDM):
    """The leap-frog run in 64 bits (kick, drift, Poisson, kick; the reference's step rule)."""
    xmax = XMAX / _H
    kin, unit, k2 = mfdm / LIGHT**2 / HBAR, _unit(mfdm), _kappa2(n)
    grav = 4.0 * math.pi * GRAV * RHOC * (xmax / math.pi) ** 2
    pitch = 2 * (n // 2 + 1)  # the maximum of |phi| is taken over the first n^3 reals of the padded array
    rows, tail = divmod(n**3, pitch)
    a = A0
    phi = _phi(psi, k2, unit)
    for _ in range(steps):
        p = phi.detach().reshape(n * n, n)
        top = float(p[:rows].abs().max())
        if tail and rows < n * n:
            top = max(top, float(p[rows, :tail].abs().max()))
        dt = 4.0 / (3.0 * math.pi) * kin * (2.0 * xmax / n) ** 2 * a**2
        dt = min(dt, 2.0 * math.pi / kin / (grav * top) * a)
        if g:
            dt = min(dt, 2.0 * math.pi * HBAR / abs(g) / float(psi.detach().abs().max()) ** 2 * a**3)
        da = HUBBLE * math.sqrt(OMEGA_M / a**3 + 1.0 - OMEGA_M) * a * dt * scale
        t_ke, t_pe, t_qi = _integral(a, da, 3), _integral(a, da, 2), _integral(a, da, 4)
        a += da

        def kick(psi, phi):
            th = 0.5 * (t_pe * kin * grav) * phi
            if g:
                th = th + 0.5 * (t_qi * g / HBAR * unit**2) * (psi / unit).abs() ** 2
            return psi * torch.polar(torch.ones_like(th), -th)

        drift = 0.5 / kin * (math.pi / xmax) ** 2 * t_ke * k2
        psi = torch.fft.ifftn(torch.fft.fftn(kick(psi, phi)) * torch.polar(torch.ones_like(drift), -drift))
        phi = _phi(psi, k2, unit)
        psi = kick(psi, phi)
    return psi, a


def exact(case, seed):
    kind, n = case["kind"], case.get("n")
    if kind == "evolve":
        psi, a = _evolved(_field(n, seed), n, case["g"] / (3.086e24) ** 3, case["steps"], _scale(n))
        return {"psi": psi if case["prec"] == "fp64" else psi / _unit(MFDM), "a": a}
    if kind == "grad":
        psi0 = _field(n, seed).requires_grad_(True)
        psi, _ = _evolved(psi0, n, case["g"] / (3.086e24) ** 3, case["steps"], 0.5 * _scale(n))
        unit = _unit(MFDM)
        # the gradient through a loss of order one, and its scale put back
        (gr,) = torch.autograd.grad(psi / unit, psi0, _cotangent(n, seed) * unit)
        if case["prec"] == "fp64":
            return {"psi": psi.detach(), "grad": gr}
        return {"psi": psi.detach() / unit, "grad": gr * unit}
    if kind == "batch":
        out = []
        for i, (m, mass) in enumerate(_boxes(case)):
            psi, _ = _evolved(_field(m, 100 * seed + i, mass), m, 0.0, case["steps"], 0.5 * _scale(m), mass)
            out.append(psi if case["prec"] == "fp64" else psi / _unit(mass))
        return out
    if kind == "fft":
        gen = torch.Generator(device="cuda")
        gen.manual_seed(int(seed))
        x = torch.randn((n, n, n), generator=gen, device="cuda",
                        dtype=torch.complex128 if case["dtype"] == "c128" else torch.complex64).to(torch.complex128)
        k = torch.fft.fftn(x)
        return [k, torch.mul(x, float(n) ** 3)]
    psi = _field(n, seed)
    unit, xmax = _unit(MFDM), XMAX / _H
    rho = (psi / unit).abs() ** 2
    mean = float(rho.mean())
    k2 = _kappa2(n)
    kk = k2.sqrt()
    power = torch.fft.fftn(rho).abs() ** 2
    edges = [10.0 ** (i * (math.log10(n / 2.0) / case["bins"])) for i in range(case["bins"] + 1)]
    edges[0], edges[-1] = 1.0, n / 2.0
    ks, ps, ms = [], [], []
    for lo, hi in zip(edges[:-1], edges[1:]):
        at = (kk >= lo) & (kk < hi)
        c = int(at.sum())
        ms.append(c)
        ks.append(float(kk[at].mean()) * math.pi / xmax if c else 0.0)
        ps.append(float(power[at].mean()) * (2.0 * xmax) ** 3 / float(n) ** 6 / mean**2 if c else 0.0)
    grav = 4.0 * math.pi * GRAV * RHOC * (xmax / math.pi) ** 2
    phi = _phi(psi, k2, unit)
    pk2 = float((k2 * torch.fft.fftn(psi / unit).abs() ** 2).sum())
    u2 = unit**2
    return {"k": np.array(ks), "pk": np.array(ps), "modes": np.array(ms, dtype=np.int64), "mean": mean * u2,
            "energies": {"mean_rho": mean * u2, "mean_grad2": pk2 / float(n) ** 6 * (math.pi / xmax) ** 2 * u2,
                         "mean_phi_rho": grav * float((phi * rho).mean()) * u2, "mean_rho2": float((rho**2).mean()) * u2**2}}
