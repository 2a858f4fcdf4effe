"""The work a user of the framework has it do, as timed cases.

A case is one pass through a public entry point (`pubsed_b200.transport`,
`.engine`, `.batch`, `.adjoint`) at sizes taken from the workload generators'
own configurations, and scaled down and up from them:

  sphere    transport::step of one 1D model, as the steady-state driver calls
            it: grid upload, opacity build, emission, propagation,
            normalisation, temperature solve, results back (Transport.step)
  batch     a step of many 1D models at once (BatchEngine.step)
  cart      a step on a 3D Cartesian grid (Engine.step)
  gradient  emergent spectrum and its gradient (torch autograd Functions)
  pulse     a time-dependent step over carried packets with discrete
            diffusion (Transport.step)
  tables    the opacity build alone, tables read back (Engine.set_opacity)

`seed` keys both the model data and the packets' streams.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from pubsed_b200 import abi, adjoint, workloads
from pubsed_b200.batch import BatchEngine
from pubsed_b200.engine import Engine
from pubsed_b200.transport import Transport

PRECISION = {"fp64": abi.PREC_FP64, "mixed": abi.PREC_MIXED}


def listed():
    return [
        # the smallest calls: a debugging or smoke run of the grey lightbulb, where the
        # slowest packet's chain and the fixed cost of a step count
        {"name": "bulb few packets", "kind": "sphere", "model": "grey", "precision": "fp64", "packets": 2000,
         "zones": 128, "bins": 1024, "lines": 0, "decay": 0},
        # the plain configuration: grey lightbulb, FP64, 1e6 packets
        {"name": "bulb", "kind": "sphere", "model": "grey", "precision": "fp64", "packets": 1_000_000, "zones": 128,
         "bins": 1024, "lines": 0, "decay": 0},
        # the FP64 form on the line-rich model: the parity runs
        {"name": "ia fp64", "kind": "sphere", "model": "lines", "precision": "fp64", "packets": 300_000, "zones": 256,
         "bins": 4096, "lines": 500_000, "decay": 0},
        # a quick look at a small model with odd sizes: the opacity build and the temperature
        # solve weigh as much as the packets
        {"name": "ia quick", "kind": "sphere", "model": "lines", "precision": "mixed", "packets": 20_001, "zones": 97,
         "bins": 1500, "lines": 30_000, "decay": 0},
        # one iteration towards radiative equilibrium at a tenth of the full packet count, as
        # all but the last iteration of a steady-state run are done
        {"name": "ia iteration", "kind": "sphere", "model": "lines", "precision": "mixed", "packets": 1_000_000,
         "zones": 256, "bins": 4096, "lines": 500_000, "decay": 0},
        # the precision configuration at its full size: the last iteration
        {"name": "ia full", "kind": "sphere", "model": "lines", "precision": "mixed", "packets": 10_000_000,
         "zones": 256, "bins": 4096, "lines": 500_000, "decay": 0},
        # core and radioactive decay packets, as the reference's Type Ia example mixes them
        {"name": "ia decay", "kind": "sphere", "model": "lines", "precision": "mixed", "packets": 300_000, "zones": 256,
         "bins": 4096, "lines": 500_000, "decay": 30_000},
        # a parameter study: the 64-model batch at a tenth of its packets
        {"name": "batch 64", "kind": "batch", "models": 64, "scale": 0.1, "lines": 30_000, "bins": 2048},
        # 3D clumped ejecta with the full line list and bins
        {"name": "cart 64", "kind": "cart", "precision": "mixed", "packets": 2_000_000, "cells": 64, "bins": 2048,
         "lines": 100_000},
        # a fit's step: spectrum and gradient with respect to the (zone, band) absorption
        {"name": "gradient", "kind": "gradient", "of": "absorption", "packets": 1_000_000, "zones": 256, "bins": 4096,
         "lines": 500_000, "bands": 64},
        # a time-dependent step of the diffusing pulse
        {"name": "pulse", "kind": "pulse", "precision": "mixed", "packets": 1_000_000},
        # the opacity build with every continuum and line term, tables back on the host
        {"name": "tables", "kind": "tables", "precision": "mixed", "zones": 128, "bins": 2048, "lines": 100_000},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sphere", "sphere", "sphere", "batch", "cart", "gradient", "pulse", "tables"])
    precision = rng.choice(["fp64", "mixed"])
    if kind == "sphere":
        model = rng.choice(["grey", "lines", "lines"])
        if model == "grey":
            return {"kind": kind, "model": model, "precision": precision, "packets": _log_int(rng, 2000, 1_000_000),
                    "zones": rng.randint(50, 256), "bins": _log_int(rng, 200, 2048), "lines": 0, "decay": 0}
        top = 300_000 if precision == "fp64" else 3_000_000
        packets = _log_int(rng, 10_000, top)
        decay = packets // 10 if rng.random() < 0.25 and packets <= 300_000 else 0
        return {"kind": kind, "model": model, "precision": precision, "packets": packets,
                "zones": rng.randint(64, 256), "bins": _log_int(rng, 800, 4096),
                "lines": _log_int(rng, 30_000, 500_000), "decay": decay}
    if kind == "batch":
        return {"kind": kind, "models": rng.randint(3, 64), "scale": round(math.exp(rng.uniform(math.log(0.005), math.log(0.1))), 5),
                "lines": _log_int(rng, 10_000, 30_000), "bins": _log_int(rng, 500, 2048)}
    if kind == "cart":
        return {"kind": kind, "precision": precision, "packets": _log_int(rng, 50_000, 2_000_000),
                "cells": rng.randint(16, 64 if precision == "mixed" else 48), "bins": _log_int(rng, 500, 2048),
                "lines": _log_int(rng, 10_000, 100_000)}
    if kind == "gradient":
        return {"kind": kind, "of": rng.choice(["absorption", "density"]), "packets": _log_int(rng, 20_000, 1_000_000),
                "zones": rng.randint(64, 256), "bins": _log_int(rng, 1000, 4096),
                "lines": _log_int(rng, 50_000, 500_000), "bands": rng.choice([16, 37, 64])}
    if kind == "pulse":
        return {"kind": kind, "precision": precision, "packets": _log_int(rng, 20_000, 1_000_000)}
    return {"kind": kind, "precision": precision, "zones": rng.randint(20, 256), "bins": _log_int(rng, 500, 2048),
            "lines": _log_int(rng, 10_000, 100_000)}


def _workload(case, seed):
    seed = int(seed)
    kind = case["kind"]
    if kind == "sphere" and case["model"] == "grey":
        return workloads.lightbulb_grey(n_packets=case["packets"], n_zones=case["zones"], n_bins=case["bins"],
                                        radiative_eq=1, seed=seed)
    if kind == "sphere":
        return workloads.type_ia(n_packets=case["packets"], n_zones=case["zones"], n_lines=case["lines"],
                                 n_bins=case["bins"], n_radioactive=case["decay"], seed=seed, data_seed=seed)
    if kind == "batch":
        # the models' sizes come with the case, their temperatures and packet streams with the seed
        b = workloads.batch64(n_models=case["models"], n_lines=case["lines"], n_bins=case["bins"],
                              packet_scale=case["scale"], seed=seed)
        rng = np.random.default_rng(seed)
        for m in b.models:
            m.zones.T = m.zones.T * rng.uniform(0.9, 1.1)
        return b
    if kind == "cart":
        return workloads.cart3d(n_packets=case["packets"], n_cells=case["cells"], n_lines=case["lines"],
                                n_bins=case["bins"], seed=seed, data_seed=seed)
    if kind == "gradient":
        # almost pure scattering lines and absorption final, as the differentiable form needs it
        return workloads.type_ia(n_packets=case["packets"], n_zones=case["zones"], n_lines=case["lines"],
                                 n_bins=case["bins"], epsilon=1e-4, radiative_eq=0, seed=seed, data_seed=seed)
    if kind == "pulse":
        return workloads.diffusing_pulse(n_initialize=case["packets"], seed=seed)
    return workloads.type_ia(n_packets=1000, n_zones=case["zones"], n_lines=case["lines"], n_bins=case["bins"],
                             bound_free=1, seed=seed, data_seed=seed)


def prepare(case, seed):
    w = _workload(case, seed)
    s = {"case": dict(case)}
    kind = case["kind"]
    if kind == "batch":
        s["engine"] = BatchEngine(w, precision=abi.PREC_MIXED)
    elif kind == "gradient":
        eng = adjoint.DiffEngine(w, case["bands"], precision=abi.PREC_MIXED)
        eng.tables()
        shape = (eng.nz, eng.n_bands) if case["of"] == "absorption" else (eng.nz,)
        g = torch.Generator(device="cuda").manual_seed(int(seed))
        s["engine"] = eng
        s["theta"] = (0.9 + 0.2 * torch.rand(shape, generator=g, device="cuda", dtype=torch.float64)).requires_grad_()
        s["weight"] = torch.rand(eng.nspec, generator=g, device="cuda", dtype=torch.float64)
    elif kind in ("sphere", "pulse"):
        s["transport"] = Transport(w, precision=PRECISION[case["precision"]])
        s["T"] = w.zones.T.copy()
    else:
        s["engine"] = Engine(w, precision=PRECISION[case["precision"]])
    return s


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "sphere":
        tr = state["transport"]
        tr.w.zones.T = state["T"]  # the gas temperature the host hands in
        tr.step(1.0)
        flux, click = tr.eng.spectrum()
        out = {"flux": flux, "click": click, "T": tr.w.zones.T}
        out.update(tr.tallies)
        if tr.radio is not None:
            out.update(tr.radio)
        return out
    if kind == "pulse":
        tr = state["transport"]
        tr.step(5e-10)
        out = dict(tr.tallies)
        out["flux"], out["click"] = tr.eng.spectrum()
        out["n_particles"] = tr.n_particles()
        return out
    eng = state["engine"]
    if kind == "batch":
        eng.step(1.0)
        out = {"escaped": eng.escaped()}
        spec = [eng.spectrum(m) for m in range(case["models"])]
        tal = [eng.tallies(m, J=False) for m in range(case["models"])]
        out["flux"] = np.concatenate([f for f, _ in spec])
        out["click"] = np.concatenate([c for _, c in spec])
        for k in ("e_abs", "e_rad", "fx", "fy", "fz", "fr"):
            out[k] = np.concatenate([t[k] for t in tal])
        return out
    if kind == "cart":
        eng.step(1.0)
        flux, click = eng.spectrum()
        out = {"flux": flux, "click": click}
        out.update(eng.tallies(J=False))  # [cells x bins] J stays on the device
        return out
    if kind == "gradient":
        fn = adjoint.spectrum_from_absorption if case["of"] == "absorption" else adjoint.spectrum_from_density
        theta = state["theta"]
        theta.grad = None
        flux = fn(theta, eng, step=0)
        flux.backward(state["weight"])
        return {"flux": flux.detach(), "grad": theta.grad}
    eng.set_opacity(1.0)
    return eng.opacity()


# Segments (a packet's flight to its next zone wall, bin edge or interaction) per packet,
# measured on the listed cases; they vary with the drawn model's data by a factor of a few.
SEGMENTS = {"grey": 360, "lines": 1800, "decay": 28_000, "batch": 300, "cart": 370, "gradient": 1750, "pulse": 41}
# FP64 operations of one segment: two wall distances, the Doppler factor, the tallies, the
# move, and an interaction's two Lorentz transforms
FLOPS_PER_SEGMENT = 200


def work(case):
    kind = case["kind"]
    bins = case.get("bins", 1)
    lines_bytes = 32.0 * case.get("lines", 0)
    if kind == "sphere":
        seg = case["packets"] * SEGMENTS[case["model"]] + case["decay"] * SEGMENTS["decay"]
        z = case["zones"]
        return {"bytes": lines_bytes + 8.0 * z * (bins + 18) + 16.0 * 1024, "flops": float(FLOPS_PER_SEGMENT) * seg}
    if kind == "batch":
        packets = case["models"] * case["scale"] * (1e7 - 1e5) / math.log(100.0)
        return {"bytes": lines_bytes + case["models"] * (16.0 * 1024 + 288 * 8.0 * 18),
                "flops": FLOPS_PER_SEGMENT * packets * SEGMENTS["batch"]}
    if kind == "cart":
        z = case["cells"] ** 3
        # the build's Sobolev terms, ~20 operations each, beside the packets
        return {"bytes": lines_bytes + 8.0 * z * 18 + 16.0 * 1024 * 16,
                "flops": FLOPS_PER_SEGMENT * case["packets"] * SEGMENTS["cart"] + 20.0 * z * case["lines"]}
    if kind == "gradient":
        n = case["zones"] * (case["bands"] if case["of"] == "absorption" else 1)
        return {"bytes": 16.0 * n + 16.0 * 1024 + 24.0 * case["zones"] * bins,
                "flops": 2.0 * FLOPS_PER_SEGMENT * case["packets"] * SEGMENTS["gradient"]}
    if kind == "pulse":
        return {"bytes": case["packets"] * 160.0, "flops": float(FLOPS_PER_SEGMENT) * case["packets"] * SEGMENTS["pulse"]}
    z = case["zones"]
    return {"bytes": lines_bytes + 24.0 * z * bins, "flops": 20.0 * z * case["lines"] + 100.0 * z * bins}


# ------------------------------------------------------------ exact values
# The opacity build in FP64 from its formulas (Sedona's constants): LTE Saha-Boltzmann
# populations with charge conservation solved to rounding, electron scattering, free-free,
# bound-free and fuzz-line expansion opacity, and the quantities formed from them.
# A transport step has no such value: its outputs are sums over random walks.
CL, HP, KB, KEV, MP, ME = 2.99792458e10, 6.6260755e-27, 1.380658e-16, 8.6173324e-5, 1.67262158e-24, 9.10938188e-28
PI, THOMSON, SIGMA_TOT, EV_PER_ERG = 3.14159, 0.66523e-24, 0.0265400193567, 624150975230.2815


def exact(case, seed):
    if case["kind"] != "tables":
        return None
    w = _workload(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    D = lambda a: torch.as_tensor(np.asarray(a, dtype=np.float64), device=dev)
    z, atoms = w.zones, w.atoms.atoms
    g = w.nu_grid()
    right = np.asarray(g.right, dtype=np.float64)
    left = np.concatenate([[g.min], right[:-1]])
    nu, dnu = D(0.5 * (left + right)), D(right - left)
    T, rho = D(z.T).clamp(1000.0, 1e8), D(z.rho)
    X = D(z.X)
    A = np.asarray(z.elem_A, dtype=np.float64)
    nz, nn = T.numel(), nu.numel()
    lt = HP * HP / (2.0 * PI * ME * KB * T)
    dens = [rho * X[:, a] / (A[a] * MP) for a in range(len(atoms))]
    boltz, part, lev_ion = [], [], []
    for a in atoms:
        b = torch.exp(-D(a.lev_E)[None, :] / (KEV * T)[:, None]) * D(np.maximum(a.lev_g, 1))[None, :]
        ion = torch.as_tensor(a.lev_ion.astype(np.int64), device=dev)
        part.append(torch.zeros(nz, a.n_ions, dtype=torch.float64, device=dev).index_add_(1, ion, b))
        boltz.append(b)
        lev_ion.append(ion)

    def stages(ne):
        out = []
        for k, a in enumerate(atoms):
            chi = D(a.ion_chi[:-1])
            saha = torch.log(part[k][:, 1:] / part[k][:, :-1]) - chi[None, :] / (KEV * T)[:, None]
            lf = torch.cumsum(saha + (math.log(2.0) - torch.log(ne) - 1.5 * torch.log(lt))[:, None], dim=1)
            lf = torch.cat([torch.zeros(nz, 1, dtype=torch.float64, device=dev), lf], dim=1)
            out.append(torch.softmax(lf, dim=1))
        return out

    def net(ne):
        f = torch.zeros_like(ne)
        for k, fr in enumerate(stages(ne)):
            f = f + dens[k] * (fr * torch.arange(fr.shape[1], device=dev, dtype=torch.float64)).sum(1)
        return f

    n_tot = (rho[:, None] * X / D(A)[None, :]).sum(1) / MP
    lo, hi = torch.log(1e-10 * n_tot), torch.log(100.0 * n_tot)
    for _ in range(200):
        mid = 0.5 * (lo + hi)
        up = net(torch.exp(mid)) > torch.exp(mid)
        lo, hi = torch.where(up, mid, lo), torch.where(up, hi, mid)
    ne = torch.exp(0.5 * (lo + hi))
    frac = stages(ne)
    zeta = HP * nu[None, :] / KB / T[:, None]
    planck = 2.0 * HP * nu[None, :] ** 3 / CL / CL / torch.expm1(zeta)
    eps = float(w.P.scalar("opacity_epsilon"))
    es = (THOMSON * ne)[:, None]
    scat = es.expand(nz, nn).clone()
    ab = 1e-20 * eps * es.expand(nz, nn).clone()
    emis = torch.zeros_like(ab)
    ff = torch.zeros(nz, dtype=torch.float64, device=dev)
    for k in range(len(atoms)):
        q = torch.arange(frac[k].shape[1], device=dev, dtype=torch.float64)
        ff += dens[k] * (frac[k] * q * q).sum(1)
    ff = 3.7e8 * ff * ne / torch.sqrt(T)
    op = ff[:, None] / nu[None, :] ** 3 * (-torch.expm1(-zeta))
    ab += op
    emis += op * planck
    E = HP * nu * EV_PER_ERG
    lam3 = lt ** 1.5
    bf_em = torch.zeros_like(ab)
    for k, a in enumerate(atoms):
        n_lev = frac[k][:, lev_ion[k]] * boltz[k] / part[k][:, lev_ion[k]]
        n_lev = dens[k][:, None] * n_lev.clamp(min=1e-30)
        for q in range(a.lev_ion.size):
            ion = int(a.lev_ion[q])
            if ion == a.n_ions - 1:
                continue
            ic = int(a.ion_ground[ion + 1])
            Eion = float(a.ion_chi[ion]) - float(a.lev_E[q])
            m = (E >= Eion) & (E <= 10.0 * Eion)
            if not bool(m.any()):
                continue
            n_eff = (1 - (float(a.ion_chi[ion]) - Eion) / float(a.ion_chi[ion])) ** -0.5
            x = Eion + np.arange(101) * (9.0 * Eion / 100)
            y = 6.3e-18 * n_eff / (ion + 1) ** 2 * (x / Eion) ** -3.0
            y[100:] = 0.0
            s = torch.zeros(nn, dtype=torch.float64, device=dev)
            s[m] = D(np.interp(E[m].cpu().numpy(), x, y))
            g_ratio = max(float(a.lev_g[q]), 1.0) / max(float(a.lev_g[ic]), 1.0)
            up = (n_lev[:, ic] * g_ratio / 2.0 * lam3)[:, None] * torch.exp((Eion - E)[None, :] / (KEV * T)[:, None])
            ab += s * (n_lev[:, q, None] - up * ne[:, None]).clamp(min=0.0)
            bf_em += 2.0 * HP * nu[None, :] ** 3 / CL / CL * s * up
    emis += bf_em * ne[:, None]
    sums = torch.zeros(nz, nn, dtype=torch.float64, device=dev)
    t = float(z.t_now)
    for k, a in enumerate(atoms):
        keep = (a.fuzz_nu > g.min) & (a.fuzz_nu < right[-1])
        fnu = a.fuzz_nu[keep]
        where = torch.as_tensor(np.searchsorted(right, fnu, side="right"), device=dev)
        ion = torch.as_tensor(a.fuzz_ion[keep].astype(np.int64), device=dev)
        c, El, h = D(SIGMA_TOT * CL / fnu * a.fuzz_gf[keep]), D(a.fuzz_El[keep] / KEV), D(HP * fnu / KB)
        n_ion = dens[k][:, None] * frac[k] / part[k]
        for i in range(0, fnu.size, 50_000):
            j = slice(i, i + 50_000)
            tau = c[j] * t * n_ion[:, ion[j]] * torch.exp(-El[j] / T[:, None]) * -torch.expm1(-h[j] / T[:, None])
            sums.index_add_(1, where[j], -torch.expm1(-tau))
    op = sums * (nu / dnu / CL / t)[None, :]
    ab += eps * op
    scat += (1 - eps) * op
    emis += planck * eps * op
    top = (float(w.P.scalar("opacity_maximum_opacity")) * rho)[:, None]
    scat, ab = torch.minimum(scat, top), torch.minimum(ab, top)
    W = planck * dnu
    ez = torch.exp(zeta)
    Wr = nu[None, :] ** 4 * ez / (ez - 1) ** 2 * dnu
    cdf = torch.cumsum(emis * dnu, dim=1)
    out = {"abs": ab.reshape(-1), "scat": scat.reshape(-1), "emis_cdf": (cdf / cdf[:, -1:]).reshape(-1), "n_elec": ne,
           "eps_imc": torch.ones_like(ne), "planck_mean": (W * ab).sum(1) / W.sum(1),
           "rosseland_mean": Wr.sum(1) / (Wr / (ab + scat)).sum(1), "L_thermal": 4 * PI * cdf[:, -1]}
    return {k: v.cpu().numpy() for k, v in out.items()}
