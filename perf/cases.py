"""Timing cases of the framework's public entry points.

A case is a dict of plain values; its "kind" says which path it takes:

  run        positions in, a batch of replicas advanced, positions out (bd_engine_*)
  observe    energy, virial, MSD and F_s of every replica
  correlate  F_s and displacement moments against many waiting-time snapshots
  gder       exact g(r) counts of every replica
  step       one time step through the reference's own entry points (cell_locate, get_forces_*, update_ermak)
  sample     one sample through the reference's own entry points (get_gder, msd, fself_isotropic)
  cv3d       Contracting_Vector3D: statistics of several configurations, then the solve
  train      Adam steps of the surrogate network, loss and parameters out
  gradients  its gradients over one batch
  predict    its outputs for host inputs

Start configurations are dense fluids of the bidisperse mixture made here with plain torch: a small
periodic cell of random points relaxed by descent on the pair energy, repeated, perturbed by thermal
amplitudes, with the particles of each species in random order, as an input file lists them.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from bd_aging_b200 import configs as CF
from bd_aging_b200 import lib as B

DEV = "cuda"
SIG_B, SIG_S = float(CF.SIGMA_BIG), float(CF.SIGMA_SML)


# ------------------------------------------------------------------ cases
def listed():
    return [
        # the smallest system of the batch workloads' conditions, alone: latency of a step
        dict(name="run_small", kind="run", replicas=1, n_min=1000, n_max=1000, phi=0.50, T0=1.0, Tf=1.0, dt=2e-5,
             steps=480, rng="philox", potential="wca_modified", seed=1),
        # one system of the aging quench on its own, as a user without a batch runs it
        dict(name="run_single", kind="run", replicas=1, n_min=32768, n_max=32768, phi=0.58, T0=1.0, Tf=0.1, dt=1e-5,
             steps=192, rng="philox", potential="wca_modified", seed=1),
        # the ragged batch that trains the surrogate: 256 systems of 500 to 8000 particles, odd sizes among them
        dict(name="run_ragged", kind="run", replicas=256, n_min=500, n_max=8000, phi=0.55, T0=1.0, Tf=0.4, dt=1e-5,
             steps=288, rng="philox", potential="wca_modified", seed=7),
        # the aging quench in its batch of 64, the headline workload
        dict(name="run_aging", kind="run", replicas=64, n_min=32768, n_max=32768, phi=0.58, T0=1.0, Tf=0.1, dt=1e-5,
             steps=480, rng="philox", potential="wca_modified", seed=1),
        # a sample step's energies and virial over part of that batch
        dict(name="observe", kind="observe", replicas=8, n_min=32768, n_max=32768, phi=0.58),
        # a sample step's waiting-time correlations, 16 waiting times
        dict(name="correlate", kind="correlate", replicas=16, n_min=32768, n_max=32768, phi=0.58, slots=16, q=6.19),
        # a sample step's g(r) with the reference scripts' 400 bins to r = 15
        dict(name="gder", kind="gder", replicas=8, n_min=32768, n_max=32768, phi=0.58, nbins=400, range=15.0),
        # a caller that keeps the reference's own time loop and arrays
        dict(name="step", kind="step", n_big=16384, n_sml=16384, phi=0.58, T=0.1, dt=1e-5, ntags=16),
        # the sampling part of that loop, odd sizes
        dict(name="sample", kind="sample", n_big=4095, n_sml=4099, phi=0.55, nbins=200, q=7.0),
        # effective-force analysis of a few configurations
        dict(name="cv3d", kind="cv3d", n=4000, configs=4, bins=24, range=3.5, phi=0.50),
        # the surrogate's training at its default shape
        dict(name="train", kind="train", n_in=5, n_out=34, width=256, depth=4, batch=4096, samples=98304, steps=20,
             lr=1e-3),
        # the surrogate's predictions, a ragged number of inputs
        dict(name="predict", kind="predict", n_in=5, n_out=34, width=256, depth=4, batch=4096, samples=10007),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run", "run", "run", "run", "observe", "correlate", "gder", "step", "sample", "cv3d", "train",
                       "gradients", "predict"])
    phi = round(rng.uniform(0.45, 0.60), 3)
    if kind in ("run", "observe", "correlate", "gder"):
        total = _log_int(rng, 500, 800000 if kind == "run" else 250000)
        replicas = rng.choice([r for r in (1, 1, 3, 8, 40, 150) if total // r >= 500])
        n = total // replicas
        c = dict(kind=kind, replicas=replicas, n_min=max(500, n // (rng.choice([1, 3]) if replicas > 1 else 1)),
                 n_max=max(500, n), phi=phi)
    if kind == "run":
        c.update(T0=1.0, Tf=round(rng.uniform(0.05, 1.0), 3), dt=rng.choice([1e-5, 2e-5]),
                 steps=min(rng.randint(90, 480), max(97, 300000000 // total)),
                 rng=rng.choice(["philox"] * 4 + ["curand"]),
                 potential=rng.choice(["wca_modified"] * 5 + ["wca"]), seed=rng.randint(1, 1 << 20))
    elif kind == "correlate":
        c.update(slots=rng.randint(1, 24), q=round(rng.uniform(4.0, 9.0), 2))
    elif kind == "gder":
        c.update(nbins=rng.randint(50, 500), range=round(rng.uniform(2.0, 15.0), 2))
    elif kind == "step":
        n = _log_int(rng, 500, 60000)
        nb = int(n * rng.uniform(0.3, 0.7))
        c = dict(kind=kind, n_big=nb, n_sml=n - nb, phi=phi, T=round(rng.uniform(0.1, 1.0), 2), dt=1e-5, ntags=16)
    elif kind == "sample":
        n = _log_int(rng, 500, 16000)
        nb = int(n * rng.uniform(0.3, 0.7))
        c = dict(kind=kind, n_big=nb, n_sml=n - nb, phi=phi, nbins=rng.randint(100, 400), q=round(rng.uniform(4, 9), 2))
    elif kind == "cv3d":
        c = dict(kind=kind, n=_log_int(rng, 500, 8000), configs=rng.randint(1, 5), bins=rng.randint(12, 28),
                 range=round(rng.uniform(2.5, 3.5), 2), phi=round(rng.uniform(0.45, 0.52), 3))
    elif kind in ("train", "gradients", "predict"):
        c = dict(kind=kind, n_in=rng.choice([3, 5, 5, 8]), n_out=rng.choice([34, 34, 17, 64]),
                 width=rng.choice([128, 192, 256, 256]), depth=rng.randint(2, 5), batch=rng.choice([1024, 2048, 4096]))
        if kind == "train":
            c.update(samples=_log_int(rng, 5000, 100000), steps=rng.randint(5, 30), lr=1e-3)
        elif kind == "predict":
            c.update(samples=_log_int(rng, 100, 50000))
    return c


# ------------------------------------------------------------------ fluids
def _fluids(sizes, phi, seed):
    """Dense fluids, one per (n_big, n_sml) of `sizes`: list of (side, positions [n, 3] in [0, side), big first),
    float32 on the GPU."""
    gen = torch.Generator(device=DEV).manual_seed(int(seed))
    cells, distinct = [], min(len(sizes), 256)
    for nb, ns in sizes:
        k = max(1, math.ceil(((nb + ns) / 512.0) ** (1.0 / 3.0)))
        cb, cs = -(-nb // k ** 3), -(-ns // k ** 3)
        cells.append((k, cb, cs, CF.side_from_phi(cb, cs, phi)))
    n = max(cb + cs for _, cb, cs, _ in cells)
    R = distinct
    side = torch.tensor([c[3] for c in cells[:R]], device=DEV).view(R, 1, 1)
    sig = torch.full((R, n), SIG_S, device=DEV)
    live = torch.zeros((R, n), device=DEV)
    for r, (_, cb, cs, _) in enumerate(cells[:R]):
        sig[r, :cb] = SIG_B
        live[r, :cb + cs] = 1.0
    s_pair = 0.5 * (sig[:, :, None] + sig[:, None, :])
    on = live[:, :, None] * live[:, None, :] * (1.0 - torch.eye(n, device=DEV))
    x = torch.rand((R, n, 3), generator=gen, device=DEV) * side
    for it in range(250):  # descent with capped moves
        inv = torch.zeros_like(s_pair)
        ds = []
        for c in range(3):
            d = x[:, None, :, c] - x[:, :, None, c]
            d -= side * torch.round(d / side)
            ds.append(d)
            inv += d * d
        r2 = torch.clamp(inv, min=0.2)
        s6 = (s_pair * s_pair / r2) ** 3
        g = torch.where(inv < s_pair * s_pair, -12.0 * (s6 * s6 - s6) / r2, torch.zeros_like(r2)) * on
        f = torch.stack([(g * d).sum(2) for d in ds], -1)
        step = f * 2e-3
        cap = 0.08 if it < 120 else 0.02
        step *= torch.clamp(cap / torch.clamp(step.norm(dim=-1, keepdim=True), min=1e-12), max=1.0)
        x = torch.remainder(x + step, side)
    out = []
    for r, (nb, ns) in enumerate(sizes):
        k, cb, cs, a = cells[r]
        box = float(np.float32(k * a))
        base = x[r % R, :cb + cs]
        grid = torch.cartesian_prod(*[torch.arange(k, device=DEV)] * 3).reshape(-1, 3).float() * a
        parts = []
        for lo, hi, want in ((0, cb, nb), (cb, cb + cs, ns)):
            p = (base[lo:hi, None, :] + grid[None]).reshape(-1, 3)
            parts.append(p[torch.randperm(len(p), generator=gen, device=DEV)[:want]])
        p = torch.cat(parts) + 0.03 * torch.randn((nb + ns, 3), generator=gen, device=DEV)
        p = torch.remainder(p + torch.rand(3, generator=gen, device=DEV) * box, box)
        out.append((box, torch.where(p >= box, torch.zeros_like(p), p).contiguous()))
    return out


def _sizes(case):
    """(n_big, n_sml) of every replica: sizes spread evenly over [n_min, n_max] in a fixed shuffled order."""
    R = case["replicas"]
    ns = [case["n_min"] + (case["n_max"] - case["n_min"]) * ((37 * r) % R) // max(1, R - 1) for r in range(R)]
    return [(n - n // 2, n // 2) for n in ns]


def _engine_inputs(case, seed):
    fl = _fluids(_sizes(case), case["phi"], seed)
    pos = torch.cat([p for _, p in fl])
    return [b for b, _ in fl], pos


def _systems(case, sides):
    return [B.System(n_big=nb, n_sml=ns, side=side, sigma_big=SIG_B, sigma_sml=SIG_S, dt=case.get("dt", 1e-5),
                     T0=case.get("T0", 1.0), Tf=case.get("Tf", 0.1), t0=0.0, tf=1e-30, protocol="linear",
                     seed=case.get("seed", 1) * 7919 + r, potential=case.get("potential", "wca_modified"))
            for r, ((nb, ns), side) in enumerate(zip(_sizes(case), sides))]


def _pinned(shape):
    return torch.empty(shape, dtype=torch.float32, pin_memory=True).numpy()


# ------------------------------------------------------------------ networks
def _layers(case):
    w = case["width"]
    return [(w, case["n_in"])] + [(w, w)] * (case["depth"] - 1) + [(case["n_out"], w)]


def _net_inputs(case, seed):
    rng = np.random.default_rng(seed)
    params = np.concatenate([np.concatenate([(rng.uniform(-1, 1, (n, k)) * math.sqrt(1.5 / k)).ravel(),
                                             rng.uniform(-0.1, 0.1, n)]) for n, k in _layers(case)])
    n = case["batch"] if case["kind"] == "gradients" else case["samples"]
    x = rng.uniform(-1.7, 1.7, (n, case["n_in"]))
    y = np.tanh(x @ rng.normal(size=(case["n_in"], case["n_out"]))) + 0.02 * rng.normal(size=(n, case["n_out"]))
    return params.astype(np.float32), x.astype(np.float32), y.astype(np.float32)


# ------------------------------------------------------------------ prepare / run
def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case, kind=kind)
    if kind in ("run", "observe", "correlate", "gder"):
        sides, pos = _engine_inputs(case, seed)
        e = B.Engine(_systems(case, sides), rng=case.get("rng", "philox"))
        s["engine"], s["pos"] = e, _pinned(tuple(pos.shape))
        s["pos"][:] = pos.cpu().numpy()
        if kind == "run":
            s["out"] = _pinned(s["pos"].shape), _pinned(s["pos"].shape)
        else:
            e.set_positions(s["pos"])
        if kind == "correlate":
            e.reserve_snapshots(case["slots"])
            for k in range(case["slots"]):
                e.snapshot(k)
                e.run(4)
            s["slots"] = list(range(case["slots"]))
    elif kind in ("step", "sample"):
        nb, ns = case["n_big"], case["n_sml"]
        side, pos = _fluids([(nb, ns)], case["phi"], seed)[0]
        s["pars"] = p = B.setup_params(side, nb, ns, SIG_B, SIG_S, ntags_big=case.get("ntags", 8),
                                       ntags_sml=case.get("ntags", 8), nbins_gder=case.get("nbins", 200),
                                       dt=case.get("dt", 1e-5), temp0=case.get("T", 1.0))
        s["rr"] = {"b": pos[:nb].clone(), "s": pos[nb:].clone()}
        n_of = {"b": nb, "s": ns}
        if kind == "step":
            s["raw"] = {t: s["rr"][t].clone() for t in "bs"}
            for name, shape in (("ff", 3), ("vir", 1), ("pot", 1)):
                s[name] = {t: torch.zeros((n_of[t], shape), device=DEV) for t in "bs"}
            cells = {"b": p.ncell_big ** 3, "s": p.ncell_sml ** 3}
            s["nocup"] = {t: torch.zeros(cells[t], dtype=torch.int32, device=DEV) for t in "bs"}
            s["cells"] = {t: torch.zeros(cells[t] * case["ntags"], dtype=torch.int32, device=DEV) for t in "bs"}
            s["rng"] = {t: torch.zeros(B.rng_state_size() * n_of[t], dtype=torch.uint8, device=DEV) for t in "bs"}
            for k, t in enumerate("bs"):
                B.setup_rng(s["rng"][t], 1234 + k, n_of[t])
        else:
            s["r0"] = _earlier(case, pos, seed)
            s["now"] = pos
            s["counts"] = torch.zeros((4, case["nbins"]), dtype=torch.int64, device=DEV)
    elif kind == "cv3d":
        s["configs"], s["side"] = _cv3d_inputs(case, seed)
    else:
        params, x, y = _net_inputs(case, seed)
        s["net"] = net = B.Surrogate(n_in=case["n_in"], n_out=case["n_out"], width=case["width"], depth=case["depth"],
                                     batch=case["batch"], seed=5)
        net.set_params(params)
        s["x"], s["y"] = x, y
        if kind == "train":
            net.set_data(x, y)
    return s


def run(s):
    case, kind = s["case"], s["kind"]
    if kind == "run":
        e = s["engine"]
        e.set_positions(s["pos"])
        e.run(case["steps"])
        return e.get_positions(*s["out"])
    if kind == "observe":
        obs = s["engine"].observe()
        return {k: np.array([o[k] for o in obs]) for k in obs[0]}
    if kind == "correlate":
        c = s["engine"].correlate(s["slots"], case["q"])
        return {k: c[k] for k in c.dtype.names}
    if kind == "gder":
        return s["engine"].gder(case["nbins"], case["range"])
    if kind == "step":
        p, rr, ff, vir, pot = s["pars"], s["rr"], s["ff"], s["vir"], s["pot"]
        for t in "bs":
            B.cell_locate(t, rr[t], s["nocup"][t], s["cells"][t], p)
        for t, o in (("b", "s"), ("s", "b")):
            ff[t].zero_()
            vir[t].zero_()
            pot[t].zero_()
            B.get_forces_same(t, rr[t], ff[t], vir[t], pot[t], s["nocup"][t], s["cells"][t], p)
            B.get_forces_diff(t, o, rr[t], ff[t], rr[o], vir[t], pot[t], s["nocup"][o], s["cells"][o], p)
        for t in "bs":
            B.update_ermak(t, rr[t], s["raw"][t], ff[t], s["rng"][t], p)
        return {"ff": ff, "vir": vir, "pot": pot, "rr": rr, "raw": s["raw"], "nocup": s["nocup"], "cells": s["cells"]}
    if kind == "sample":
        p, rr, counts = s["pars"], s["rr"], s["counts"]
        counts.zero_()
        for k, (t, o) in enumerate((("b", "b"), ("b", "s"), ("s", "b"), ("s", "s"))):
            B.get_gder(t, o, rr[t], rr[o], counts[k], p)
        nb = case["n_big"]
        fs = np.zeros(1, np.float32)
        B.fself_isotropic(s["now"][:nb], s["r0"][:nb], nb, fs, 0, case["q"])
        return {"counts": counts, "fself": fs, "msd_big": B.msd(s["now"][:nb], s["r0"][:nb], nb),
                "msd_sml": B.msd(s["now"][nb:], s["r0"][nb:], case["n_sml"])}
    if kind == "cv3d":
        cv = B.Contracting_Vector3D(case["bins"], case["range"])
        for rr, xx in s["configs"]:
            cv.add_statistics(rr, xx, case["n"], s["side"])
        cv.calculate_vector()
        return cv.get_vector()
    net = s["net"]
    if kind == "train":
        loss = net.train(case["steps"], case["lr"])
        return {"loss": loss, "params": net.get_params()}
    if kind == "gradients":
        g, loss = net.gradients(s["x"], s["y"])
        return {"gradients": g, "loss": loss}
    return net.predict(s["x"])


# ------------------------------------------------------------------ work
def work(case):
    kind = case["kind"]
    if kind in ("run", "observe", "correlate", "gder"):
        sizes = _sizes(case)
        P = sum(a + b for a, b in sizes)
    if kind == "run":  # positions in, wrapped and unwrapped positions out; about 10 pairs and one update per step
        return {"bytes": 36.0 * P, "flops": case["steps"] * P * (10 * 30.0 + 150.0)}
    if kind == "observe":
        return {"bytes": 40.0 * P, "flops": P * (10 * 35.0 + 60.0)}
    if kind == "correlate":
        return {"bytes": 24.0 * P * (case["slots"] + 1), "flops": 60.0 * P * case["slots"]}
    if kind == "gder":  # the unordered pairs within range
        pairs = 0.0
        for nb, ns in sizes:
            v = CF.side_from_phi(nb, ns, case["phi"]) ** 3
            pairs += 0.5 * (nb + ns) ** 2 * min(1.0, 4.0 / 3.0 * math.pi * case["range"] ** 3 / v)
        return {"bytes": 12.0 * P + 32.0 * len(sizes) * case["nbins"], "flops": 15.0 * pairs}
    if kind == "step":
        n = case["n_big"] + case["n_sml"]
        return {"bytes": n * (48.0 + 20.0 + 2 * 48.0), "flops": n * (10 * 35.0 + 150.0)}
    if kind == "sample":
        n = case["n_big"] + case["n_sml"]
        return {"bytes": 24.0 * n + 32.0 * case["nbins"], "flops": 0.5 * n * n * 15.0}
    if kind == "cv3d":
        n, b = case["n"], case["bins"]
        return {"bytes": 24.0 * n * case["configs"], "flops": case["configs"] * (8.0 * n * n + 6.0 * n * b * b)}
    fwd = sum(2.0 * n * k for n, k in _layers(case))
    par = sum(n * k + n for n, k in _layers(case))
    io = 4.0 * (case["n_in"] + case["n_out"])
    if kind == "predict":
        return {"bytes": 4.0 * par + io * case["samples"], "flops": fwd * case["samples"]}
    steps = case.get("steps", 1)
    return {"bytes": 8.0 * par + io * case["batch"] * steps, "flops": 3.0 * fwd * case["batch"] * steps}


# ------------------------------------------------------------------ 64-bit values
def _earlier(case, pos, seed):
    """Positions at an earlier time: displacements of a few tenths of a diameter."""
    gen = torch.Generator(device=DEV).manual_seed(int(seed) + 77)
    return pos - 0.2 * torch.randn(pos.shape, generator=gen, device=DEV)


def _cv3d_inputs(case, seed):
    """Configurations and the force on every particle: a smooth repulsion of the neighbours within range, with noise."""
    n = case["n"]
    fl = _fluids([(n - n // 2, n // 2)] * case["configs"], case["phi"], seed)
    side = fl[0][0]
    gen = torch.Generator(device=DEV).manual_seed(int(seed) + 99)
    out = []
    for _, p in fl:
        xx = torch.empty((n, 3), device=DEV)
        for i in range(0, n, 1024):
            d = p[i:i + 1024, None, :] - p[None]
            d -= side * torch.round(d / side)
            r = d.norm(dim=-1)
            f = torch.where((r > 0) & (r < case["range"]), torch.exp(-r), torch.zeros_like(r))
            xx[i:i + 1024] = (f[..., None] * d / torch.clamp(r, min=1e-6)[..., None]).sum(1)
        out.append((p, xx + 0.01 * torch.randn((n, 3), generator=gen, device=DEV)))
    return out, side


def _pairs(x, side, reach):
    """Ordered pairs (i, j) closer than `reach`."""
    ii, jj = [], []
    step = max(1, (1 << 25) // len(x))
    for i in range(0, len(x), step):
        d2 = torch.zeros((min(step, len(x) - i), len(x)), dtype=x.dtype, device=x.device)
        for c in range(3):
            d = x[None, :, c] - x[i:i + step, None, c]
            d -= side * torch.round(d / side)
            d2 += d * d
        a, b = torch.nonzero(d2 < reach * reach, as_tuple=True)
        keep = a + i != b
        ii.append(a[keep] + i)
        jj.append(b[keep])
    return torch.cat(ii), torch.cat(jj)


def _forces(x, sig, side, ii, jj, potential="wca_modified"):
    """Force, energy and virial of every particle."""
    d = x[jj] - x[ii]
    d = d - side * torch.round(d / side)
    r2 = (d * d).sum(1)
    s = 0.5 * (sig[ii] + sig[jj])
    s6 = (s * s / r2) ** 3
    if potential == "wca":
        on = r2 < (1.12246205 * s) ** 2
        g, u = -4.0 * (12.0 * s6 * s6 - 6.0 * s6) / r2, 4.0 * (s6 * s6 - s6) + 1.0
    else:
        on = r2 < s * s
        g, u = -12.0 * (s6 * s6 - s6) / r2, s6 * s6 - 2.0 * s6 + 1.0
    g, u = torch.where(on, g, torch.zeros_like(g)), torch.where(on, u, torch.zeros_like(u))
    z = torch.zeros(len(x), dtype=x.dtype, device=x.device)
    f = torch.zeros_like(x).index_add_(0, ii, g[:, None] * d)
    return f, z.index_add(0, ii, u), z.index_add(0, ii, -0.5 * g * r2)


def _gauss(n, seed, step):
    """Three N(0, 1) values per particle: Philox4x32-10 counted on (particle, step), Box-Muller."""
    m = 0xFFFFFFFF
    c = [torch.arange(n, dtype=torch.int64, device=DEV), torch.full((n,), step & m, dtype=torch.int64, device=DEV),
         torch.full((n,), step >> 32, dtype=torch.int64, device=DEV), torch.zeros(n, dtype=torch.int64, device=DEV)]
    k0, k1 = seed & m, seed >> 32
    for _ in range(10):
        p0, p1 = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57
        c = [((p1 >> 32) & m) ^ c[1] ^ k0, p1 & m, ((p0 >> 32) & m) ^ c[3] ^ k1, p0 & m]
        k0, k1 = (k0 + 0x9E3779B9) & m, (k1 + 0xBB67AE85) & m
    u = [(v >> 9).double() * 2.0 ** -23 + 2.0 ** -24 for v in c]
    r0, r1 = torch.sqrt(-2.0 * torch.log(u[0])), torch.sqrt(-2.0 * torch.log(u[2]))
    return torch.stack([r0 * torch.cos(2 * math.pi * u[1]), r0 * torch.sin(2 * math.pi * u[1]),
                        r1 * torch.cos(2 * math.pi * u[3])], 1)


def _exact_run(case, seed):
    if case["rng"] != "philox" or case["replicas"] > 4 or max(a + b for a, b in _sizes(case)) > 40000:
        return None
    sides, pos = _engine_inputs(case, seed)
    reach = 1.25 * SIG_B + 0.4
    hi, raw, at = [], [], 0
    for r, ((nb, ns), side) in enumerate(zip(_sizes(case), sides)):
        n = nb + ns
        x = pos[at:at + n].double()
        at += n
        sig = torch.cat([torch.full((nb,), SIG_B), torch.full((ns,), SIG_S)]).double().to(DEV)
        mob = 1.0 / sig
        built = None
        for step in range(case["steps"]):
            if built is None or float((x - built).norm(dim=1).max()) > 0.15:
                built = x.clone()
                ii, jj = _pairs(x, side, reach)
            f, _, _ = _forces(x, sig, side, ii, jj, case["potential"])
            T = case["T0"] if step == 0 else case["Tf"]
            amp = torch.sqrt(2.0 * T * mob * case["dt"])
            x = x + f * (mob * case["dt"])[:, None] + amp[:, None] * _gauss(n, case["seed"] * 7919 + r, step)
        raw.append(x.cpu())
        hi.append(torch.remainder(x, side).cpu())
    return [torch.cat(hi), torch.cat(raw)]


def _exact_observe(case, seed):
    sides, pos = _engine_inputs(case, seed)
    out = {k: [] for k in ("energy_big", "energy_sml", "virial", "msd_big", "msd_sml", "fself_big")}
    at = 0
    for (nb, ns), side in zip(_sizes(case), sides):
        x = pos[at:at + nb + ns].double()
        at += nb + ns
        sig = torch.cat([torch.full((nb,), SIG_B), torch.full((ns,), SIG_S)]).double().to(DEV)
        _, u, v = _forces(x, sig, side, *_pairs(x, side, SIG_B))
        vals = (0.5 * float(u[:nb].sum()) / nb, 0.5 * float(u[nb:].sum()) / ns, float(v.sum()), 0.0, 0.0, 1.0)
        for k, val in zip(out, vals):
            out[k].append(val)
    return {**{k: np.array(v) for k, v in out.items()}, "nbr_pairs": None, "temperature": None}


def _exact_step(case, seed):
    nb, ns = case["n_big"], case["n_sml"]
    side, pos = _fluids([(nb, ns)], case["phi"], seed)[0]
    x = pos.double()
    sig = torch.cat([torch.full((nb,), SIG_B), torch.full((ns,), SIG_S)]).double().to(DEV)
    f, u, v = _forces(x, sig, side, *_pairs(x, side, SIG_B))
    two = lambda a: {"b": a[:nb], "s": a[nb:]}  # noqa: E731
    none = {"b": None, "s": None}
    return {"ff": two(f), "vir": two(v[:, None]), "pot": two(u[:, None]), "rr": none, "raw": none, "nocup": none,
            "cells": none}


def _exact_sample(case, seed):
    nb = case["n_big"]
    _, pos = _fluids([(nb, case["n_sml"])], case["phi"], seed)[0]
    d2 = ((pos.double() - _earlier(case, pos, seed).double()) ** 2).sum(1)
    qr = case["q"] * torch.sqrt(d2[:nb])
    return {"counts": None, "fself": (torch.sin(qr) / qr).mean().reshape(1).cpu(), "msd_big": float(d2[:nb].mean()),
            "msd_sml": float(d2[nb:].mean())}


def _exact_cv3d(case, seed):
    configs, side = _cv3d_inputs(case, seed)
    n, bins = case["n"], case["bins"]
    ata = torch.zeros((3, bins, bins), dtype=torch.float64, device=DEV)
    atb = torch.zeros((3, bins), dtype=torch.float64, device=DEV)
    for rr, xx in configs:
        x = rr.double()
        ii, jj = _pairs(x, side, case["range"])
        d = x[ii] - x[jj]
        d = d - side * torch.round(d / side)
        r = d.norm(dim=1)
        at = ii * bins + torch.clamp((r * (bins / case["range"])).long(), max=bins - 1)
        for c in range(3):
            h = torch.zeros(n * bins, dtype=torch.float64, device=DEV).index_add_(0, at, d[:, c] / r).view(n, bins)
            ata[c] += h.T @ h
            atb[c] += h.T @ xx[:, c].double()
    v = torch.zeros(bins, dtype=torch.float64)
    for c in range(3):
        v += torch.linalg.pinv(ata[c].cpu(), rtol=1e-6, hermitian=True) @ atb[c].cpu()
    return v / 3.0


def _mlp(params, case):
    out, at = [], 0
    for n, k in _layers(case):
        w = params[at:at + n * k].reshape(n, k)
        b = params[at + n * k:at + n * k + n]
        at += n * k + n
        out.append((w, b))
    return out


def _forward(params, case, x):
    layers = _mlp(params, case)
    for w, b in layers[:-1]:
        x = torch.nn.functional.gelu(x @ w.T + b)
    return x @ layers[-1][0].T + layers[-1][1]


def _minibatch(step, case):
    """The rows of training step `step`: a counter hash of (seed, step, row) modulo the number of samples."""
    def mix(v):
        v = v + np.uint64(0x9E3779B97F4A7C15)
        v = (v ^ (v >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        v = (v ^ (v >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        return v ^ (v >> np.uint64(31))
    with np.errstate(over="ignore"):
        rows = np.arange(case["batch"], dtype=np.uint64) + np.uint64(step) * np.uint64(1315423911)
        return (mix(np.uint64(5) ^ mix(rows)) % np.uint64(case["samples"])).astype(np.int64)


def _exact_net(case, seed):
    params, x, y = _net_inputs(case, seed)
    p = torch.tensor(params, dtype=torch.float64, device=DEV)
    x, y = torch.tensor(x, dtype=torch.float64, device=DEV), torch.tensor(y, dtype=torch.float64, device=DEV)
    if case["kind"] == "predict":
        return _forward(p, case, x).cpu()

    def loss_and_grad(p, xb, yb):
        p = p.detach().requires_grad_(True)
        loss = ((_forward(p, case, xb) - yb) ** 2).mean()
        return float(loss.detach()), torch.autograd.grad(loss, p)[0]
    if case["kind"] == "gradients":
        loss, g = loss_and_grad(p, x, y)
        return {"gradients": g.cpu(), "loss": loss}
    m, v = torch.zeros_like(p), torch.zeros_like(p)
    for t in range(case["steps"]):
        rows = torch.from_numpy(_minibatch(t, case)).to(DEV)
        loss, g = loss_and_grad(p, x[rows], y[rows])
        m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
        p = p - case["lr"] * (m / (1 - 0.9 ** (t + 1))) / (torch.sqrt(v / (1 - 0.999 ** (t + 1))) + 1e-8)
    return {"loss": loss, "params": p.cpu()}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("gder", "correlate"):  # counts; moments of displacements that no formula gives
        return None
    return {"run": _exact_run, "observe": _exact_observe, "step": _exact_step, "sample": _exact_sample,
            "cv3d": _exact_cv3d}.get(kind, _exact_net)(case, seed)
