"""The workloads that the engine's performance is measured on, through its public entry points.

The path of a user's program is the particle-mesh step (CIC deposit, FFT Poisson solve, CIC force
gather with kick and drift), called in four ways: one function at a time on device arrays
(density, potential, integrate), as a whole drop-in step on device or on pinned host arrays, as
whole resident runs (single simulations and mixed ensembles), and the initial conditions that
such runs start from.  Sizes are those of the configurations this repository names (64^3
particles on 128^3 cells, 256^3 on 512^3, 512^3 on 1024^3, ensembles and request streams of 32^3 to
256^3 particles) and generic odd ones; states are early (a = 0.02, Zel'dovich displacements and
the +-2 cell jitter of the initial conditions) or late (clustered).

``listed()`` the cases, ``draw(rng)`` another one of the same ranges, ``prepare(case, seed)`` the inputs
and handles, ``run(state)`` one pass, ``work(case)`` the bytes and operations a pass cannot do
without, ``exact(case, seed)`` the pass in 64 bits with plain torch and numpy.
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.abspath("cosmological-particle-mesh-simulation_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

OM, OL, OK, H0 = 0.3, 0.7, 0.0, 0.7  # the default cosmology of the configuration
DA = 0.00098                          # 1000 steps from a = 0.02 to 1

# supported grid sizes within the measured range
GRIDS = (32, 48, 64, 96, 128, 192, 256, 384, 512, 768)


def listed():
    return [
        # one step of the smallest ensemble member: launches and latency
        {"name": "step-32p-64g", "kind": "step", "n_parts": 32, "n_cells": 64, "box": 100.0, "a": 0.02, "late": False},
        # the CIC deposit alone on a ragged particle count and a radix-3 grid: small diagnostics
        {"name": "density-101377p-96g", "kind": "density", "count": 101377, "n_cells": 96, "a": 0.02, "late": True},
        # the Poisson solve alone with the caller's own Green table, a radix-3 grid
        {"name": "potential-192g-table", "kind": "potential", "n_cells": 192, "a": 0.3, "table": True},
        # kick and drift alone on a clustered state, the reference's own per-function loop
        {"name": "integrate-96p-192g-late", "kind": "integrate", "n_parts": 96, "n_cells": 192, "box": 200.0, "a": 0.5,
         "late": True},
        # an ordinary drop-in step on device arrays, clustered
        {"name": "step-128p-256g-late", "kind": "step", "n_parts": 128, "n_cells": 256, "box": 200.0, "a": 0.5, "late": True},
        # the drop-in step of the headline run
        {"name": "step-256p-512g", "kind": "step", "n_parts": 256, "n_cells": 512, "box": 250.0, "a": 0.02, "late": False},
        # the same through pinned host arrays: what a caller with numpy-side state pays
        {"name": "step_host-256p-512g", "kind": "step_host", "n_parts": 256, "n_cells": 512, "box": 250.0, "a": 0.02,
         "late": False},
        # initial conditions of a mid-size request of the served stream
        {"name": "ics-128p", "kind": "ics", "n_parts": 128, "box": 200.0, "a": 0.02},
        # a resident ensemble of uneven sizes, early and late simulations together
        {"name": "ensemble-24", "kind": "resident", "late": False, "steps": 40, "a": 0.02,
         "parts": "32,48,64,96,128,48,64,32,96,128,64,48,32,96,64,128,48,32,64,96,128,48,64,32"},
        # one mid-size clustered simulation, resident
        {"name": "resident-128p-256g-late", "kind": "resident", "late": True, "steps": 40, "a": 0.5, "parts": "128"},
        # the headline run's steps, resident
        {"name": "resident-256p-512g", "kind": "resident", "late": False, "steps": 25, "a": 0.02, "parts": "256"},
        # the largest single simulation
        {"name": "resident-512p-1024g", "kind": "resident", "late": False, "steps": 7, "a": 0.02, "parts": "512"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("step", "step", "density", "potential", "integrate", "step_host", "ics", "resident", "resident"))
    late = rng.random() < 0.5
    a = round(rng.uniform(0.2, 0.9), 3) if late else round(rng.uniform(0.02, 0.1), 3)
    box = round(rng.uniform(50.0, 500.0), 1)
    if kind in ("step", "integrate", "step_host"):
        n = rng.choice(GRIDS)
        # mostly two cells per particle spacing, sometimes another (odd) lattice
        p = n // 2 if rng.random() < 0.6 else max(8, int(n * rng.uniform(0.3, 0.7)))
        return {"kind": kind, "n_parts": p, "n_cells": n, "box": box, "a": a, "late": late}
    if kind == "density":
        n = rng.choice(GRIDS)
        return {"kind": kind, "count": _log_int(rng, max(1, n ** 3 // 64), n ** 3 // 4), "n_cells": n, "a": a, "late": late}
    if kind == "potential":
        return {"kind": kind, "n_cells": rng.choice(GRIDS), "a": a, "table": rng.random() < 0.3}
    if kind == "ics":
        return {"kind": kind, "n_parts": rng.choice((32, 48, 64, 96, 128, 192, 256)), "box": box, "a": 0.02}
    if rng.random() < 0.5:  # one simulation; an odd lattice now and then
        p = rng.choice((32, 48, 64, 96, 128, 192, 256))
        return {"kind": kind, "late": late, "steps": rng.randint(5, 25), "a": a, "parts": str(p)}
    parts = [rng.choice((32, 48, 64, 96, 128)) for _ in range(rng.randint(3, 24))]
    return {"kind": kind, "late": late, "steps": rng.randint(5, 30), "a": a, "parts": ",".join(map(str, parts))}


# ---- inputs ---------------------------------------------------------------------------------


def _gen(seed, salt):
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1000003 + salt) % (1 << 62))
    return g


def _displacement(m, seed, smooth):
    """Three Gaussian displacement components on an m^3 lattice (m, m, m), unit rms per axis, from a
    cold-dark-matter-like spectrum cut below `smooth` lattice spacings."""
    white = torch.randn((m, m, m), generator=_gen(seed, 1), device="cuda")
    dk = torch.fft.rfftn(white)
    f = torch.fft.fftfreq(m, device="cuda") * (2 * math.pi)
    fx = torch.arange(m // 2 + 1, device="cuda") * (2 * math.pi / m)
    k2 = f[:, None, None] ** 2 + f[None, :, None] ** 2 + fx[None, None, :] ** 2
    k2[0, 0, 0] = 1.0
    k = k2.sqrt()
    dk *= (k ** 0.5 / (1.0 + (k * 6.0) ** 1.8) * torch.exp(-0.5 * k2 * smooth * smooth))
    dk[0, 0, 0] = 0.0
    dk /= k2
    out = []
    for axis in range(3):
        kk = (f[:, None, None], f[None, :, None], fx[None, None, :])[axis]
        out.append(torch.fft.irfftn(dk * (1j * kk), s=(m, m, m)))
    scale = 1.0 / math.sqrt(sum(float(c.square().mean()) for c in out) / 3.0)
    return [c * scale for c in out]


def _f(a):
    """f(a) as the reference's step evaluates it (H0 in the matter slot)."""
    return 1.0 / math.sqrt((H0 + OK * a + OL * a ** 3) / a)


# Particles are kept this many cells off the box faces, so that no coordinate wraps within the
# compared passes: a wrap would turn a rounding into a box length.
MARGIN = 2.5


def _keep_off_faces(x, n):
    m = min(MARGIN, n / 16)
    x = torch.where(x < m, 2 * m - x, x)
    return torch.where(x > n - m, 2 * (n - m) - x, x)


def _halos(x, n, seed):
    """Contracts the particles around one random centre per block of 16 cells (radius up to 8):
    r -> r^2 / R inside R, the cuspy profile of a collapsed halo."""
    nb = max(1, n // 16)
    side = n / nb
    c = torch.rand((nb * nb * nb, 4), generator=_gen(seed, 3), device="cuda")
    b = [(x[d] / side).long().clamp_(0, nb - 1) for d in range(3)]
    at = (b[0] * nb + b[1]) * nb + b[2]
    cc = c[at]
    r2 = torch.zeros_like(x[0])
    off = []
    for d in range(3):
        o = x[d] - (b[d] + 0.5 + 0.3 * (cc[:, d] - 0.5)) * side
        off.append(o)
        r2 += o * o
    big = (0.3 + 0.7 * cc[:, 3]) * (side / 2)
    f = (r2.sqrt() / big).clamp_(max=1.0)
    return [x[d] + off[d] * (f - 1.0) for d in range(3)]


def _particles(n_parts, n_cells, box, a, late, seed):
    """Positions in cells and velocities in code units, (3, n_parts^3) float32, particle order
    of the reference's lattice (the first axis slowest)."""
    # an even lattice for the transform, cut to n_parts
    m = n_parts + (n_parts & 1)
    psi = [c[:n_parts, :n_parts, :n_parts].reshape(-1) for c in _displacement(m, seed, 1.5 if late else 0.5)]
    rms = 6.0 * n_cells / box * a  # one-dimensional rms displacement: about 6 Mpc/h at a = 1
    rms = min(rms, n_cells / 16)
    q = torch.arange(n_parts, device="cuda", dtype=torch.float32) * (n_cells / n_parts) + 0.5
    grid = [q[:, None, None], q[None, :, None], q[None, None, :]]
    x = [(grid[d].expand(n_parts, n_parts, n_parts).reshape(-1) + psi[d] * rms).remainder_(n_cells) for d in range(3)]
    if late:
        x = _halos(x, n_cells, seed)
    else:  # the jitter of the initial conditions
        j = torch.rand((3, n_parts ** 3), generator=_gen(seed, 2), device="cuda")
        x = [(x[d] + (j[d] * 4 - 2)).remainder_(n_cells) for d in range(3)]
    pos = torch.stack([_keep_off_faces(c, n_cells) for c in x]).contiguous()
    vel = torch.stack([c * (rms / a * a * a / _f(a)) for c in psi]).contiguous()
    return pos, vel


def _ragged(case, seed):
    """`count` particles of a lattice state in random order: a caller's own selection."""
    n, count = case["n_cells"], case["count"]
    p = int(math.ceil(count ** (1 / 3)))
    pos, _ = _particles(p, n, 200.0, case["a"], case["late"], seed)
    keep = torch.randperm(p ** 3, generator=_gen(seed, 4), device="cuda")[:count]
    return pos[:, keep].contiguous()


def _density_field(n, seed):
    """A positive density grid with a log-normal distribution, mean about 8 (two cells per
    particle spacing)."""
    d = _displacement(n, seed, 1.0)[0]
    return (8.0 * torch.exp(1.2 * d - 0.72)).contiguous()


def _green_table(n):
    s2 = torch.sin(math.pi * torch.arange(n, device="cuda", dtype=torch.float64) / n) ** 2
    k = s2[:, None, None] + s2[None, :, None] + s2[None, None, :]
    k[0, 0, 0] = 1.0
    g = 1.0 / k
    g[0, 0, 0] = 0.0
    return g


def _phi_field(n, seed, a):
    rk = torch.fft.rfftn(_density_field(n, seed))
    rk *= (-3.0 * OM / 8.0 / a) * _green_table(n)[:, :, : n // 2 + 1].float()
    return torch.fft.irfftn(rk, s=(n, n, n)).contiguous()


def _uniform_pairs(n_parts, seed):
    """Uniform points of the open unit disc (the accepted pairs of the polar method), float32."""
    g = _gen(seed, 5)
    total = n_parts ** 3
    r = torch.sqrt(torch.rand(total, generator=g, device="cuda", dtype=torch.float64) * 0.999998 + 1e-6)
    t = torch.rand(total, generator=g, device="cuda", dtype=torch.float64) * (2 * math.pi)
    return (r * torch.cos(t)).float(), (r * torch.sin(t)).float()


def _sims(case):
    """(n_parts, n_cells, box, a) of each simulation of a resident case."""
    parts = [int(p) for p in case["parts"].split(",")]
    out = []
    for i, p in enumerate(parts):
        a = case["a"]
        if len(parts) > 1 and i % 3 == 2:  # an ensemble holds simulations at different stages
            a = round(0.02 + 0.3 * ((i * 7) % 10) / 10, 3) if not case["late"] else round(case["a"] * 0.5, 3)
        out.append((p, 2 * p, 100.0 + 50.0 * (i % 8) if len(parts) > 1 else 250.0 * (p / 256) ** 0.5, a))
    return out


# ---- the passes -----------------------------------------------------------------------------


def _config(n_parts, n_cells, box, a, steps=1000, seed=0):
    from pmgpu.config import Config
    return Config(n_parts=n_parts, n_cells=n_cells, box_size=box, a_init=a, a_end=a + DA * steps, steps=steps,
                  random_seed=seed)


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind}
    if kind == "resident":
        from pmgpu.batch import Batch
        s["sims"] = []
        for i, (p, n, box, a) in enumerate(_sims(case)):
            pos, vel = _particles(p, n, box, a, case["late"], seed + 7919 * i)
            s["sims"].append((_config(p, n, box, a, case["steps"]), pos, vel))
        s["steps"] = case["steps"]
        s["batch"] = Batch(device=0)
        return s
    if kind == "ics":
        from pmgpu.device_ics import DeviceICs
        p = case["n_parts"]
        s["cfg"] = _config(p, 2 * p, case["box"], case["a"], seed=int(seed) % 100000)
        s["uv"] = _uniform_pairs(p, seed)
        s["ics"] = DeviceICs(p, 0)
        return s
    from pmgpu.context import PMContext
    n = case["n_cells"]
    p = case.get("n_parts", max(1, n // 2))
    cfg = _config(p, n, case.get("box", 200.0), case["a"])
    s["ctx"] = PMContext(cfg, 0)
    s["a"] = case["a"]
    if kind == "density":
        s["pos"] = _ragged(case, seed)
        s["mass"] = n ** 3 / case["count"]
    elif kind == "potential":
        s["rho"] = _density_field(n, seed)
        s["table"] = _green_table(n).float().contiguous() if case["table"] else None
    else:
        s["pos"], s["vel"] = _particles(p, n, case["box"], case["a"], case["late"], seed)
        s["mass"] = cfg.mass
        if kind == "integrate":
            s["phi"] = _phi_field(n, seed, case["a"])
        if kind == "step_host":
            s["pos"], s["vel"] = s["pos"].cpu().pin_memory(), s["vel"].cpu().pin_memory()
    return s


def run(s):
    kind = s["kind"]
    if kind == "step":  # the driver's loop body: the state moves on and so does a
        r = s["ctx"].step(s["pos"], s["vel"], s["mass"], s["a"], DA)
        s["a"] += DA
        return r
    if kind == "step_host":
        r = s["ctx"].step_host(s["pos"], s["vel"], s["mass"], s["a"], DA)
        s["a"] += DA
        return r
    if kind == "density":
        return s["ctx"].density(s["pos"], s["mass"])
    if kind == "potential":
        return s["ctx"].potential(s["rho"], s["table"], s["a"])
    if kind == "integrate":
        r = s["ctx"].integrate(s["pos"], s["vel"], s["a"], _f(s["a"] + DA), DA, s["phi"])
        s["a"] += DA
        return r
    if kind == "ics":
        return s["ics"].generate(s["cfg"], uv=s["uv"], want_grf=True)
    # resident: admit, run to the end, collect, release
    b = s["batch"]
    ids = [b.add(cfg, pos, vel) for cfg, pos, vel in s["sims"]]
    b.step(s["steps"])
    out = [b.get(i, device=True)[:2] for i in ids]
    for i in ids:
        b.remove(i)
    return out


# ---- the bytes and operations a pass cannot do without ---------------------------------------


def _flops_step(np_, n):
    # CIC weights and adds (40), gather, kick and drift (200), two real transforms and the Green multiply
    return 240.0 * np_ + n ** 3 * (5.0 * math.log2(n ** 3) + 3.0)


def work(case):
    kind = case["kind"]
    if kind == "resident":
        b = fl = 0.0
        for p, n, _, _ in _sims(case):
            # every step reads and writes positions and velocities
            b += case["steps"] * 48.0 * p ** 3
            fl += case["steps"] * _flops_step(p ** 3, n)
        return {"bytes": b, "flops": fl}
    if kind == "ics":
        np_ = case["n_parts"] ** 3
        # pairs in; positions, velocities and the field out; five real transforms
        return {"bytes": np_ * (8.0 + 24.0 + 4.0), "flops": np_ * (5 * 2.5 * math.log2(np_) + 150.0)}
    n3 = float(case["n_cells"]) ** 3
    if kind == "density":
        return {"bytes": 12.0 * case["count"] + 4 * n3, "flops": 40.0 * case["count"]}
    if kind == "potential":
        return {"bytes": 8 * n3 + (2 * n3 if case["table"] else 0), "flops": n3 * (5.0 * math.log2(n3) + 3.0)}
    np_ = float(case["n_parts"]) ** 3
    if kind == "integrate":
        return {"bytes": 48 * np_ + 4 * n3, "flops": 200.0 * np_}
    return {"bytes": 48 * np_, "flops": _flops_step(np_, case["n_cells"])}


# ---- the same in 64 bits ----------------------------------------------------------------------


def _cells64(pos, n):
    p = torch.remainder(pos, float(n))
    fl = torch.floor(p)
    return [c % n for c in fl.long()], [c for c in (p - fl)]


def _corner_weight(d, ox, oy, oz):
    return ((d[0] if ox else 1 - d[0]) * (d[1] if oy else 1 - d[1])) * (d[2] if oz else 1 - d[2])


_CORNERS = [(ox, oy, oz) for oz in (0, 1) for oy in (0, 1) for ox in (0, 1)]
_CHUNK = 1 << 24


def _density64(pos, mass, n):
    grid = torch.zeros(n ** 3, dtype=torch.float64, device="cuda")
    for at in range(0, pos.shape[1], _CHUNK):
        c, d = _cells64(pos[:, at:at + _CHUNK].double(), n)
        for ox, oy, oz in _CORNERS:
            i = (((c[2] + oz) % n) * n + (c[1] + oy) % n) * n + (c[0] + ox) % n
            grid.index_add_(0, i, _corner_weight(d, ox, oy, oz) * mass)
    return grid.view(n, n, n)


def _potential64(rho, green, a):
    n = rho.shape[0]
    rk = torch.fft.rfftn(rho)
    rk *= green[:, :, : n // 2 + 1]
    rk *= -3.0 * OM / 8.0 / a
    return torch.fft.irfftn(rk, s=(n, n, n))


def _integrate64(pos, vel, a, f1, da, phi):
    """Kick and drift of float64 positions and velocities, in place."""
    n = phi.shape[0]
    flat = phi.reshape(-1)
    for at in range(0, pos.shape[1], _CHUNK):
        p, v = pos[:, at:at + _CHUNK], vel[:, at:at + _CHUNK]
        c, d = _cells64(p, n)
        for axis in range(3):
            e = [0, 0, 0]
            e[axis] = 1
            g = torch.zeros_like(v[0])
            for ox, oy, oz in _CORNERS:
                lo = (((c[2] + oz - e[2]) % n) * n + (c[1] + oy - e[1]) % n) * n + (c[0] + ox - e[0]) % n
                hi = (((c[2] + oz + e[2]) % n) * n + (c[1] + oy + e[1]) % n) * n + (c[0] + ox + e[0]) % n
                g += _corner_weight(d, ox, oy, oz) * (flat[lo] - flat[hi])
            v[axis] += da * f1 * 0.5 * g
        p += da / (a + da) ** 2 * f1 * v
        p.remainder_(float(n))


def _step64(pos, vel, mass, a, da, n, green):
    phi = _potential64(_density64(pos, mass, n), green, a)
    _integrate64(pos, vel, a, _f(a + da), da, phi)


def _ics64(case, seed):
    p, box, a0 = case["n_parts"], case["box"], case["a"]
    n_cells, total = 2 * p, p ** 3
    u, v = (t.double() for t in _uniform_pairs(p, seed))
    s = u * u + v * v
    t = torch.sqrt(torch.clamp(-2.0 * torch.log(s) / s, min=0.0))
    noise = torch.complex(u * t, v * t).view(p, p, p)
    freq = torch.fft.fftfreq(p, dtype=torch.float64, device="cuda") * p
    m2 = freq[:, None, None] ** 2 + freq[None, :, None] ** 2 + freq[None, None, :] ** 2
    k = 2 * math.pi / box * m2.sqrt()
    q = k / (OM * H0 * math.exp(-0.04 - 0.04 / OM))
    x = torch.where(q > 0, 2.34 * q, torch.ones_like(q))
    tr = (torch.log1p(x) / x) ** 2 / torch.sqrt(1 + 3.89 * q + (16.1 * q) ** 2 + (5.46 * q) ** 3 + (6.71 * q) ** 4)
    shape = torch.where(k > 0, k.clamp(min=1e-30) ** 0.96 * tr, torch.zeros_like(k))
    power = 64.0 * H0 ** 2 * float(total) ** 2 / shape.sum() * shape
    growth = 2.5 / OM / (OM ** (4 / 7) - OL + (1 + OM / 2) * (1 + OL / 70)) * a0
    rho = torch.fft.ifftn(torch.sqrt(power) * growth * noise).real
    rk = torch.fft.fftn(rho)
    res, fres = n_cells / p, n_cells / box
    l = 2 * math.pi * p / box * torch.fft.fftfreq(p, dtype=torch.float64, device="cuda")
    l2 = l[:, None, None] ** 2 + l[None, :, None] ** 2 + l[None, None, :] ** 2
    pot = torch.where(l2 > 0, -rk / torch.where(l2 > 0, l2, torch.ones_like(l2)), torch.zeros_like(rk))
    fa = 1.0 / math.sqrt((OM + OK * a0 + OL * a0 ** 3) / a0)
    h = math.sqrt(H0 ** 2 * (OM / a0 ** 3 + OK / a0 ** 2 + OL))
    jitter = np.random.Generator(np.random.PCG64(int(seed) % 100000))
    lattice = torch.linspace(0, n_cells - res, p, dtype=torch.float64, device="cuda") + 0.5
    pos, vel = [], []
    for axis in range(3):
        shape3 = [1, 1, 1]
        shape3[axis] = p
        disp = torch.fft.ifftn(-1j * l.view(shape3) * pot * res).real.reshape(-1) * fres
        j = torch.from_numpy(jitter.uniform(-2, 2, total)).cuda()
        x0 = lattice.view(shape3).expand(p, p, p).reshape(-1)
        pos.append(torch.remainder(x0 + growth * disp + j, float(n_cells)))
        vel.append(a0 * fa * h * growth * disp)
    return torch.stack(pos), torch.stack(vel), rho


def exact(case, seed):
    kind = case["kind"]
    if kind == "ics":
        pos, vel, grf = _ics64(case, seed)
        return None, vel, grf  # (a position near a face may wrap: displacements come back in the velocities)
    if kind == "resident":
        out = []
        for i, (p, n, box, a) in enumerate(_sims(case)):
            pos, vel = (t.double() for t in _particles(p, n, box, a, case["late"], seed + 7919 * i))
            green, end = _green_table(n), a + DA * case["steps"]
            da = (end - a) / case["steps"]
            while a < end - da:
                _step64(pos, vel, (n / p) ** 3, a, da, n, green)
                a += da
            out.append((pos, vel))
        return out
    n = case["n_cells"]
    if kind == "density":
        return _density64(_ragged(case, seed), n ** 3 / case["count"], n)
    green = _green_table(n)
    if kind == "potential":
        if case["table"]:
            green = green.float().double()
        return _potential64(_density_field(n, seed).double(), green, case["a"])
    pos, vel = (t.double() for t in _particles(case["n_parts"], n, case["box"], case["a"], case["late"], seed))
    if kind == "integrate":
        _integrate64(pos, vel, case["a"], _f(case["a"] + DA), DA, _phi_field(n, seed, case["a"]).double())
    else:
        _step64(pos, vel, (n / case["n_parts"]) ** 3, case["a"], DA, n, green)
    return pos, vel
