"""Performance cases of libttsh: what a user of the TTSH3D timestep has it compute.

A simulation case ("sim") is a batch of droplets that its program advances by `steps` explicit steps
(ttsh_step), optionally with the per-step diagnostics of every droplet (ttsh_reduce_all_async into
page-locked rows), and reads back at a snapshot time: phi, P, u and both pressures of every droplet
(ttsh_get_state into page-locked arrays). A "noalloc" case is ttsh_step_noalloc on the caller's own
device arrays. Snapshots are thousands of steps apart at the reference's defaults (dte / dt = 5000);
`steps` is shorter here, long enough that the steps and not the read-back are most of a pass.

Keys of a case: precision 64 (the library's default) or 32; `sizes`, the droplets' N, comma
separated; k2 (0 the reference's continuous wavenumbers, 1 discrete), quirks (1 the reference's stale
halo), zeta (active stress), init ("noise": the reference program's InitCond 1; "droplet": the seeded
droplet of the batched sweeps), monitor (0 none, 1 the FP64 mass after every step, 2 all diagnostics).
"""
import ctypes
import math
import os
import random
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "bacterial-droplet_gb300"))

import ttsh  # noqa: E402


def _sim(name, precision, sizes, steps, k2=0, quirks=1, zeta=0.0, init="droplet", monitor=0):
    c = {"kind": "sim", "precision": precision, "sizes": ",".join(str(n) for n in sizes), "steps": steps, "k2": k2,
         "quirks": quirks, "zeta": zeta, "init": init, "monitor": monitor}
    return dict(c, name=name) if name else c


def _noalloc(name, n, steps, quirks=1, zeta=0.0):
    c = {"kind": "noalloc", "precision": 64, "sizes": str(n), "steps": steps, "k2": 0, "quirks": quirks, "zeta": zeta,
         "init": "noise"}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest call: one step of a caller that cannot allocate device memory
        _noalloc("noalloc_32", 32, 1),
        # run_cuda.pl's own defaults: one 64^3 droplet, FP64, the reference's noise, no active stress
        _sim("fp64_64", 64, [64], 40, init="noise"),
        # the same at the size of the benchmark
        _sim("fp64_256", 64, [256], 3, init="noise"),
        # forEach.pl's sweep in the default precision on boxes that are no power of two
        _sim("fp64_sweep_4x100", 64, [100] * 4, 6, zeta=0.01),
        # small droplets with all diagnostics (mass, max |D.u|, max |u|) after every step
        _sim("fp64_monitored_8x48", 64, [48] * 8, 20, zeta=0.02, monitor=2),
        # the default box in FP32: one droplet, bound by launches and latency
        _sim("fp32_64", 32, [64], 200, zeta=0.01),
        # the benchmark's line: two 256^3 droplets, the mass of each after every step
        _sim("fp32_2x256", 32, [256] * 2, 40, zeta=0.02, monitor=1),
        # the parameter sweep of 128^3 boxes
        _sim("fp32_sweep_12x128", 32, [128] * 12, 40, zeta=0.01),
        # the uneven batch
        _sim("fp32_mixed_8", 32, [96, 96, 128, 128, 160, 160, 192, 192], 40, zeta=0.03),
        # the large droplet
        _sim("fp32_512", 32, [512], 16, zeta=0.02),
        # boxes that are no multiple of 32: the FP32 step without its tiled form
        _sim("fp32_ragged_4x100", 32, [100] * 4, 20, zeta=0.01),
        # the solenoidal projection (discrete wavenumbers, fresh halo) with all diagnostics every step
        _sim("fp32_discrete_160", 32, [160], 40, k2=1, quirks=0, zeta=0.02, monitor=2),
    ]


# the sizes the library takes (products of 2, 3 and 5), odd ones among them
SMOOTH = sorted(n for n in {2 ** a * 3 ** b * 5 ** c for a in range(10) for b in range(7) for c in range(5)} if 8 <= n <= 512)


def draw(rng: random.Random):
    if rng.random() < 0.12:
        return _noalloc(None, rng.choice([n for n in SMOOTH if n <= 32]), rng.randint(1, 4), rng.randint(0, 1),
                        rng.choice([0.0, 0.02]))
    precision = rng.choice([32, 64])
    lo, hi = (16, 480) if precision == 32 else (16, 240)
    want = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    n = min((m for m in SMOOTH if lo <= m <= hi), key=lambda m: abs(math.log(m / want)))
    if precision == 32 and rng.random() < 0.4:
        n = max(32, n // 32 * 32)  # most FP32 boxes of the configurations are multiples of 32
        while n not in SMOOTH:
            n -= 32
    budget = 2.0e8 if precision == 32 else 2.0e7  # sites x steps of a pass
    most = max(1, min(12, int(budget / 4 / n ** 3)))
    sizes = [n] * rng.randint(1, most)
    if len(sizes) > 2 and rng.random() < 0.4:  # an uneven batch
        other = rng.choice([m for m in SMOOTH if n / 2 <= m <= n])
        sizes[len(sizes) // 2:] = [other] * (len(sizes) - len(sizes) // 2)
    steps = max(2, min(100, int(budget * rng.uniform(0.3, 1.0) / sum(m ** 3 for m in sizes))))
    k2 = 1 if rng.random() < 0.25 else 0
    return _sim(None, precision, sizes, steps, k2, 1 - k2, rng.choice([0.0, 0.005, 0.02]),
                rng.choice(["noise", "droplet"]), rng.choice([0, 0, 1, 2]))


def _sizes(case):
    return [int(n) for n in case["sizes"].split(",")]


def _inputs(case, seed):
    """The host state of each droplet, as torch FP64 arrays made on the GPU: phi, P, u, u*, P* (None: zeros)."""
    out = []
    for i, n in enumerate(_sizes(case)):
        g = torch.Generator(device="cuda").manual_seed(1000 * seed + i)
        x = torch.arange(n, device="cuda", dtype=torch.float64) - n // 2
        r = (x[:, None, None] ** 2 + x[None, :, None] ** 2 + x[None, None, :] ** 2).sqrt()
        if case["init"] == "noise":  # TTSH3D.cu's InitCond 1: a droplet of radius N/4 and noise of amplitude 1e-4
            phi = 0.5 * (1 - torch.tanh((r - n / 4) * 2))
            P, u, us, ps = (1e-4 * (torch.rand((3, n, n, n), generator=g, device="cuda", dtype=torch.float64) - 0.5)
                            for _ in range(4))
        else:  # radius 0.15 .. 0.3 N, interface width 2, random directions inside smoothed by three passes
            radius = n * (0.15 + 0.15 * float(torch.rand((), generator=g, device="cuda")))
            phi = 0.5 * (1 - torch.tanh((r - radius) / 2))
            P = torch.randn((3, n, n, n), generator=g, device="cuda", dtype=torch.float64)
            P *= (phi > 0.5) / P.square().sum(0).sqrt()
            for _ in range(3):
                for b in range(3):
                    P[b] = (P[b] + sum(P[b].roll(s, d) for d in range(3) for s in (-1, 1))) / 7
            P *= phi > 0.5
            u, us, ps = torch.zeros((3, n, n, n), device="cuda", dtype=torch.float64), None, None
        out.append({"phi": phi, "P": P, "u": u, "us": us, "ps": ps})
    return out


def _pinned(*shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=True)


def prepare(case, seed):
    sizes = _sizes(case)
    inps = [ttsh.default_input(Nx=n, Ny=n, Nz=n) for n in sizes]
    exts = [ttsh.default_ext(precision=case["precision"], k2_mode=case["k2"], quirks=case["quirks"], zeta=case["zeta"])
            for _ in sizes]
    made = _inputs(case, seed)
    if case["kind"] == "noalloc":
        n, d = sizes[0], made[0]
        d["pv"], d["pp"] = (torch.zeros((n, n, n), device="cuda", dtype=torch.float64) for _ in range(2))
        return {"case": case, "inp": inps[0], "ext": exts[0], "d": d}
    sim = ttsh.Sim(inps, exts, device=0)
    for i, d in enumerate(made):
        host = {}
        for k, v in d.items():
            host[k] = None if v is None else _pinned(*v.shape).copy_(v).numpy()
        sim.set_state(i, host["phi"], host["P"], host["u"], host["us"], host["ps"])
    outs = [{"phi": _pinned(n, n, n), "P": _pinned(3, n, n, n), "u": _pinned(3, n, n, n), "pv": _pinned(n, n, n),
             "pp": _pinned(n, n, n)} for n in sizes]
    rows = _pinned(case["steps"], sim.partials_size()).numpy() if case["monitor"] else None
    return {"case": case, "sim": sim, "outs": outs, "out": [{k: v.numpy() for k, v in o.items()} for o in outs], "rows": rows}


def run(state):
    case = state["case"]
    if case["kind"] == "noalloc":
        d = state["d"]
        ttsh._check(ttsh.lib().ttsh_step_noalloc(
            ctypes.byref(state["inp"]), ctypes.byref(state["ext"]), case["steps"], d["phi"].data_ptr(), d["P"].data_ptr(),
            d["u"].data_ptr(), d["us"].data_ptr(), d["ps"].data_ptr(), d["pv"].data_ptr(), d["pp"].data_ptr(),
            torch.cuda.current_stream().cuda_stream))
        return d
    sim, rows = state["sim"], state["rows"]
    if rows is None:
        sim.step(case["steps"])
    else:
        for row in rows:
            sim.step(1)
            sim.reduce_all_async(row, mass_only=case["monitor"] == 1)
    for i, o in enumerate(state["out"]):
        ttsh._check(ttsh.lib().ttsh_get_state(sim.handle, i, *(ttsh._p(o[k]) for k in ("phi", "P", "u", "pv", "pp"))))
    out = {"fields": state["out"]}
    if rows is not None:
        stats = [sim.stats_from_partials(row, check=False) for row in rows]
        keys = ("mass", "max_abs_u", "max_div_u") if case["monitor"] == 2 else ("mass",)
        out["stats"] = {k: np.array([[s[k] for s in step] for step in stats]) for k in keys}
    return out


def work(case):
    """Per site and step: phi, P, u read once and written once (14 words), about 550 operations of the
    separable stencils and 5 log2(N) per point for each of the six 1-D transforms; then the nine FP64
    fields written at the end."""
    word = case["precision"] // 8
    b = f = 0
    for n in _sizes(case):
        b += n ** 3 * (14 * word * case["steps"] + 9 * 8)
        f += n ** 3 * case["steps"] * (550 + 30 * math.log2(n))
    return {"bytes": b, "flops": f}


# ---- the step in plain torch, 64 bits ---------------------------------------------------------


def _pad(f, old=None):
    """f with a halo of one site: the periodic image of `old` (default f)."""
    o = f if old is None else old
    for d in range(3):
        n = o.shape[d]
        o = torch.cat([o.narrow(d, n - 1, 1), o, o.narrow(d, 0, 1)], d)
    if old is not None:
        o[1:-1, 1:-1, 1:-1] = f
    return o


def _s(f, d):  # [1, 4, 1] along dimension d
    n = f.shape[d] - 2
    return f.narrow(d, 0, n) + 4 * f.narrow(d, 1, n) + f.narrow(d, 2, n)


def _diff(f, d):  # [-1, 0, 1]
    n = f.shape[d] - 2
    return f.narrow(d, 2, n) - f.narrow(d, 0, n)


def _D(p, axis, h):
    """27-point first derivative along axis (0 = x, the last dimension) of a padded field."""
    for d in range(3):
        p = _diff(p, d) if d == 2 - axis else _s(p, d)
    return p / (72 * h)


def _L(p, h):
    """15-point Laplacian of a padded field."""
    c, m = slice(1, -1), p
    for d in range(3):
        n = m.shape[d] - 2
        m = m.narrow(d, 0, n) + m.narrow(d, 2, n)
    faces = (p[:-2, c, c] + p[2:, c, c] + p[c, :-2, c] + p[c, 2:, c] + p[c, c, :-2] + p[c, c, 2:])
    return (m + 8 * faces - 56 * p[c, c, c]) / (12 * h * h)


def _solve(v, old, case, p):
    """The pressure of provisional field v: the divergence (with the stale halo) over dt, then the
    Poisson solve with the chosen wavenumbers."""
    n, h = v.shape[1], p.h
    F = sum(_D(_pad(v[a], old[a] if case["quirks"] else None), a, h) for a in range(3)) / p.dt0
    k = 2 * math.pi * torch.fft.fftfreq(n, h, dtype=torch.float64, device=v.device)
    if n % 2:  # the reference's wavenumbers turn negative from N / 2 rounded down
        k[n // 2] -= 2 * math.pi / h
    x, y, z = k[None, None, :], k[None, :, None], k[:, None, None]
    if case["k2"] == 0:
        k2 = x * x + y * y + z * z
        k2[0, 0, 0] = 1
        inv = -1 / k2
    else:
        S, C = (k * h).sin() / h, (2 + (k * h).cos()) / 3
        S = {0: S[None, None, :], 1: S[None, :, None], 2: S[:, None, None]}
        C = {0: C[None, None, :], 1: C[None, :, None], 2: C[:, None, None]}
        k2 = (S[0] * C[1] * C[2]) ** 2 + (C[0] * S[1] * C[2]) ** 2 + (C[0] * C[1] * S[2]) ** 2
        null = k2 < 1e-8 / (h * h)
        inv = torch.where(null, torch.zeros_like(k2), -1 / torch.where(null, torch.ones_like(k2), k2))
    return torch.fft.ifftn(torch.fft.fftn(F) * inv).real.contiguous()


def _step(s, case, p):
    h, dt, zeta = p.h, p.dt0, case["zeta"]
    phi, P, u = s["phi"], s["P"], s["u"]
    pp, Pp, up = _pad(phi), [_pad(P[b]) for b in range(3)], [_pad(u[b]) for b in range(3)]
    g = [_D(pp, a, h) for a in range(3)]
    mu0 = 2 * p.aPhi * phi * (1 - phi) * (1 - 2 * phi) - p.kPhi * _L(pp, h)
    P2 = P[0] ** 2 + P[1] ** 2 + P[2] ** 2
    G2 = g[0] ** 2 + g[1] ** 2 + g[2] ** 2
    GP = g[0] * P[0] + g[1] * P[1] + g[2] * P[2]
    us, ps = torch.empty_like(u), torch.empty_like(P)
    for b in range(3):
        dP = [_D(Pp[b], a, h) for a in range(3)]
        r = p.mu * _L(up[b], h) + mu0 * g[b]
        for a in range(3):
            r += _D(_pad(p.cA * phi * dP[a] - zeta * phi * P[a] * P[b]), a, h) - u[a] * _D(up[b], a, h)
        us[b] = u[b] + dt * r
        r = p.eta * _L(_pad(phi * P[b] + p.La ** 2 * _L(Pp[b], h)), h) - p.alpha * phi * P[b] - p.beta * P2 * P[b]
        for a in range(3):
            r -= (u[a] + p.lambda0 * P[a]) * dP[a]
        ps[b] = P[b] + dt * (r - p.A * (G2 * P2 * P[b] + P2.sqrt() * GP * g[b]))
    phi = phi + dt * (p.gamma * _L(_pad(mu0), h) - u[0] * g[0] - u[1] * g[1] - u[2] * g[2])
    pv, pq = _solve(us, s["us"], case, p), _solve(ps, s["ps"], case, p)
    pvp, pqp = _pad(pv), _pad(pq)
    return {"phi": phi, "P": torch.stack([ps[b] - dt * _D(pqp, b, h) for b in range(3)]),
            "u": torch.stack([us[b] - dt * _D(pvp, b, h) for b in range(3)]), "us": us, "ps": ps, "pv": pv, "pp": pq}


def exact(case, seed):
    if case["k2"] == 0 and any(n % 2 for n in _sizes(case)):
        # the reference's wavenumbers are not symmetric for odd N, so the two pressures that the library
        # solves as one complex field mix in the highest mode: no value
        return None
    if sum(n ** 3 for n in _sizes(case)) * case["steps"] > 3e9:
        return None
    fields, mass, umax = [], [], []
    for n, s in zip(_sizes(case), _inputs(case, seed)):
        p = ttsh.default_input(Nx=n, Ny=n, Nz=n)  # the reference's constants
        for k in ("us", "ps"):
            s[k] = torch.zeros_like(s["u"]) if s[k] is None else s[k]
        m, v = [], []
        for _ in range(case["steps"]):
            s = _step(s, case, p)
            m.append(float(s["phi"].sum()) * p.h ** 3)
            v.append(float(s["u"].abs().max()))
        mass.append(m)
        umax.append(v)
        if case["kind"] == "noalloc":
            return s
        fields.append({k: s[k].cpu().numpy() for k in ("phi", "P", "u", "pv", "pp")})
    out = {"fields": fields}
    if case["monitor"]:  # max |D.u| is what rounding leaves of zero: no value
        out["stats"] = {"mass": np.array(mass).T}
        if case["monitor"] == 2:
            out["stats"].update(max_abs_u=np.array(umax).T, max_div_u=None)
    return out
