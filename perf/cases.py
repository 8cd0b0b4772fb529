"""The work a user of this library has it do, as timed cases.

A case is a dict of plain values.  ``listed()`` names twelve of them, ``draw(rng)`` gives
more of the same ranges, ``prepare(case, seed)`` makes the inputs and the handles a
program keeps, ``run(state)`` is one pass through the public entry points and returns its
results, ``work(case)`` the bytes and operations of a pass and ``exact(case, seed)`` the
results in plain 64-bit torch where they have such a form.

Kinds:

* ``step``     particle state on the GPU: put_state, step(k), the state read back
* ``advance``  the same with ADV_PARTICLE_ELLP alone (tracking without collisions)
* ``cycle``    the reference's main loop: ADV_PARTICLE_ELLP and COLLISION called each
               cycle, with the fluid and collision statistics
* ``classes``  several particle classes on one field, stepped together
* ``host``     an ensemble in host memory, one call per step (step_host)
* ``serve``    tracking jobs on resident fields through the serving loop
* ``points``   INTERP_LAG3 of the velocity at given points
* ``fluid``    a live fluid: particles, ADV_FLUID and the coupling each cycle
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from gazpart_b200 import _lib, config
from gazpart_b200.api import FIELD_KEYS, PROP_KEYS, STATE_KEYS, Context
from gazpart_b200.dns import Fluid
from gazpart_b200.serving import Job, serve

TWO_PI = 2.0 * math.pi
DEV = "cuda"


def _spheroids(name, kind, n, grid, precision, steps, ar, b, b_sigma, st, dt):
    """n spheroids of aspect ratios ar (log-uniform), minor semi-axis b (log-normal with
    b_sigma) and Stokes numbers st (uniform) on a grid^3 field in a 2 pi box."""
    c = {"kind": kind, "n": n, "grid": grid, "precision": precision, "steps": steps, "ar_lo": ar[0], "ar_hi": ar[1],
         "b": b, "b_sigma": b_sigma, "st_lo": st[0], "st_hi": st[1], "dt": dt}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest ensemble: 10,000 equal spheroids on a 64^3 field, plain FP64; a
        # study's parameter sweep, where launches and latency are the time
        _spheroids("small_fp64", "step", 10_000, 64, "fp64", 10, (3.0, 3.0), 0.005, 0.0, (1.0, 1.0), 1e-3),
        # 20,000 thick spheroids packed so that thousands of pairs are in contact
        _spheroids("dense_fp64", "step", 20_000, 48, "fp64", 5, (0.4, 3.0), 0.03, 0.0, (1.0, 1.0), 1e-3),
        # a production ensemble: 1e6 prolate spheroids on a 256^3 field, mixed precision
        _spheroids("million_mixed", "step", 1_000_000, 256, "mixed", 5, (1.0, 5.0), 0.002, 0.0, (0.5, 0.5), 5e-4),
        # the same size in plain FP64, polydisperse and with an odd count
        _spheroids("million_fp64", "step", 1_000_003, 256, "fp64", 3, (0.2, 5.0), 0.002, 0.3, (0.1, 10.0), 5e-4),
        # the largest: 512^3 field, 16.8 M polydisperse spheroids, mixed precision
        _spheroids("largest_mixed", "step", 16_777_216, 512, "mixed", 4, (0.2, 5.0), 0.001, 0.3, (0.1, 10.0), 5e-4),
        # one-way tracking without collisions, plain FP64, odd sizes
        _spheroids("advance_fp64", "advance", 777_777, 129, "fp64", 2, (0.2, 5.0), 0.002, 0.3, (0.1, 10.0), 5e-4),
        # the main loop with statistics every cycle
        _spheroids("cycle_stats_mixed", "cycle", 262_144, 128, "mixed", 3, (0.2, 5.0), 0.004, 0.3, (0.1, 10.0), 5e-4),
        # 24 classes from 2,000 to 400,000 particles on one field, one launch for all
        dict(_spheroids("classes_mixed", "classes", 2_000_000, 256, "mixed", 4, (0.2, 5.0), 0.002, 0.0, (0.1, 10.0),
                        5e-4), classes=24),
        # the particles live in (pinned) host memory, one call per time step
        _spheroids("host_mixed", "host", 1_500_000, 256, "mixed", 1, (0.2, 5.0), 0.002, 0.3, (0.1, 10.0), 5e-4),
        # four tracking jobs of different sizes and lengths on two resident fields
        dict(_spheroids("serve_mixed", "serve", 400_000, 128, "mixed", 30, (0.2, 5.0), 0.002, 0.0, (0.1, 10.0), 1e-4),
             jobs=4),
        # the velocity at given points of a plain FP64 field
        {"name": "points_fp64", "kind": "points", "n": 2_000_000, "grid": 256, "precision": "fp64"},
        # particles in a live fluid: each cycle the particles, then the spectral step
        _spheroids("fluid_fp64", "fluid", 100_000, 128, "fp64", 2, (1.0, 3.0), 0.004, 0.0, (0.5, 2.0), 5e-4),
    ]


def draw(rng):
    def logu(lo, hi):
        return math.exp(rng.uniform(math.log(lo), math.log(hi)))

    kind = rng.choice(["step", "step", "step", "step", "advance", "cycle", "classes", "host", "serve", "points",
                       "fluid"])
    prec = rng.choice(["fp64", "mixed"])
    top = {"step": 4e6, "advance": 2e6, "cycle": 1e6, "classes": 2e6, "host": 2e6, "serve": 6e5, "points": 4e6,
           "fluid": 3e5}[kind]
    n = int(logu(5e3, top))
    grid = int(logu(40, 320))
    if kind == "points":
        return {"kind": kind, "n": n, "grid": grid, "precision": prec}
    if kind == "fluid":
        grid = 2 * int(logu(16, 80))
    if kind == "serve":
        grid = min(grid, 160)
    lo = logu(0.2, 3.0)
    ar = (lo, lo * logu(1.0, 5.0 / lo) if rng.random() < 0.8 else lo)
    # solid volume fraction of the ensemble, from dilute to packed (packed when small)
    phi = logu(6e-5, 1.2e-2 if n < 50_000 else 2e-3)
    mean = math.sqrt(ar[0] * ar[1])
    shape = mean if mean >= 1.0 else 1.0 / mean ** 2     # volume over (4/3) pi b^3
    b = (phi * TWO_PI ** 3 / (n * 4.0 / 3.0 * math.pi * shape)) ** (1.0 / 3.0)
    b = min(b, 0.05 / max(ar[1], 1.0 / ar[0]))
    st_lo = logu(0.1, 2.0)
    st = (st_lo, st_lo * logu(1.0, 5.0))
    steps = {"step": rng.randint(1, 6), "advance": rng.randint(1, 3), "cycle": rng.randint(1, 4),
             "classes": rng.randint(1, 4), "host": 1, "serve": rng.randint(5, 30), "fluid": rng.randint(1, 2)}[kind]
    sigma = rng.choice([0.0, 0.3])
    if kind in ("classes", "serve"):
        sigma = 0.0
    c = _spheroids(None, kind, n, grid, prec, steps, ar, b, sigma, st, rng.choice([1e-4, 5e-4, 1e-3]))
    if kind == "classes":
        c["classes"] = rng.randint(2, 40)
    if kind == "serve":
        c["jobs"] = rng.randint(1, 4)
    return c


# ----------------------------------------------------------------------------- inputs
def _gen(seed, k):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 1000 + k)
    return g


def _field(n, period, seed, vorticity=True):
    """A solenoidal random-phase velocity with E(k) ~ k^4 exp(-2 k^2 / k0^2), k0 = 4 (unit
    r.m.s. components), and its spectral vorticity, on n^3 nodes of one period."""
    m = min(20, (n - 1) // 2 - 1)
    g = _gen(seed, 1)
    side = 2 * m + 1
    h = torch.complex(*(torch.randn((3, side, side, m + 1), generator=g, device=DEV, dtype=torch.float64)
                        for _ in range(2)))
    h[..., 0] = (h[..., 0] + h[..., 0].flip(1, 2).conj()) * math.sqrt(0.5)   # real field
    k1 = torch.arange(-m, m + 1, device=DEV, dtype=torch.float64)
    kz, ky, kx = k1.view(-1, 1, 1), k1.view(1, -1, 1), k1[m:].view(1, 1, -1)
    k2 = kx * kx + ky * ky + kz * kz
    k2s = torch.where(k2 > 0, k2, torch.ones_like(k2))
    dot = (kx * h[0] + ky * h[1] + kz * h[2]) / k2s
    h = torch.stack([h[0] - kx * dot, h[1] - ky * dot, h[2] - kz * dot]) * (k2 * torch.exp(-k2 / 16.0)).sqrt()
    h[:, m, m, 0] = 0
    weight = torch.full_like(k2, 2.0)
    weight[..., 0] = 1.0
    h = h / ((weight * h.abs() ** 2).sum() / 3.0).sqrt()
    s = TWO_PI / period
    hats = [h[0], h[1], h[2]]
    if vorticity:
        hats += [1j * s * (ky * h[2] - kz * h[1]), 1j * s * (kz * h[0] - kx * h[2]), 1j * s * (kx * h[1] - ky * h[0])]
    idx = torch.arange(-m, m + 1, device=DEV) % n
    out = {}
    for name, hat in zip(FIELD_KEYS, hats):
        full = torch.zeros((n, n, n // 2 + 1), dtype=torch.complex128, device=DEV)
        full[idx.view(-1, 1, 1), idx.view(1, -1, 1), torch.arange(m + 1, device=DEV).view(1, 1, -1)] = hat
        out[name] = torch.fft.irfftn(full, s=(n, n, n), norm="forward")
        del full
    return out


def _spec(c, **kw):
    ar = dict(ar=c["ar_lo"]) if c["ar_lo"] == c["ar_hi"] else dict(ar_range=(c["ar_lo"], c["ar_hi"]))
    b = dict(b_lognormal=(math.log(c["b"]), c["b_sigma"])) if c["b_sigma"] > 0 else dict(b=c["b"])
    st = dict(st=c["st_lo"]) if c["st_lo"] == c["st_hi"] else dict(st_uniform=(c["st_lo"], c["st_hi"]))
    return config.ParticleSpec(n=c["n"], **ar, **b, **st)


def _setup(c):
    return config.Setup(nx=c["grid"], ny=c["grid"], nz=c["grid"],
                        visc=config.viscosity_for(_spec(c), config.integral_time()), dtime=c["dt"])


def _trilinear(f, keys, dx, xyz):
    """Fluid values at the particles, close enough for an initial state."""
    n = f[keys[0]].shape[0]
    i, w = [], []
    for p in xyz:
        t = p / dx
        k = t.floor().long().clamp_(0, n - 2)
        i.append(k)
        w.append(t - k)
    out = [torch.zeros_like(xyz[0]) for _ in keys]
    for corner in range(8):
        cx, cy, cz = corner & 1, corner >> 1 & 1, corner >> 2
        at = ((i[2] + cz) * n + (i[1] + cy)) * n + (i[0] + cx)
        wt = (w[0] if cx else 1 - w[0]) * (w[1] if cy else 1 - w[1]) * (w[2] if cz else 1 - w[2])
        for o, k in zip(out, keys):
            o += wt * f[k].reshape(-1)[at]
    return out


def _rot_t(q, v):
    """R(q)^T v with the rotation of a unit quaternion q = (a, b, c, d)."""
    a, b, c, d = q
    r = ((1 - 2 * (c * c + d * d), 2 * (b * c - a * d), 2 * (b * d + a * c)),
         (2 * (b * c + a * d), 1 - 2 * (b * b + d * d), 2 * (c * d - a * b)),
         (2 * (b * d - a * c), 2 * (c * d + a * b), 1 - 2 * (b * b + c * c)))
    return [r[0][i] * v[0] + r[1][i] * v[1] + r[2][i] * v[2] for i in range(3)], r


def _particles(c, setup, f, seed, n=None, one_shape=False):
    """Positions uniform in the box (clear of the x planes for the pass's steps),
    orientations uniform on S^3, shapes and Stokes numbers of the case, velocities near
    the fluid's and spins near half its vorticity."""
    n = c["n"] if n is None else n
    g = _gen(seed, 2)

    def rand(k=n):
        return torch.rand(k, generator=g, device=DEV, dtype=torch.float64)

    def randn():
        return torch.randn(n, generator=g, device=DEV, dtype=torch.float64)

    few = 1 if one_shape else n
    ar = torch.exp(math.log(c["ar_lo"]) + rand(few) * math.log(c["ar_hi"] / c["ar_lo"])).expand(n)
    b = c["b"] * torch.exp(c["b_sigma"] * randn()) if c["b_sigma"] > 0 else torch.full((n,), c["b"], device=DEV,
                                                                                     dtype=torch.float64)
    stokes = (c["st_lo"] + rand(few) * (c["st_hi"] - c["st_lo"])).expand(n)
    emaj = torch.where(ar >= 1.0, ar * b, b)
    deq = 2.0 * emaj / ar ** (2.0 / 3.0)
    eb = emaj / ar
    r = torch.maximum(emaj, eb)
    st = {"emaj": emaj, "apr": ar.contiguous(),
          "rhop": stokes * 18.0 * setup.visc * config.integral_time() / (deq * deq),
          "ipxx": (eb * eb + eb * eb) / 5.0, "ipyy": (emaj * emaj + eb * eb) / 5.0,
          "ipzz": (emaj * emaj + eb * eb) / 5.0}
    margin = torch.clamp(r, min=min(TWO_PI / 4, 7.0 * c["dt"] * (c["steps"] + 1))) + r
    st["x"] = margin + rand() * (setup.lx - 2.0 * margin)
    st["y"] = r + rand() * (setup.ly - 2.0 * r)
    st["z"] = r + rand() * (setup.lz - 2.0 * r)
    u1, u2, u3 = rand(), rand(), rand()
    st["qa"], st["qb"] = u1.sqrt() * torch.cos(TWO_PI * u3), (1 - u1).sqrt() * torch.sin(TWO_PI * u2)
    st["qc"], st["qd"] = (1 - u1).sqrt() * torch.cos(TWO_PI * u2), u1.sqrt() * torch.sin(TWO_PI * u3)
    keys = [k for k in FIELD_KEYS if k in f]
    fl = _trilinear(f, keys, setup.dx, [st[k] for k in "xyz"])
    for k, v in zip("uvw", fl):
        st[k] = v + 0.05 * randn()
    if len(keys) == 6:
        spin, _ = _rot_t([st[k] for k in ("qa", "qb", "qc", "qd")], fl[3:])
    else:
        spin = [torch.zeros_like(emaj)] * 3
    for k, v in zip(("ox", "oy", "oz"), spin):
        st[k] = 0.5 * v + 0.1 * randn()
    return {k: v.contiguous() for k, v in st.items()}


def _points(c, setup, seed):
    g = _gen(seed, 3)
    return [torch.rand(c["n"], generator=g, device=DEV, dtype=torch.float64) * setup.lx for _ in range(3)]


def _classes(c, setup, f, seed):
    """Class sizes spread over two decades, one aspect ratio and Stokes number a class."""
    k = c["classes"]
    w = torch.exp(-torch.linspace(0.0, math.log(200.0), k, dtype=torch.float64))
    counts = [max(1000, int(x)) for x in (w / w.sum() * c["n"]).tolist()]
    return [_particles(c, setup, f, seed * 100 + i, n=m, one_shape=True) for i, m in enumerate(counts)]


def _host(st):
    return {k: v.cpu().numpy() for k, v in st.items()}


def _points_setup(c):
    return config.Setup(nx=c["grid"], ny=c["grid"], nz=c["grid"])


def prepare(case, seed):
    c = dict(case)
    kind = c["kind"]
    setup = _points_setup(c) if kind == "points" else _setup(c)
    n = c["grid"]
    s = {"case": c}
    if kind == "fluid":
        f = _field(n, TWO_PI, seed, vorticity=False)
        s["fluid"] = Fluid(setup)
        s["vel"] = [f[k] for k in "uvw"]
        ctx = Context(setup, c["precision"])
        s["fluid"].set_velocity(*s["vel"])
        s["fluid"].couple(ctx, with_vorticity=True)
        s["vel_out"] = [torch.empty_like(v) for v in s["vel"]]
    else:
        # the stencil's index period is n nodes of spacing L / (n - 1)
        f = _field(n, n * setup.dx, seed, vorticity=kind != "points")
        zero = None if kind != "points" else torch.zeros_like(f["u"])
        ctx = Context(setup, c["precision"], store_fluid=kind == "cycle",
                      max_particles=2 * c["n"] if kind == "serve" else 0)
        ctx.set_fields({k: f.get(k, zero) for k in FIELD_KEYS})
    s["ctx"] = ctx
    if kind == "points":
        s["xyz"] = _points(c, setup, seed)
    elif kind == "classes":
        parts = [_host(p) for p in _classes(c, setup, f, seed)]
        ctx.upload_classes(parts)
        s["st"] = {k: torch.from_numpy(np.concatenate([p[k] for p in parts])).to(DEV) for k in STATE_KEYS}
    elif kind == "serve":
        f2 = _field(n, n * setup.dx, seed + 1)
        slot = ctx.add_field(n)
        ctx.set_fields(f2, slot=slot)
        frac = [0.5, 0.3, 0.15, 0.05][: c["jobs"]]
        s["jobs"] = []
        for i, x in enumerate(frac):
            p = _particles(c, setup, f2 if i % 2 else f, seed * 10 + i, n=max(1000, int(c["n"] * x)), one_shape=True)
            s["jobs"].append((_host(p), max(1, c["steps"] * (i + 1) // len(frac)), slot if i % 2 else 0))
    else:
        st = _particles(c, setup, f, seed)
        ctx.upload(st)
        s["st"] = {k: st[k] for k in STATE_KEYS}
        if kind == "host":
            s["in"] = {k: st[k].cpu().pin_memory().numpy() for k in STATE_KEYS}
            s["out"] = {k: torch.empty(c["n"], dtype=torch.float64, pin_memory=True).numpy() for k in STATE_KEYS}
        if kind == "cycle":
            ctx.set_class_groups(1, (np.arange(c["n"]) % 3 + 1).astype(np.int32), 3)
            ctx.enable_collision_stats(True)
    if kind in ("step", "advance", "cycle", "classes", "fluid"):
        s["res"] = {k: torch.empty_like(s["st"][k]) for k in STATE_KEYS}
    del f
    if n >= 200:
        torch.cuda.empty_cache()
    torch.cuda.synchronize()
    return s


# ------------------------------------------------------------------------------- a pass
def _read_state(ctx, out):
    """The state columns into device tensors (gp_download_state, on_device)."""
    cols = (C.c_void_p * 13)(*[C.c_void_p(out[k].data_ptr()) for k in STATE_KEYS])
    _lib.check(_lib.lib().gp_download_state(ctx._h, ctx.n, cols, None, 1), "gp_download_state")
    return out


def run(s):
    c, ctx = s["case"], s["ctx"]
    kind = c["kind"]
    if kind == "points":
        return [ctx.interp_lag3(k, *s["xyz"]) for k in range(3)]
    if kind == "host":
        return ctx.step_host(s["in"], s["out"])
    if kind == "serve":
        jobs = [Job(state=st, steps=k, field=slot) for st, k, slot in s["jobs"]]
        done = serve(ctx, jobs, hbm_budget=100e9)
        return {"particle_steps": done["particle_steps"], "jobs": [j.result for j in jobs]}
    if kind == "fluid":
        # the particles sample the velocity the last coupling left, then the fluid moves on
        fluid = s["fluid"]
        fluid.set_velocity(*s["vel"])
        fluid.couple(ctx, with_vorticity=True)
        ctx.put_state(s["st"])
        for k in range(c["steps"]):
            ctx.adv_particle_ellp(k)
            ctx.collision(k, k * c["dt"])
            fluid.adv_fluid(k)
            fluid.couple(ctx, with_vorticity=True)
        _lib.check(_lib.lib().gp_dns_get_velocity(fluid._h, *(C.c_void_p(v.data_ptr()) for v in s["vel_out"]), 1),
                   "gp_dns_get_velocity")
        return {"velocity": s["vel_out"], "state": _read_state(ctx, s["res"])}
    ctx.put_state(s["st"])
    if kind == "advance":
        for k in range(c["steps"]):
            ctx.adv_particle_ellp(k)
        return _read_state(ctx, s["res"])
    if kind == "cycle":
        counts, stats = [], []
        for k in range(c["steps"]):
            ctx.adv_particle_ellp(k)
            got = ctx.collision(k, k * c["dt"])
            counts.append([got["n_near"], got["n_contact"], got["n_coll"]])
            stats.append(ctx.stat_partfluid(1))
        coll, _ = ctx.collision_stats(1)
        return {"state": _read_state(ctx, s["res"]), "counts": np.array(counts), "stats": np.stack(stats),
                "collisions": coll}
    ctx.step(c["steps"])
    return _read_state(ctx, s["res"])


# ------------------------------------------------------------------- what it cannot avoid
def work(case):
    c = case
    n, elem = c["n"], 8 if c["precision"] == "fp64" else 4
    nodes = c["grid"] ** 3
    if c["kind"] == "points":
        return {"bytes": 3 * (32 * n + elem * min(nodes, 64 * n)), "flops": 3 * n * 2 * (64 + 16 + 4)}
    steps = c["steps"]
    # each step reads the 13 state and 6 property columns and the field, writes the state
    per_step = n * (13 * 8 * 2 + 6 * 8) + 6 * elem * min(nodes, 64 * n)
    flops = n * (6 * 2 * (64 + 16 + 4) + 1500)
    if c["kind"] == "fluid":
        # a spectral step: 21 transforms (each its data in and out once), the state updates
        per_step += 21 * 2 * 8 * nodes + 6 * 8 * nodes
        flops += 21 * 2.5 * nodes * 3 * math.log2(c["grid"])
    return {"bytes": float(steps * per_step), "flops": float(steps * flops)}


# ------------------------------------------------------------------ the same in 64 bits
def _lagrange(comps, ghosts, dx, xyz):
    """Third-order Lagrange interpolation (interp_lag3.f90): nodes (i - 1) dx, index
    period n in x, and in y and z periodic or zero ghost planes per component."""
    n = comps[0].shape[0]
    i, w = [], []
    for p in xyz:
        k = (p / dx).floor()
        a = p / dx - k
        i.append(k.long())
        w.append([-a * (a - 1) * (a - 2) / 6, (a + 1) * (a - 1) * (a - 2) / 2, -(a + 1) * a * (a - 2) / 2,
                  (a + 1) * a * (a - 1) / 6])
    out = [torch.zeros_like(xyz[0]) for _ in comps]
    for kz in range(4):
        z = i[2] + kz - 1
        for ky in range(4):
            y = i[1] + ky - 1
            inside = ((z >= 0) & (z < n) & (y >= 0) & (y < n)).to(torch.float64)
            row = ((z % n) * n + y % n) * n
            wyz = w[2][kz] * w[1][ky]
            for kx in range(4):
                at = row + (i[0] + kx - 1) % n
                for o, f, gh in zip(out, comps, ghosts):
                    v = wyz * w[0][kx] * f.reshape(-1)[at]
                    o += v if gh else v * inside
    return out


def _force_torque(u, un, uf, vort, o, q, deq, pmass_inv, visc):
    """Zastawny et al. drag, lift and torque per unit mass: the force from the slip of u,
    the torque from that of un; the force in the lab frame, the torque in the body's."""
    def slip(vel):
        p, r = _rot_t(q, [a - b for a, b in zip(uf, vel)])
        mag = (p[0] ** 2 + p[1] ** 2 + p[2] ** 2).sqrt()
        perp = (p[1] ** 2 + p[2] ** 2).sqrt()
        phi = torch.atan(perp / p[0]).abs()
        return p, r, mag, perp, mag * deq / visc, torch.sin(phi), torch.cos(phi)

    p, r, mag, perp, re, s, cs = slip(u)
    cd0, cd90 = 18.12 / re ** 1.023 + 4.26 / re ** 0.384, 21.52 / re ** 0.990 + 2.86 / re ** 0.260
    cd = cd0 + (cd90 - cd0) * s ** 1.95
    cl = (0.083 * re ** 0.21 + 1.582 / re ** 0.851) * s ** (1.842 - 0.802 * re ** -0.006) * \
        cs ** (0.874 + 0.009 * re ** 0.570)
    k = 0.125 * math.pi * deq ** 2 * pmass_inv
    lift = k * cl * mag ** 2
    fb = [k * cd * mag * p[0] - lift * s * torch.sign(p[0]), k * cd * mag * p[1] + lift * cs * p[1] / perp,
          k * cd * mag * p[2] + lift * cs * p[2] / perp]
    force = [r[i][0] * fb[0] + r[i][1] * fb[1] + r[i][2] * fb[2] for i in range(3)]
    p, r, mag, perp, re, s, cs = slip(un)
    ct = (0.935 / re ** 0.146 - 0.469 / re ** 0.145) * s ** (0.116 + 0.748 * re ** 0.041) * \
        cs ** (0.221 + 0.657 * re ** 0.044)
    cp = math.pi / 16.0 * deq ** 3 * pmass_inv * ct * mag ** 2 / perp
    curl, _ = _rot_t(q, vort)
    d = [0.5 * a - b for a, b in zip(curl, o)]
    dm = (d[0] ** 2 + d[1] ** 2 + d[2] ** 2).sqrt()
    dp = (d[1] ** 2 + d[2] ** 2).sqrt()
    rr = dm * deq ** 2 / visc
    kr = 0.5 * pmass_inv * (0.5 * deq) ** 5
    c1, c2 = 0.573 * rr ** -0.154 + 116.61 / rr, 1.244 * rr ** 0.239 + 378.12 / rr ** 0.789
    torque = [kr * c1 * d[0].abs() * d[0], kr * c2 * dp * d[1] + cp * p[2].abs() * torch.sign(p[0] * p[2]),
              kr * c2 * dp * d[2] + cp * p[1].abs() * torch.sign(p[0] * p[1])]
    return force, torque


def _turn(q, o, dt):
    """q after a rotation at body-frame spin o for dt."""
    _, r = _rot_t(q, o)
    g = [r[i][0] * o[0] + r[i][1] * o[1] + r[i][2] * o[2] for i in range(3)]
    m = (g[0] ** 2 + g[1] ** 2 + g[2] ** 2).sqrt()
    s, a = torch.sin(m * dt / 2) / m, torch.cos(m * dt / 2)
    b, c, d = (s * x for x in g)
    return [a * q[0] - b * q[1] - c * q[2] - d * q[3], a * q[1] + b * q[0] + c * q[3] - d * q[2],
            a * q[2] - b * q[3] + c * q[0] + d * q[1], a * q[3] + b * q[2] - c * q[1] + d * q[0]]


def _exact_advance(c, seed):
    setup = _setup(c)
    f = _field(c["grid"], c["grid"] * setup.dx, seed)
    st = _particles(c, setup, f, seed)
    comps = [f[k] for k in FIELD_KEYS]
    dt, visc = c["dt"], setup.visc
    deq = 2.0 * st["emaj"] / st["apr"] ** (2.0 / 3.0)
    mi = 1.0 / (st["rhop"] * (4.0 / 3.0) * math.pi * st["emaj"] ** 3 / st["apr"] ** 2)
    ip = [st["ipxx"], st["ipyy"], st["ipzz"]]
    x, u = [st[k] for k in "xyz"], [st[k] for k in "uvw"]
    q, o = [st[k] for k in ("qa", "qb", "qc", "qd")], [st[k] for k in ("ox", "oy", "oz")]

    def spin_rate(t, w):
        return [(t[0] + w[1] * w[2] * (ip[1] - ip[2])) / ip[0], (t[1] + w[2] * w[0] * (ip[2] - ip[0])) / ip[1],
                (t[2] + w[0] * w[1] * (ip[0] - ip[1])) / ip[2]]

    for _ in range(c["steps"]):
        fl = _lagrange(comps, [True] * 3 + [False] * 3, setup.dx, x)
        f1, t1 = _force_torque(u, u, fl[:3], fl[3:], o, q, deq, mi, visc)
        k1o = spin_rate(t1, o)
        u1 = [a + dt * b for a, b in zip(u, f1)]
        o1 = [a + dt * b for a, b in zip(o, k1o)]
        q1 = _turn(q, o1, dt)
        f2, t2 = _force_torque(u1, u, fl[:3], fl[3:], o1, q1, deq, mi, visc)
        k2o = spin_rate(t2, o1)
        x = [a + 0.5 * dt * (b + d) for a, b, d in zip(x, u, u1)]
        u = [a + 0.5 * dt * (b + d) for a, b, d in zip(u, f1, f2)]
        o = [a + 0.5 * dt * (b + d) for a, b, d in zip(o, k1o, k2o)]
        q = _turn(q1, o, dt)
        x = [torch.where(a > setup.lx, a - setup.lx, torch.where(a < 0, a + setup.lx, a)) for a in x]
    return dict(zip(STATE_KEYS, x + u + q + o))


def _exact_fluid(c, seed):
    """ADV_FLUID (adv_fluid.f90): two-stage scheme, integrating factor, projected rotational
    nonlinear term, smooth filter."""
    setup = _setup(c)
    n, dt = c["grid"], c["dt"]
    f = _field(n, TWO_PI, seed, vorticity=False)
    vel = [f[k] for k in "uvw"]
    kf = TWO_PI / setup.lx
    k1 = torch.arange(n, device=DEV, dtype=torch.float64)
    k1 = torch.where(k1 <= n // 2, k1, k1 - n) * kf
    k = [(torch.arange(n // 2 + 1, device=DEV, dtype=torch.float64) * kf).view(1, 1, -1), k1.view(1, -1, 1),
         k1.view(-1, 1, 1)]
    k2 = k[0] ** 2 + k[1] ** 2 + k[2] ** 2
    k2s = torch.where(k2 > 0, k2, torch.full_like(k2, 1e33))
    decay = torch.exp(-setup.visc * k2 * dt)
    klast = math.pi / (setup.lx / n)
    kr = k2.sqrt() / klast
    rt = 8.0 / 9.0
    filt = torch.where(kr <= rt, 1.0, torch.where(kr > 1.0, 0.0, torch.cos(math.pi / 2 * (kr - rt) / (1 - rt)) ** 4))

    def fwd(v):
        return [torch.fft.rfftn(a, norm="forward") for a in v]

    def bwd(h):
        return [torch.fft.irfftn(a, s=(n, n, n), norm="forward") for a in h]

    def project(h):
        div = (k[0] * h[0] + k[1] * h[1] + k[2] * h[2]) / k2s
        return [a - b * div for a, b in zip(h, k)]

    def nonlinear(v, h):
        w = bwd([1j * (k[1] * h[2] - k[2] * h[1]), 1j * (k[2] * h[0] - k[0] * h[2]), 1j * (k[0] * h[1] - k[1] * h[0])])
        r = project(fwd([v[1] * w[2] - v[2] * w[1], v[2] * w[0] - v[0] * w[2], v[0] * w[1] - v[1] * w[0]]))
        # with k = 0 the sums of squares over the guarded k^2 vanish, and with them the mean
        return [torch.where(k2 > 0, a, torch.zeros_like(a)) for a in r]

    for _ in range(c["steps"]):
        h = fwd(vel)
        r = nonlinear(vel, h)
        half = [(a + 0.5 * dt * b) * decay for a, b in zip(h, r)]
        h = [(a + dt * b) * decay for a, b in zip(h, r)]
        vel = bwd(h)
        r = nonlinear(vel, h)
        vel = bwd([a * filt for a in project([a + 0.5 * dt * b for a, b in zip(half, r)])])
    return vel


def exact(case, seed):
    """Trajectories with collisions have no plain form here: which pairs touch, where and
    in what order they are accepted is decided by the contact solver's own iterates."""
    c = dict(case)
    if c["kind"] == "points":
        setup = _points_setup(c)
        f = _field(c["grid"], c["grid"] * setup.dx, seed, vorticity=False)
        return _lagrange([f[k] for k in "uvw"], [True] * 3, setup.dx, _points(c, setup, seed))
    if c["kind"] == "advance":
        return _exact_advance(c, seed)
    if c["kind"] == "fluid":
        return {"velocity": _exact_fluid(c, seed), "state": None}
    return None
