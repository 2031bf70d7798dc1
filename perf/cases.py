"""Performance cases: the calls a user of jellyfih_b200 makes, over the sizes they make them at.

Every case goes through the public entry points (Engine, jellyfih_b200.autograd)
and returns what the call gives its caller.  The inputs are tanks from the
package's generator (seeded genomes), the sizes those of the reference's runs
and of this repository's benchmark and tests: 80,000 slots on 128^2, 160,000 on
the 128x256 tall tank, 20,000 on 64^2, 6,000 on 32^2.

Kinds:
  step      an analysis script on a saved tank: its particle fields written,
            a few substeps, the fields read back
  plain     the per-instance launch path: load a tank, run it, rows
  episode   one evaluation of a CMA-ES generation in one call (run_episode):
            host arrays in, rows and fitness out
  generate  the same with the water filled on the GPU (load_robot per instance)
  gradient  the torch.autograd rollout, forward and backward, positions among
            the gradients
  refine    the gradient-refinement step of a search (refine_timing_genes), or,
            in double precision, the gradients themselves (grad_step)
  frame     one 1024^2 viewer frame of the current state, read back

The axisymmetric variant has no case: its substep is unstable as the reference
defines it (infinite within eight substeps), so there is no run of it to time.
The horizon of a run is 128 substeps, two re-sort chunks of the batched path
(64, one chunk, for a few tanks): the water amplifies rounding, so that longer
runs of the same inputs differ among themselves; the cost per substep does not
depend on the horizon.  Fitness, a function of the displacement alone, is asked
for by populations only.
"""
from __future__ import annotations

import math

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

from jellyfih_b200 import Engine, InstanceSpec, autograd, tank

DT = 2e-5
T0 = 0.02  # start time of the gradient rollouts: inside every instance's contraction, before its drop

# Particle-substep cost: x, v, C, F read and written, material read (FP32), and
# the arithmetic of the stencil, G2P, the 2x2 SVD, the stress and P2G.
BYTES, FLOPS = 100.0, 600.0


def listed():
    return [
        # the smallest call: a small tank written, advanced by two substeps and read back (latency)
        dict(name="step 1x6k 32x32", kind="step", m=1, slots=6000, grid=32, tall=False, substeps=2, glow=False),
        # a saved full-size tank resumed for a few substeps and saved again
        dict(name="step 1x80k", kind="step", m=1, slots=80000, grid=128, tall=False, substeps=4, glow=True),
        # one jittered tank on the per-instance launch path
        dict(name="plain 1x80k", kind="plain", m=1, slots=80000, grid=128, tall=False, substeps=64),
        # one jittered tank evaluated alone on the batched path
        dict(name="episode 1x80k", kind="episode", m=1, slots=80000, grid=128, tall=False, substeps=64, spread=False),
        # the reference's default population of 16, tanks generated on the GPU
        dict(name="generate 16x80k", kind="generate", m=16, slots=80000, grid=128, tall=False, substeps=128),
        # the benchmark's batch: 32 instances of 80K slots
        dict(name="episode 32x80k", kind="episode", m=32, slots=80000, grid=128, tall=False, substeps=128, spread=False),
        # a small population on the tall tank
        dict(name="episode 8x160k tall", kind="episode", m=8, slots=160000, grid=128, tall=True, substeps=128,
             spread=False),
        # the uneven batch: 48 square tanks of 40K to 120K particles beside 16 tall ones
        dict(name="episode uneven 48+16", kind="episode", m=64, slots=160000, grid=128, tall=False, substeps=128,
             spread=True),
        # the differentiable rollout of 8 instances through torch.autograd
        dict(name="gradient 8x80k", kind="gradient", m=8, slots=80000, grid=128, substeps=64, every=32),
        # the gradient-refined search step: 256 small tanks
        dict(name="refine 256x20k 64x64", kind="refine", m=256, slots=20000, grid=64, substeps=48, every=24,
             fp64=False),
        # a gradient checked in double precision
        dict(name="refine fp64 2x80k", kind="refine", m=2, slots=80000, grid=128, substeps=48, every=24, fp64=True),
        # one viewer frame of the benchmark's batch
        dict(name="frame 32x80k", kind="frame", m=32, slots=80000, grid=128, tall=False, res=1024),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["step", "plain", "episode", "episode", "generate", "gradient", "refine", "frame"])
    grid = rng.choice([48, 56, 64, 80, 96, 112, 128])
    cells = grid * grid
    slots = int(rng.uniform(3.0, 5.2) * cells)  # the lattice fills about 3.8 slots per cell; fewer cut the water
    most = min(64, 32 * 16384 // cells)
    m = log(8, most) if rng.random() < 0.7 else rng.randint(1, 4)
    run_steps = rng.randint(32, 128) if m >= 8 else rng.randint(32, 64)
    if kind == "step":
        tall = rng.random() < 0.3
        return dict(kind=kind, m=1, slots=slots * (2 if tall else 1), grid=grid, tall=tall,
                    substeps=rng.randint(1, 4), glow=rng.random() < 0.5)
    if kind == "plain":
        return dict(kind=kind, m=min(m, 4), slots=slots, grid=grid, tall=False, substeps=rng.randint(16, 64))
    if kind == "episode":
        tall = rng.random() < 0.3
        spread = not tall and rng.random() < 0.3
        return dict(kind=kind, m=m, slots=slots * (2 if tall or spread else 1), grid=grid, tall=tall,
                    substeps=run_steps, spread=spread)
    if kind == "generate":
        return dict(kind=kind, m=min(m, 32), slots=slots, grid=grid, tall=False, substeps=run_steps)
    if kind == "gradient":
        every = rng.randint(8, 32)
        return dict(kind=kind, m=min(m, 8), slots=slots, grid=grid, substeps=rng.randint(16, 64), every=every)
    if kind == "refine":
        fp64 = rng.random() < 0.3
        return dict(kind=kind, m=min(m, 2) if fp64 else log(8, most), slots=slots, grid=grid, substeps=rng.randint(16, 48),
                    every=rng.randint(8, 24), fp64=fp64)
    return dict(kind=kind, m=min(m, 36), slots=slots, grid=grid, tall=False, res=rng.choice([360, 512, 720, 1024]))


# --- inputs ------------------------------------------------------------------

def _specs(c):
    """The instances' shapes.  `spread`: three of four instances square tanks of uneven particle
    counts, one of four a tall tank."""
    g = c["grid"]
    tall = InstanceSpec(c["slots"], g, 2 * g, 2.0)
    if c.get("spread"):
        n_tall = max(1, c["m"] // 4)
        return [InstanceSpec(c["slots"] * 3 // 4, g, g, 1.0)] * (c["m"] - n_tall) + [tall] * n_tall
    return [tall if c.get("tall") else InstanceSpec(c["slots"], g, g, 1.0)] * c["m"]


def _tanks(c, seed):
    """Per instance: positions, materials, fibres, muscle count, (contraction, frequency), genome."""
    specs = _specs(c)
    rng = np.random.default_rng(seed)
    # a few tanks: jittered by the seed, as the plain method's configuration is; populations: the lattice
    out = []
    for s, g in zip(specs, tank.gaussian_genomes(len(specs), seed)):
        is_tall = s.domain_height > 1.0
        # uneven batches: lattice densities of 1.55 to 2.7 particles per cell side
        div = float(rng.uniform(1.55, 2.7)) if c.get("spread") and not is_tall else 2.0
        pos, mat, fib, st = tank.fill_tank(g, s.n_slots, grid_res=s.n_grid, domain_height=s.domain_height,
                                           spawn_offset=tank.TALL_SPAWN if is_tall else None, spacing_div=div,
                                           jitter=0.25 if c["m"] < 8 else 0.0, seed=seed)
        out.append((pos, mat, fib, st["muscle_count"], tank.timing_params(g), g))
    return specs, out


def _state(spec, tk, seed):
    """A tank in motion: a smooth swirl with its velocity gradient, water under hydrostatic
    pressure, a slightly strained robot, positions off the lattice."""
    pos, mat = tk[0], tk[1]
    rng = np.random.default_rng(seed)
    live = mat >= 0
    h, dx = spec.domain_height, 1.0 / spec.n_grid
    x = pos.astype(np.float64)
    x[live] += rng.uniform(-0.25 * dx, 0.25 * dx, size=(int(live.sum()), 2))
    x[live] = np.clip(x[live], 0.002, [1.0 - 0.002, h - 0.002])
    amp, ph = rng.uniform(0.1, 0.3), rng.uniform(0.0, 1.0)
    a, b = np.pi, np.pi / h
    sx, cx, sy, cy = np.sin(a * x[:, 0]), np.cos(a * x[:, 0]), np.sin(b * x[:, 1]), np.cos(b * x[:, 1])
    # stream function amp sin^2(a x) sin^2(b y): at rest on the walls
    v = np.stack([amp * sx * sx * 2 * b * sy * cy, -amp * 2 * a * sx * cx * sy * sy], -1)
    c00 = amp * 2 * a * sx * cx * 2 * b * sy * cy
    c01 = amp * sx * sx * 2 * b * b * (cy * cy - sy * sy)
    c10 = -amp * 2 * a * a * (cx * cx - sx * sx) * sy * sy
    C = np.stack([np.stack([c00, c01], -1), np.stack([c10, -c00], -1)], -2)
    J = 1.0 - 1e-4 * (h - x[:, 1]) * (1.0 + 0.2 * np.sin(6.0 * (x[:, 0] + ph)))
    F = np.sqrt(J)[:, None, None] * np.eye(2)
    solid = (mat == 1) | (mat == 3)
    F[solid] = np.eye(2) + 0.01 * np.sin(20.0 * x[solid][:, :, None] + 10.0 * ph + np.array([0.0, 1.0]))
    F[mat == 2] = np.eye(2)
    v[~live] = 0.0
    C[~live] = 0.0
    F[~live] = np.eye(2)
    f32 = np.float32
    return dict(x=x.astype(f32), v=v.astype(f32), C=C.astype(f32), F=F.astype(f32),
                glow=np.zeros(len(mat), f32), Jp=np.ones(len(mat), f32))


def _grid(spec, seed):
    """A grid velocity field with vortices, and its mass."""
    rng = np.random.default_rng(seed)
    i, j = np.meshgrid(np.arange(spec.n_grid) / spec.n_grid, np.arange(spec.n_grid_y) / spec.n_grid, indexing="ij")
    p = rng.uniform(0, 2 * np.pi, 4)
    gv = 0.2 * np.stack([np.sin(9 * i + p[0]) * np.cos(14 * j + p[1]), np.cos(11 * i + p[2]) * np.sin(8 * j + p[3])], -1)
    return gv.astype(np.float32), np.full(gv.shape[:2], 6e-5, np.float32)


def _set_timing(e, tanks):
    e.set_params(contraction=[t[4][0] for t in tanks], freq=[t[4][1] for t in tanks])


def prepare(case, seed):
    c, kind = case, case["kind"]
    s = {"case": c}
    specs, tanks = _tanks(c, seed)
    if kind == "step":
        e = Engine(specs, glow=c["glow"])
        _set_timing(e, tanks)
        for m, tk in enumerate(tanks):
            e.load(m, *tk[:3])
        s["states"] = [_state(specs[m], tk, seed + m) for m, tk in enumerate(tanks)]
    elif kind == "plain":
        e = Engine(specs, path="plain")
        _set_timing(e, tanks)
        s["tanks"] = [t[:3] for t in tanks]
    elif kind == "episode":
        e = Engine(specs)
        s["pos"], s["mat"], s["fib"] = (np.concatenate([t[k] for t in tanks]) for k in (0, 1, 2))
        s["con"] = np.array([t[4][0] for t in tanks], np.float32)
        s["freq"] = np.array([t[4][1] for t in tanks], np.float32)
        s["muscle"] = np.array([t[3] for t in tanks], np.int32) if c["m"] >= 8 else None
    elif kind == "generate":
        e = Engine(specs)
        s["timing"] = ([t[4][0] for t in tanks], [t[4][1] for t in tanks])
        s["robots"] = [tank.generate_phenotype(t[5], tank.DEFAULT_SPAWN, grid_res=c["grid"])[:3] for t in tanks]
        s["muscle"] = np.array([t[3] for t in tanks], np.int32) if c["m"] >= 8 else None
    elif kind == "gradient":
        e = Engine(specs)
        dev = torch.device("cuda")
        s["params"] = [torch.tensor(v, dtype=torch.float32, device=dev, requires_grad=True) for v in (
            [500.0] * c["m"], [t[4][0] for t in tanks], [t[4][1] for t in tanks])]
        s["pos"] = torch.tensor(np.stack([t[0] for t in tanks]), device=dev, requires_grad=True)
        s["mats"], s["fibs"] = [t[1] for t in tanks], [t[2] for t in tanks]
    elif kind == "refine":
        e = Engine(specs, grad_fp64=c["fp64"])
        _set_timing(e, tanks)
        s["tanks"] = [t[:3] for t in tanks]
        s["genomes"] = np.stack([t[5] for t in tanks])
    else:  # frame
        e = Engine(specs)
        _set_timing(e, tanks)
        for m, tk in enumerate(tanks):
            e.load(m, *tk[:3])
            st = _state(specs[m], tk, seed + m)
            e.write(m, x=st["x"], v=st["v"])
            e.write_grid(m, *_grid(specs[m], seed + m))
        e.time = T0
        e.frame_create(c["res"])
        rng = np.random.default_rng(seed)
        s["hue"], s["mhue"] = (rng.uniform(0, 1, c["m"]).astype(np.float32) for _ in range(2))
    s["engine"] = e
    return s


def run(s):
    c, e = s["case"], s["engine"]
    kind = c["kind"]
    if kind == "step":
        for m, st in enumerate(s["states"]):
            e.write(m, **st)
        e.time = T0
        e.step(c["substeps"])
        return [e.read(m) for m in range(c["m"])]
    if kind == "plain":
        for m, t in enumerate(s["tanks"]):
            e.load(m, *t)
        return e.run_headless(c["substeps"])
    if kind == "episode":
        return e.run_episode(s["pos"], s["mat"], s["con"], c["substeps"], fibers=s["fib"], freq=s["freq"],
                             muscle_counts=s["muscle"])
    if kind == "generate":
        counts = [e.load_robot(m, *r) for m, r in enumerate(s["robots"])]
        e.set_params(contraction=s["timing"][0], freq=s["timing"][1])
        rows = e.run_headless(c["substeps"])
        return counts, rows, None if s["muscle"] is None else e.fitness(rows, s["muscle"], s["timing"][0])
    if kind == "gradient":
        for p in (*s["params"], s["pos"]):
            p.grad = None
        loss = autograd.rollout_displacement(e, *s["params"], s["pos"], s["mats"], s["fibs"], c["substeps"],
                                             checkpoint_every=c["every"], t0=T0)
        loss.sum().backward()
        return loss, [p.grad for p in s["params"]], s["pos"].grad
    if kind == "refine" and not c["fp64"]:
        pos, mats, fibs = zip(*s["tanks"])
        return autograd.refine_timing_genes(e, s["genomes"], pos, mats, fibs, c["substeps"], iterations=1,
                                            checkpoint_every=c["every"])
    if kind == "refine":
        for m, t in enumerate(s["tanks"]):
            e.load(m, *t)
        e.time = T0
        loss, g = e.grad_step(c["substeps"], c["every"])
        return loss, g
    # frame: the viewers' pipeline
    side = int(math.ceil(math.sqrt(c["m"])))
    sub = c["res"] // side
    e.frame_clear(0.0)
    e.render_abyss(sub, side, 1.5, s["hue"], s["mhue"], 2)
    e.render_vorticity_overlay(sub, side, 0.02)
    e.tone_map()
    e.compute_vorticity(0.05)
    e.render_vorticity(sub, side, 0.6, 0)
    return e.read_frame()


def work(case):
    """Bytes and operations one pass cannot do without.  A substep reads and writes every live
    particle's state once; a backward substep reads the state and its adjoint and writes the
    adjoint, at about three times the arithmetic."""
    c, kind = case, case["kind"]
    slots = sum(s.n_slots for s in _specs(c))
    # the lattice fills the tank but its margins; the slots may cut it
    live = sum(min(s.n_slots, 3.8 * s.n_grid * s.n_grid_y) for s in _specs(c))
    n = c.get("substeps", 0)
    wide = 2.0 if c.get("fp64") else 1.0
    if kind == "step":
        return {"bytes": BYTES * live * n + 128.0 * slots, "flops": FLOPS * live * n}
    if kind in ("plain", "episode"):
        return {"bytes": BYTES * live * n + 20.0 * slots, "flops": FLOPS * live * n}
    if kind == "generate":
        return {"bytes": BYTES * live * n + 16.0 * live, "flops": FLOPS * live * n}
    if kind in ("gradient", "refine"):
        return {"bytes": wide * (BYTES + 152.0) * live * n + 28.0 * slots, "flops": 4 * FLOPS * live * n}
    px = float(c["res"]) ** 2
    return {"bytes": 24.0 * live + 12.0 * px, "flops": 60.0 * live + 100.0 * px}


# --- the same in 64 bits, in plain torch --------------------------------------

def _lame(E, nu):
    return E / (2 * (1 + nu)), E * nu / ((1 + nu) * (1 - 2 * nu))


def _svd(A):
    """Rotation (c, s) of the polar decomposition, the Jacobi rotation (cc, ss) of the symmetric
    factor (none while its off-diagonal is below 1e-5) and the singular values."""
    a, b, d, f = A[:, 0, 0], A[:, 0, 1], A[:, 1, 0], A[:, 1, 1]
    x, y = a + f, d - b
    r = torch.sqrt(x * x + y * y)
    c, s = x / r, y / r
    p, q, w = c * a + s * d, c * b + s * f, c * f - s * b
    flat = q.abs() < 1e-5
    one, zero = torch.ones_like(q), torch.zeros_like(q)
    qs = torch.where(flat, one, q)
    half = 0.5 * (p - w)
    root = torch.sqrt(half * half + qs * qs)
    t = torch.where(flat, zero, qs / torch.where(half > 0, half + root, half - root))
    cc = 1.0 / torch.sqrt(t * t + 1.0)
    ss = -t * cc
    s1 = torch.where(flat, p, cc * cc * p - 2 * cc * ss * q + ss * ss * w)
    s2 = torch.where(flat, w, ss * ss * p + 2 * cc * ss * q + cc * cc * w)
    return c, s, cc, ss, s1, s2


def _mat(a, b, c, d):
    return torch.stack([torch.stack([a, b], -1), torch.stack([c, d], -1)], -2)


def _substep(x, v, C, F, k, act, con, freq, t):
    """One substep of all particles (live ones, of instances that share a grid shape) in 64 bits."""
    nx, ny, mat, inst = k["nx"], k["ny"], k["mat"], k["inst"]
    N, dx = x.shape[0], 1.0 / nx
    vol = (dx * 0.5) ** 2
    base = torch.trunc(x.detach() * nx - 0.5).long()
    inr = (base[:, 0] >= 0) & (base[:, 1] >= 0) & (base[:, 0] < nx - 2) & (base[:, 1] < ny - 2)
    fx = x * nx - base
    w = [0.5 * (1.5 - fx) ** 2, 0.75 - (fx - 1) ** 2, 0.5 * (fx - 0.5) ** 2]
    eye = torch.eye(2, dtype=x.dtype, device=x.device)
    Fs = (eye + DT * C) @ F
    c, s, cc, ss, s1, s2 = _svd(Fs)
    s1, s2 = s1.clamp(min=1e-6), s2.clamp(min=1e-6)
    water, pay, musc = mat == 0, mat == 2, mat == 3
    n1 = torch.where(pay, s1.clamp(0.995, 1.005), s1)
    n2 = torch.where(pay, s2.clamp(0.995, 1.005), s2)
    J = n1 * n2
    R, V = _mat(c, -s, s, c), _mat(cc, ss, -ss, cc)
    Fp = R @ V @ torch.diag_embed(torch.stack([n1, n2], -1)) @ V.transpose(1, 2)
    sj = torch.sqrt(J)[:, None, None] * eye
    Fn = torch.where(water[:, None, None], sj, torch.where(pay[:, None, None], Fp, Fs))
    tau = (2 * k["mu"])[:, None, None] * (Fn - R) @ Fn.transpose(1, 2) + (k["la"] * J * (J - 1))[:, None, None] * eye
    period = 1.0 / freq
    phase = (t - period * torch.floor(t / period).detach()) / period
    wave = torch.where(phase < con, 0.5 * (1.0 - torch.cos(phase / con * 3.14159265)), torch.zeros_like(phase))
    fib = k["fib"]
    tau = tau + (musc * (act * wave)[inst] * J)[:, None, None] * fib[:, :, None] * fib[:, None, :]
    mass = torch.where(pay, 2.5 * vol, vol).to(x.dtype)
    A = -DT * vol * 4 * nx * nx * tau + mass[:, None, None] * C
    row0 = inst * ny
    rows = k["n_inst"] * ny
    gp = torch.zeros((rows * nx, 3), dtype=x.dtype, device=x.device)
    keep = inr.to(x.dtype)
    nodes = []
    for i in range(3):
        for j in range(3):
            o = torch.tensor([i, j], dtype=x.dtype, device=x.device)
            wt = w[i][:, 0] * w[j][:, 1] * keep
            mom = wt[:, None] * (mass[:, None] * v + (A @ ((o - fx) * dx)[:, :, None])[:, :, 0])
            node = ((row0 + (base[:, 1] + j).clamp(0, ny - 1)) * nx + (base[:, 0] + i).clamp(0, nx - 1))
            gp = gp.index_add(0, node, torch.cat([mom, (wt * mass)[:, None]], 1))
            nodes.append((i, j, o, node))
    gm = gp[:, 2]
    has = gm > 0
    n = torch.arange(rows * nx, device=x.device)
    gi, gj = (n % nx).to(x.dtype), ((n // nx) % ny).to(x.dtype)
    damp = torch.ones_like(gm)
    for g, size in ((gi, nx), (gj, ny)):
        d = size // 20
        damp = torch.where(g < d, damp * (0.95 + 0.05 * g / max(d, 1)), damp)
        damp = torch.where(g > size - d, damp * (0.95 + 0.05 * (size - g) / max(d, 1)), damp)
    u = gp[:, :2] / torch.where(has, gm, torch.ones_like(gm))[:, None] * damp[:, None]
    z = torch.zeros_like(gm)
    ux = torch.where(((gi < 3) & (u[:, 0] < 0)) | ((gi > nx - 3) & (u[:, 0] > 0)), z, u[:, 0])
    uy = torch.where(((gj < 3) & (u[:, 1] < 0)) | ((gj > ny - 3) & (u[:, 1] > 0)), z, u[:, 1])
    u = torch.where(has[:, None], torch.stack([ux, uy], -1), gp[:, :2])
    nv, nC = torch.zeros_like(v), torch.zeros_like(C)
    for i, j, o, node in nodes:
        g = u[node]
        wt = w[i][:, 0] * w[j][:, 1]
        nv = nv + wt[:, None] * g
        nC = nC + (4 * nx * wt)[:, None, None] * g[:, :, None] * (o - fx)[:, None, :]
    v = torch.where(inr[:, None], nv, v) - torch.tensor([0.0, DT * 10.0], dtype=x.dtype, device=x.device)
    C = torch.where(inr[:, None, None], nC, C)
    F = torch.where(inr[:, None, None], Fn, F)
    x = x + DT * v
    x = torch.stack([x[:, 0].clamp(0.001, 0.999), x[:, 1].clamp(0.001, k["h"] - 0.001)], -1)
    ratio = torch.where(pay & inr, (s1 / n1) * (s2 / n2), torch.ones_like(J))
    return x, v, C, F, ratio


def _consts(spec, mats, fibs, n_inst):
    """What _substep needs of the live particles of instances that share a grid shape."""
    dev = torch.device("cuda")
    live = [m >= 0 for m in mats]
    mat = torch.tensor(np.concatenate([m[k] for m, k in zip(mats, live)]).astype(np.int64), device=dev)
    fib = torch.tensor(np.concatenate([f[k] for f, k in zip(fibs, live)]).astype(np.float64), device=dev)
    inst = torch.tensor(np.concatenate([np.full(int(k.sum()), i) for i, k in enumerate(live)]), device=dev)
    E = {0: (0.0, 1e5), 1: _lame(700.0, 0.3), 2: _lame(2e5, 0.2), 3: _lame(700.0, 0.3)}
    mu = torch.tensor([E[q][0] for q in range(4)], dtype=torch.float64, device=dev)[mat]
    la = torch.tensor([E[q][1] for q in range(4)], dtype=torch.float64, device=dev)[mat]
    return dict(nx=spec.n_grid, ny=spec.n_grid_y, h=spec.domain_height, mat=mat, fib=fib, inst=inst, mu=mu, la=la,
                n_inst=n_inst), live


def _com(x, k):
    """Centre of mass (y, x) of each instance's payload, else of its jelly and muscle."""
    pay = (k["mat"] == 2).to(x.dtype)
    body = ((k["mat"] == 1) | (k["mat"] == 3)).to(x.dtype)
    zero = torch.zeros(k["n_inst"], dtype=x.dtype, device=x.device)
    n_pay = zero.index_add(0, k["inst"], pay)
    sel = torch.where(n_pay[k["inst"]] > 0, pay, body)
    cnt = zero.index_add(0, k["inst"], sel).clamp(min=1.0)
    return [zero.index_add(0, k["inst"], sel * x[:, a]) / cnt for a in (1, 0)]


def _from_rest(pos, live):
    x = torch.tensor(np.concatenate([p[k] for p, k in zip(pos, live)]).astype(np.float64), device="cuda")
    v = torch.zeros_like(x)
    C = torch.zeros((len(x), 2, 2), dtype=x.dtype, device=x.device)
    return x, v, C, torch.eye(2, dtype=x.dtype, device=x.device).repeat(len(x), 1, 1)


def _timing(tanks, n):
    dev = torch.device("cuda")
    f = lambda a: torch.tensor(np.asarray(a, np.float32).astype(np.float64), device=dev)  # noqa: E731
    return f([500.0] * n), f([t[4][0] for t in tanks]), f([t[4][1] for t in tanks])


def _exact_rows(c, seed):
    specs, tanks = _tanks(c, seed)
    rows = np.zeros((len(specs), 5))
    for spec in dict.fromkeys(specs):
        which = [m for m, s in enumerate(specs) if s == spec]
        sub = [tanks[m] for m in which]
        k, live = _consts(spec, [t[1] for t in sub], [t[2] for t in sub], len(sub))
        x, v, C, F = _from_rest([t[0] for t in sub], live)
        act, con, freq = _timing(sub, len(sub))
        y0, x0 = _com(x, k)
        with torch.no_grad():
            for n in range(c["substeps"]):
                x, v, C, F, _ = _substep(x, v, C, F, k, act, con, freq, n * DT)
        y1, x1 = _com(x, k)
        rows[which] = torch.stack([y0, x0, y1, x1, (y1 >= 0.01).to(y1.dtype)], 1).cpu().numpy()
    if c["m"] < 8:
        return rows, None
    fit = np.full(len(specs), np.nan)
    for m, s in enumerate(specs):
        if rows[m, 4] and tanks[m][3] >= 200:
            disp = min(rows[m, 2], s.domain_height - 0.07) - rows[m, 0]
            fit[m] = -disp / math.sqrt(tanks[m][3] * min(max(tanks[m][4][0], 0.05), 0.60) / 500.0)
    worst = np.nanmax(fit) + 1.0 if np.isfinite(fit).any() else 100.0
    return rows, np.where(np.isnan(fit), worst, fit)


def _exact_gradient(c, seed, t0):
    specs, tanks = _tanks(c, seed)
    M = len(specs)
    k, live = _consts(specs[0], [t[1] for t in tanks], [t[2] for t in tanks], M)
    x, v, C, F = _from_rest([t[0] for t in tanks], live)
    start = x.clone().requires_grad_(True)
    params = [p.requires_grad_(True) for p in _timing(tanks, M)]
    x, y0 = start, _com(start, k)[0]
    for n in range(c["substeps"]):
        x, v, C, F, _ = checkpoint(_substep, x, v, C, F, k, *params, t0 + n * DT, use_reentrant=False)
    loss = _com(x, k)[0] - y0
    loss.sum().backward()
    dpos = torch.zeros((M, specs[0].n_slots, 2), dtype=torch.float64, device="cuda")
    dpos[torch.tensor(np.stack(live), device="cuda")] = start.grad
    return loss.detach(), [p.grad for p in params], dpos


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "frame":
        return None  # which pixels a particle covers is decided by 32-bit comparisons
    if kind in ("gradient", "refine"):
        steps_genes = kind == "refine" and not c["fp64"]
        loss, grads, dpos = _exact_gradient(c, seed, 0.0 if steps_genes else T0)
        if kind == "gradient":
            return loss, grads, dpos
        if steps_genes:  # genes 9 and 10 moved by a twentieth of their range up the gradient
            g = np.stack([t[5] for t in _tanks(c, seed)[1]])
            lo, hi = tank.GENOME_LOWER, tank.GENOME_UPPER
            for q, d in ((9, grads[1]), (10, grads[2])):
                g[:, q] = np.clip(g[:, q] + 0.05 * (hi[q] - lo[q]) * np.sign(d.cpu().numpy()), lo[q], hi[q])
            return g, [loss]
        return loss, dict(zip(("actuation", "contraction", "freq"), grads))
    if kind == "episode":
        return _exact_rows(c, seed)
    if kind == "generate":
        return (None, *_exact_rows(c, seed))
    if kind == "plain":
        return _exact_rows(c, seed)[0]
    specs, tanks = _tanks(c, seed)
    st = _state(specs[0], tanks[0], seed)
    k, live = _consts(specs[0], [tanks[0][1]], [tanks[0][2]], 1)
    at = torch.tensor(live[0], device="cuda")
    full = {q: torch.tensor(st[q].astype(np.float64), device="cuda") for q in st}
    x, v, C, F = (full[q][at] for q in ("x", "v", "C", "F"))
    act, con, freq = _timing(tanks, 1)
    jp = torch.ones_like(x[:, 0])
    glow, dead = torch.zeros_like(jp), 0.0
    for n in range(c["substeps"]):
        x, v, C, F, ratio = _substep(x, v, C, F, k, act, con, freq, T0 + n * DT)
        jp = jp * ratio
        glow = torch.maximum(glow * 0.9, (1.0 - jp).abs())
    for q, val in (("x", x), ("v", v), ("C", C), ("F", F), ("Jp", jp), ("glow", glow if c["glow"] else dead)):
        full[q][at] = val
    return [dict(full, material=None, fiber=None)]
