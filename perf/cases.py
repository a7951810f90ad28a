"""Timed cases: what programs have this framework do, from one frame of a small
scene to one step of 512 ragged scenes.

A case is one of five kinds:

* ``frame``:  toImage of a resident scene into host memory (8-bit RGBA).
* ``solve``:  the allocation-free pressure solve on the caller's device arrays.
* ``update``: one update() of one handle whose fields the caller owns between
  steps (hands in velocity, density and temperature, adds an inflow, steps,
  takes every field back); steps 2-8 of the tutorial in both precisions.
* ``batch``:  one step of many resident ragged scenes, then every field of
  every scene read back.  The scenes keep moving from pass to pass.
* ``serve``:  a burst of requests through the serving loop, from submission to
  the fields of every finished request.

Initial fields are smooth random vortices around the bodies with a small part
that is not divergence free, smoke and heat blobs, and the inflow rectangles
and bodies of the scene generators (ifluids/scenes.py).
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "incremental-fluids_gb300"))
import ifluids  # noqa: E402
from ifluids.scenes import batch_scenes, random_bodies  # noqa: E402

FIELDS = ("d", "t", "u", "v")
AIR, SOOT, DIFFUSION = 0.1, 1.0, 0.01  # densities and diffusion of the reference's mains


def listed():
    return [
        # a movie's frame of the reference main's grid, heat panel and all: the smallest call
        {"name": "frame-128", "kind": "frame", "variant": 7, "w": 128, "h": 128, "bits": 64, "heat": True},
        # a host framework's own pressure system, solved inside its memory pool
        {"name": "solve-97x61", "kind": "solve", "w": 97, "h": 61},
        # the drop-in on the grid that every reference main uses: smoke in a box
        {"name": "plain64-128", "kind": "update", "variant": 3, "w": 128, "h": 128, "bits": 64, "bodies": 0},
        # the drop-in on a ragged grid with turning bodies
        {"name": "solid64-203x150", "kind": "update", "variant": 4, "w": 203, "h": 150, "bits": 64, "bodies": 2},
        # Gauss-Seidel tutorial step on the reference main's grid
        {"name": "gs64-128", "kind": "update", "variant": 2, "w": 128, "h": 128, "bits": 64, "bodies": 0},
        # FLIP on the reference main's grid with the FP32-form solves
        {"name": "flip32-128", "kind": "update", "variant": 8, "w": 128, "h": 128, "bits": 32, "bodies": 1},
        # an ordinary scene in the FP32 form, odd sides
        {"name": "plain32-257x190", "kind": "update", "variant": 3, "w": 257, "h": 190, "bits": 32, "bodies": 0},
        # the benchmark's kind of single scene: a large square with three turning bodies
        {"name": "solid32-768", "kind": "update", "variant": 4, "w": 768, "h": 768, "bits": 32, "bodies": 3},
        # the benchmark's kind of large scene: heat, variable density, two PCG solves
        {"name": "vardens32-1536", "kind": "update", "variant": 7, "w": 1536, "h": 1536, "bits": 32, "bodies": 1},
        # a small batch of small scenes: too few to fill the GPU
        {"name": "batch32-24", "kind": "batch", "mix": 7, "scenes": 24, "lo": 64, "hi": 256},
        # the benchmark's kind of batch
        {"name": "batch32-512", "kind": "batch", "mix": 2, "scenes": 512, "lo": 64, "hi": 768},
        # a burst of short requests through the serving loop
        {"name": "serve32-12", "kind": "serve", "mix": 11, "requests": 12, "lo": 64, "hi": 256, "steps": 3},
    ]


# Sides of the FP32 form's scenes end where its solves still converge whatever the
# seed places (with several bodies on 1024^2 some run into the iteration cap, at
# which the fields say nothing).
def draw(rng: random.Random):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["frame", "solve", "update", "update", "update", "update", "update", "batch", "serve"])
    if kind == "frame":
        variant = rng.randint(3, 7)
        return {"kind": kind, "variant": variant, "w": log(32, 2048), "h": log(32, 2048), "bits": rng.choice([32, 64]),
                "heat": variant >= 6}
    if kind == "solve":
        return {"kind": kind, "w": log(24, 256), "h": log(24, 256)}
    if kind == "update":
        variant = rng.choice([2, 3, 3, 4, 4, 5, 6, 7, 8])
        if variant in (2, 8):
            bits = 64 if variant == 2 else 32
            w, h = log(64, 320), log(64, 320)
        else:
            bits = rng.choice([32, 32, 64])
            hi = 320 if bits == 64 else 768 if variant <= 4 else 512
            w, h = log(64, hi), log(64, hi)
        if variant >= 7:  # the reference's index of the v-face densities needs h < w + 2
            w, h = max(w, h), min(w, h)
        return {"kind": kind, "variant": variant, "w": w, "h": h, "bits": bits,
                "bodies": 0 if variant < 4 else 1 if variant == 8 else rng.randint(1, 3)}
    if kind == "batch":
        return {"kind": kind, "mix": rng.randint(100, 999), "scenes": log(8, 128), "lo": 64, "hi": rng.choice([256, 512, 768])}
    return {"kind": kind, "mix": rng.randint(100, 999), "requests": rng.randint(4, 20), "lo": 64, "hi": rng.choice([192, 256, 384]),
            "steps": rng.randint(2, 5)}


# ------------------------------------------------------------------- inputs
def _names(variant):
    return FIELDS if variant >= 6 else ("d", "u", "v")


def _fields(w, h, rng, bodies=()):
    """Cell-centred d and t, face-centred u and v (zero on the walls) as FP64 CUDA tensors.
    The vortices die out towards the bodies, so that no flow enters one (as in a running
    scene, where each step's projection saw the bodies)."""
    hx = 1.0 / min(w, h)
    # everything that needs the generator is drawn on the host: a few numbers per field
    m = np.arange(1, 7)
    amp = torch.from_numpy(rng.normal(size=(6, 6)) / np.add.outer(m ** 1.5, m ** 1.5)).cuda()
    pot = torch.from_numpy(rng.normal(size=(6, 6)) / np.add.outer(m ** 2, m ** 2)).cuda()
    blobs = rng.uniform(size=(6, 4))

    def waves(n, pts, fn):
        return fn(torch.outer(torch.arange(1, 7, device="cuda", dtype=torch.float64), pts / n * math.pi))

    def at(n, off):
        return torch.arange(n, device="cuda", dtype=torch.float64) + off

    psi = waves(h, at(h + 1, 0.0), torch.sin).T @ amp @ waves(w, at(w + 1, 0.0), torch.sin)
    phi = waves(h, at(h, 0.5), torch.cos).T @ pot @ waves(w, at(w, 0.5), torch.cos)
    cx, cy = at(w + 1, 0.0)[None, :] * hx, at(h + 1, 0.0)[:, None] * hx
    for b in bodies:
        reach = 0.5 * (math.hypot(b[3], b[4]) if b[0] == 0 else b[3])
        away = (((cx - b[1]) ** 2 + (cy - b[2]) ** 2).sqrt() - reach - 0.01) / 0.1
        away = away.clamp(0.0, 1.0)
        psi = psi * away * away * (3.0 - 2.0 * away)
    u = (psi[1:, :] - psi[:-1, :]) / hx
    v = -(psi[:, 1:] - psi[:, :-1]) / hx
    scale = 1.5 / max(float(u.abs().max()), float(v.abs().max()))
    u, v = u * scale, v * scale
    gu, gv = (phi[:, 1:] - phi[:, :-1]) / hx, (phi[1:, :] - phi[:-1, :]) / hx
    small = 0.02 / max(float(gu.abs().max()), float(gv.abs().max()))
    u[:, 1:-1] += gu * small
    v[1:-1, :] += gv * small
    u[:, 0] = u[:, -1] = 0.0
    v[0, :] = v[-1, :] = 0.0
    x, y = at(w, 0.5)[None, :] / w, at(h, 0.5)[:, None] / h
    smoke = torch.zeros((h, w), device="cuda", dtype=torch.float64)
    for bx, by, br, ba in blobs:
        r2 = ((x - 0.1 - 0.8 * bx) ** 2 + (y - 0.1 - 0.8 * by) ** 2) / (0.05 + 0.1 * br) ** 2
        smoke += (0.2 + 0.8 * ba) * torch.exp(-r2)
    return {"d": smoke.clamp(max=1.0), "t": 294.0 + 250.0 * smoke.clamp(max=1.0), "u": u, "v": v}


def _pinned(shape, dtype):
    return torch.empty(shape, dtype=dtype, pin_memory=True).numpy()


def _host_fields(case, seed, bodies=()):
    """The input fields of an `update` or `frame` case in pinned host arrays of the handle's element type."""
    f = _fields(case["w"], case["h"], np.random.default_rng([int(seed), 1]), bodies)
    dt = torch.float64 if case["bits"] == 64 else torch.float32
    out = {}
    for k in _names(case["variant"]):
        a = _pinned(tuple(f[k].shape), dt)
        a[...] = f[k].to(dt).cpu().numpy()
        out[k] = a
    return out


def _bodies(rng, count, variant):
    """Rotating bodies in step 4; from step 5 on they stand still (a rotating body in
    a closed domain gives the fractional steps an inconsistent pressure system)."""
    bodies = random_bodies(rng, count)
    if variant >= 5:
        bodies = [b[:6] + (0.0, 0.0, 0.0) for b in bodies]
    return bodies


def _solver(variant, w, h, bits, bodies):
    precision = ifluids.FP64 if bits == 64 else ifluids.FP32
    if variant <= 3:
        return ifluids.FluidSolver(w, h, AIR, variant=variant, precision=precision)
    if variant <= 5:
        return ifluids.FluidSolver(w, h, AIR, bodies, variant=variant, precision=precision)
    soot = 0.25 if variant == 8 else SOOT
    return ifluids.FluidSolver(w, h, AIR, soot, DIFFUSION, bodies, variant=variant, precision=precision)


def _inflow(variant):
    """(arguments of addInflow, time step) as in the reference's mains and the benchmark."""
    if variant >= 7:
        return (0.45, 0.2, 0.1, 0.05, 1.0, 700.0 if variant == 7 else 294.0, 0.0, 0.0), 0.0025 if variant == 8 else 0.001
    if variant == 6:
        return (0.35, 0.2, 0.2, 0.1, 1.0, 594.0, 0.0, 0.0), 0.0025
    return (0.45, 0.2, 0.15, 0.03, 1.0, 0.0, 3.0), 0.0025


class _Frame:
    def __init__(self, case, seed):
        rng = np.random.default_rng([int(seed), 0])
        self.heat = case["heat"]
        bodies = _bodies(rng, 1, case["variant"]) if case["variant"] >= 4 else []
        self.g = _solver(case["variant"], case["w"], case["h"], case["bits"], bodies)
        self.g.run_phase(ifluids.PH_FILL_SOLID, 0.0025)
        for k, a in _host_fields(case, seed, bodies).items():
            self.g.write_field(k, a)

    def run(self):
        return self.g.to_image(self.heat)


def _system(w, h, seed):
    """aDiag, aPlusX, aPlusY and the right-hand side of step 3 for the seed's velocities (FP64 CUDA tensors)."""
    f = _fields(w, h, np.random.default_rng([int(seed), 1]))
    hx = 1.0 / min(w, h)
    rhs = -(f["u"][:, 1:] - f["u"][:, :-1] + f["v"][1:, :] - f["v"][:-1, :]) / hx
    scale = 0.0025 / (AIR * hx * hx)
    ax, ay = torch.full_like(rhs, -scale), torch.full_like(rhs, -scale)
    ax[:, -1] = 0.0
    ay[-1, :] = 0.0
    diag = torch.full_like(rhs, 4.0 * scale)
    diag[:, 0] -= scale
    diag[:, -1] -= scale
    diag[0, :] -= scale
    diag[-1, :] -= scale
    return diag, ax, ay, rhs.contiguous()


class _Solve:
    def __init__(self, case, seed):
        self.w, self.h = case["w"], case["h"]
        self.a = _system(self.w, self.h, seed)
        self.p = torch.zeros((self.h, self.w), dtype=torch.float64, device="cuda")
        self.stats = torch.zeros(16, dtype=torch.uint8, device="cuda")  # ifl_pcg_stats

    def run(self):
        diag, ax, ay, rhs = (t.data_ptr() for t in self.a)
        status = ifluids.pcg_solve_noalloc(self.w, self.h, diag, ax, ay, rhs, self.p.data_ptr(), 600,
                                           self.stats.data_ptr(), torch.cuda.current_stream().cuda_stream)
        if status != ifluids.OK:
            raise RuntimeError("solve returned %d" % status)
        return self.p


class _Update:
    def __init__(self, case, seed):
        self.variant = case["variant"]
        rng = np.random.default_rng([int(seed), 0])
        bodies = _bodies(rng, case["bodies"], self.variant)
        self.g = _solver(self.variant, case["w"], case["h"], case["bits"], bodies)
        self.inflow, self.dt = _inflow(self.variant)
        self.fields = _host_fields(case, seed, bodies)
        if self.variant == 2:  # the Gauss-Seidel steps keep the pressure from step to step: it is handed in, too
            self.fields["p"] = _pinned((case["h"], case["w"]), torch.float64)
            self.fields["p"][...] = 0.0
        self.out = {k: _pinned(a.shape, torch.from_numpy(a).dtype) for k, a in self.fields.items()}

    def run(self):
        for k, a in self.fields.items():
            self.g.write_field(k, a)
        self.g.addInflow(*self.inflow)
        self.g.update(self.dt)
        return {k: self.g.read_field(k, out=a) for k, a in self.out.items()}


class _Flip:
    """The particles are the state: the caller hands them in, steps, and takes them and the grid back."""

    def __init__(self, case, seed):
        w, h = case["w"], case["h"]
        rng = np.random.default_rng([int(seed), 0])
        bodies = [(0, 0.5, 0.6, 0.7, 0.1, math.pi * 0.25, 0.0, 0.0, 0.0)]
        self.g = _solver(8, w, h, case["bits"], bodies)
        self.inflow, self.dt = _inflow(8)
        f = {k: a.cpu().numpy() for k, a in _fields(w, h, np.random.default_rng([int(seed), 1]), bodies).items()}
        # four jittered particles per cell, none inside the body (the reference's placement)
        cx = np.repeat(np.tile(np.arange(w), h), 4)
        cy = np.repeat(np.repeat(np.arange(h), w), 4)
        x, y = cx + rng.random(len(cx)), cy + rng.random(len(cy))
        hx = 1.0 / min(w, h)
        px, py = x * hx - 0.5, y * hx - 0.6
        c, s = math.cos(math.pi * 0.25), math.sin(math.pi * 0.25)
        keep = (np.abs(c * px + s * py) > 0.35) | (np.abs(-s * px + c * py) > 0.05)
        x, y, cx, cy = x[keep], y[keep], cx[keep], cy[keep]
        # values at the particle's cell, plus the spread that carried particles have
        u = 0.5 * (f["u"][cy, cx] + f["u"][cy, cx + 1]) + 0.02 * rng.normal(size=len(x))
        v = 0.5 * (f["v"][cy, cx] + f["v"][cy + 1, cx]) + 0.02 * rng.normal(size=len(x))
        self.particles = (x, y, f["d"][cy, cx].copy(), f["t"][cy, cx].copy(), u, v)
        self.taken = [np.zeros(12 * w * h, dtype=np.float32) for _ in range(6)]

    def run(self):
        g = self.g
        g.set_particles(self.particles)
        g.rng_state = 0xBA5EBA11
        g.addInflow(*self.inflow)
        g.update(self.dt)
        out = {k: g.read_field(k, dtype=np.float32) for k in FIELDS}
        for k, a in enumerate(self.taken):  # as a renderer takes them, into arrays of the particles' capacity
            live = g.particles(k)
            a[:len(live)] = live
            a[len(live):] = 0.0
            out["particles%d" % k] = a
        return out


def _scenes(count, case, seed):
    """The sides of a generated mix of scenes; the seed places its bodies and inflows."""
    scenes = batch_scenes(count, case["mix"], case["lo"], case["hi"])
    rng = np.random.default_rng([int(seed), 2])
    for s in scenes:
        s.bodies = random_bodies(rng, len(s.bodies))
        s.inflows = [(float(rng.uniform(0.1, 0.8)),) + f[1:7] + (float(rng.uniform(1.0, 4.0)),) for f in s.inflows]
    return scenes


class _Batch:
    def __init__(self, case, seed):
        scenes = _scenes(case["scenes"], case, seed)
        self.dt = scenes[0].dt
        self.members = [_solver(4, s.w, s.h, 32, s.bodies) for s in scenes]
        rng = np.random.default_rng([int(seed), 1])
        for g, s in zip(self.members, scenes):
            f = _fields(s.w, s.h, rng, s.bodies)
            for k in ("d", "u", "v"):
                g.write_field(k, f[k].float().cpu().numpy())
        self.batch = ifluids.Batch(self.members)
        for i, s in enumerate(scenes):
            self.batch.set_inflows(i, s.inflows)
        self.flat, self.views = {}, {}
        for k, dw, dh in (("d", 0, 0), ("u", 1, 0), ("v", 0, 1)):
            shapes = [(s.h + dh, s.w + dw) for s in scenes]
            flat = _pinned((sum(a * b for a, b in shapes),), torch.float32)
            at, views = 0, []
            for a, b in shapes:
                views.append(flat[at:at + a * b].reshape(a, b))
                at += a * b
            self.flat[k], self.views[k] = flat, views

    def run(self):
        self.batch.update(self.dt)
        for k, views in self.views.items():
            for g, a in zip(self.members, views):
                g.read_field(k, out=a)
        return self.flat


class _Serve:
    def __init__(self, case, seed):
        self.scenes = _scenes(case["requests"], case, seed)
        # requests of uneven length, so that the batch is rebuilt as they leave
        self.steps = [1 + (case["steps"] - 1) * (i % 3) // 2 for i in range(len(self.scenes))]
        self.server = ifluids.Server(precision=ifluids.FP32, dt=self.scenes[0].dt, hbm_budget_bytes=64 << 30)

    def run(self):
        srv, ids, out = self.server, {}, {}
        for i, s in enumerate(self.scenes):
            ids[srv.submit(s.w, s.h, self.steps[i], bodies=s.bodies, inflows=s.inflows)] = i
        while srv.step() != (0, 0):
            pass
        for c in srv.completions():
            for k in ("d", "u", "v"):
                out["%s%d" % (k, ids[c["id"]])] = srv.read_field(c["id"], k, dtype=np.float32)
            srv.release(c["id"])
        return out


def prepare(case, seed):
    if case["kind"] == "update" and case["variant"] == 8:
        return _Flip(case, seed)
    return {"frame": _Frame, "solve": _Solve, "update": _Update, "batch": _Batch, "serve": _Serve}[case["kind"]](case, seed)


def run(state):
    return state.run()


# --------------------------------------------------------------------- work
def _step_work(w, h, bits, variant):
    """(bytes, flops) of one update(): fields in and out once; the flops of the solve at
    0.6 iterations per cell of the longer side (2 for the heat and density steps'
    worse conditioning is not counted), 36 per cell and iteration, and 400 per cell for
    the rest of the step."""
    cells, nf = w * h, 4 if variant >= 6 else 3
    iters = 0.6 * max(w, h)
    return 2.0 * nf * cells * bits / 8, cells * (400.0 + 36.0 * iters)


def work(case):
    kind = case["kind"]
    if kind == "frame":
        cells = case["w"] * case["h"]
        return {"bytes": cells * ((3 if case["heat"] else 1) * case["bits"] / 8 + 4 * (2 if case["heat"] else 1)),
                "flops": 30.0 * cells}
    if kind == "solve":
        cells = case["w"] * case["h"]
        return {"bytes": 5 * 8.0 * cells, "flops": 36.0 * cells * 0.6 * max(case["w"], case["h"])}
    if kind == "update":
        b, f = _step_work(case["w"], case["h"], case["bits"], case["variant"])
        if case["variant"] == 8:  # particles: six values in and out, and the transfers
            n = 4 * case["w"] * case["h"]
            b, f = b + 2 * 48.0 * n, f + 600.0 * n
        return {"bytes": b, "flops": f}
    # batches and requests: sides log-uniform in [lo, hi]; their mean work per scene
    n = case["scenes"] if kind == "batch" else sum(1 + (case["steps"] - 1) * (i % 3) // 2 for i in range(case["requests"]))
    mean = (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"])
    b, f = _step_work(mean, mean, 32, 4)
    return {"bytes": n * b, "flops": n * f}


# -------------------------------------------------------------------- exact
# Plain numpy in 64 bits: the small solves, and the small updates without bodies.
class _Wave:
    """Flat indices of the anti-diagonals of a w x h grid, in order."""

    def __init__(self, w, h):
        self.diags = []
        for d in range(w + h - 1):
            y = np.arange(max(0, d - w + 1), min(h, d + 1))
            self.diags.append((y + 1) * (w + 2) + (d - y) + 1)  # on a grid with a border of zeros


def _mic_pcg(diag, ax, ay, rhs, limit):
    """MIC(0)-preconditioned conjugate gradients as the tutorial writes it, by anti-diagonals."""
    h, w = rhs.shape
    P = w + 2
    pad = lambda a: np.pad(a, 1).reshape(-1)  # noqa: E731
    diag, ax, ay, r = pad(diag), pad(ax), pad(ay), pad(rhs)
    wave = _Wave(w, h).diags
    pc = np.zeros_like(diag)
    for i in wave:
        pxl, pyl = ax[i - 1] * pc[i - 1], ay[i - 1] * pc[i - 1]
        pxd, pyd = ax[i - P] * pc[i - P], ay[i - P] * pc[i - P]
        e = diag[i] - (pxl * pxl + 0.97 * pxl * pyl) - (pyd * pyd + 0.97 * pxd * pyd)
        e = np.where(e < 0.25 * diag[i], diag[i], e)
        pc[i] = 1.0 / np.sqrt(e)
    lx, ly = ax * pc, ay * pc

    def apply(r):
        q = np.zeros_like(r)
        for i in wave:
            q[i] = (r[i] - lx[i - 1] * q[i - 1] - ly[i - P] * q[i - P]) * pc[i]
        z = np.zeros_like(r)
        for i in reversed(wave):
            z[i] = (q[i] - lx[i] * z[i + 1] - ly[i] * z[i + P]) * pc[i]
        return z

    p = np.zeros_like(r)
    if np.abs(r).max() < 1e-5:
        return p.reshape(h + 2, P)[1:-1, 1:-1]
    z = apply(r)
    s = z.copy()
    sigma = z @ r
    left, down = np.roll(ax, 1), np.roll(ay, P)
    for _ in range(limit):
        z = diag * s + left * np.roll(s, 1) + down * np.roll(s, P) + ax * np.roll(s, -1) + ay * np.roll(s, -P)
        alpha = sigma / (z @ s)
        p += alpha * s
        r = r - alpha * z
        if np.abs(r).max() < 1e-5:
            break
        z = apply(r)
        new = z @ r
        s = z + (new / sigma) * s
        sigma = new
    return p.reshape(h + 2, P)[1:-1, 1:-1].copy()


def _gauss_seidel(rhs, scale, limit):
    h, w = rhs.shape
    P = w + 2
    inside = np.pad(np.ones_like(rhs), 1).reshape(-1)
    r, p = np.pad(rhs, 1).reshape(-1), np.zeros((h + 2) * P)
    near = np.zeros_like(p)
    for o in (-1, 1, -P, P):
        near += np.roll(inside, -o)
    wave = _Wave(w, h).diags
    div = [1.0 / (scale * near[i]) for i in wave]
    for _ in range(limit):
        worst = 0.0
        for i, c in zip(wave, div):
            new = (r[i] + scale * (p[i - 1] + p[i - P] + p[i + 1] + p[i + P])) * c
            worst = max(worst, float(np.abs(new - p[i]).max()))
            p[i] = new
        if worst < 1e-5:
            break
    return p.reshape(h + 2, P)[1:-1, 1:-1].copy()


def _clamped(a, ox, oy, x, y):
    h, w = a.shape
    x, y = np.clip(x - ox, 0.0, w - 1.001), np.clip(y - oy, 0.0, h - 1.001)
    ix, iy = x.astype(int), y.astype(int)
    return ix, iy, x - ix, y - iy


def _lerp(a, ox, oy, x, y):
    ix, iy, fx, fy = _clamped(a, ox, oy, x, y)
    top = a[iy, ix] * (1 - fx) + a[iy, ix + 1] * fx
    bottom = a[iy + 1, ix] * (1 - fx) + a[iy + 1, ix + 1] * fx
    return top * (1 - fy) + bottom * fy


def _cerp(a, ox, oy, x, y):
    h, w = a.shape
    ix, iy, fx, fy = _clamped(a, ox, oy, x, y)

    def cubic(q, t):
        lo, hi = np.minimum.reduce(q), np.maximum.reduce(q)
        t2, t3 = t * t, t * t * t
        out = q[0] * (-0.5 * t + t2 - 0.5 * t3) + q[1] * (1.0 - 2.5 * t2 + 1.5 * t3) + \
            q[2] * (0.5 * t + 2.0 * t2 - 1.5 * t3) + q[3] * (-0.5 * t2 + 0.5 * t3)
        return np.clip(out, lo, hi)

    xs = [np.maximum(ix - 1, 0), ix, ix + 1, np.minimum(ix + 2, w - 1)]
    ys = [np.maximum(iy - 1, 0), iy, iy + 1, np.minimum(iy + 2, h - 1)]
    return cubic([cubic([a[yy, xx] for xx in xs], fx) for yy in ys], fy)


def _exact_update(case, seed):
    """One update() of steps 2 and 3: inflow, projection, advection."""
    w, h = case["w"], case["h"]
    hx, (inflow, dt) = 1.0 / min(w, h), _inflow(case["variant"])
    f = {k: a.astype(np.float64) for k, a in _host_fields(case, seed).items()}
    off = {"d": (0.5, 0.5), "u": (0.0, 0.5), "v": (0.5, 0.0)}
    x0, y0, x1, y1 = inflow[0], inflow[1], inflow[0] + inflow[2], inflow[1] + inflow[3]
    for k, val in zip(("d", "u", "v"), inflow[4:]):
        a, (ox, oy) = f[k], off[k]
        for y in range(max(int(y0 / hx - oy), 0), min(int(y1 / hx - oy), a.shape[0])):
            for x in range(max(int(x0 / hx - ox), 0), min(int(x1 / hx - ox), a.shape[0])):
                l = min(math.hypot((2.0 * (x + 0.5) * hx - (x0 + x1)) / (x1 - x0),
                                   (2.0 * (y + 0.5) * hx - (y0 + y1)) / (y1 - y0)), 1.0)
                new = (1.0 - l * l * (3.0 - 2.0 * l)) * val
                if abs(a[y, x]) < abs(new):
                    a[y, x] = new
    u, v = f["u"], f["v"]
    rhs = -(u[:, 1:] - u[:, :-1] + v[1:, :] - v[:-1, :]) / hx
    scale = dt / (AIR * hx * hx)
    if case["variant"] == 2:
        p = _gauss_seidel(rhs, scale, 600)
    else:
        inside = np.pad(np.ones((h, w)), 1)
        near = inside[1:-1, :-2] + inside[1:-1, 2:] + inside[:-2, 1:-1] + inside[2:, 1:-1]
        ax, ay = np.full((h, w), -scale), np.full((h, w), -scale)
        ax[:, -1] = 0.0
        ay[-1, :] = 0.0
        p = _mic_pcg(scale * near, ax, ay, rhs, 600)
    u[:, 1:-1] -= dt / (AIR * hx) * (p[:, 1:] - p[:, :-1])
    v[1:-1, :] -= dt / (AIR * hx) * (p[1:, :] - p[:-1, :])
    u[:, 0] = u[:, -1] = 0.0
    v[0, :] = v[-1, :] = 0.0
    out = {"p": p} if case["variant"] == 2 else {}
    for k in ("d", "u", "v"):
        (ox, oy), (fh, fw) = off[k], f[k].shape
        y, x = np.mgrid[0:fh, 0:fw].astype(np.float64)
        x, y = x + ox, y + oy
        vel = lambda px, py: (_lerp(u, 0.0, 0.5, px, py), _lerp(v, 0.5, 0.0, px, py))  # noqa: E731
        u1, v1 = (a / hx for a in vel(x, y))
        u2, v2 = (a / hx for a in vel(x - 0.5 * dt * u1, y - 0.5 * dt * v1))
        u3, v3 = vel(x - 0.75 * dt * u2, y - 0.75 * dt * v2)  # not divided by hx, as in the reference
        out[k] = _cerp(f[k], ox, oy, x - dt * (2 / 9 * u1 + 3 / 9 * u2 + 4 / 9 * u3),
                       y - dt * (2 / 9 * v1 + 3 / 9 * v2 + 4 / 9 * v3))
    return out


def exact(case, seed):
    if case["kind"] == "solve":
        return _mic_pcg(*(t.cpu().numpy() for t in _system(case["w"], case["h"], seed)), 600)
    if case["kind"] == "update" and case["variant"] in (2, 3) and case["w"] + case["h"] <= 640:
        return _exact_update(case, seed)
    return None
