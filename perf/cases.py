"""Measured cases: what programs built on plgpu ask of it, over the range they ask it.

A case is a dict of plain values; `kind` says which public calls one pass makes:

  frame   Physics.update() with the snapshot after it (the app's loop: one
          step, then the renderer reads the arrays).  The world moves on from
          pass to pass, as in the app.
  state   GpuWorld.upload + GpuWorld.step_download(steps): a state comes from
          the host, advances `steps` steps and is read back.  steps = 1 is the
          end-to-end frame of a program that owns the state on the host.
  sweep   GpuBatch.update (last job's worlds out, this job's worlds in) +
          GpuBatch.step(steps) + one download per world: a parameter sweep.
  image   Physics.thumbnail: the picture stored with a saved state.

Worlds: `dist` "uniform" (a freshly made world) or "blobs" (a world that has
clustered: Gaussian blobs of width `sigma`).  Positions, velocities and matrix
entries are FP32 values, so the FP32 state equals the 64-bit one at the start.
"""
from __future__ import annotations

import math
import sys
from pathlib import Path

import numpy as np
import torch

_PKG = str(Path(__file__).resolve().parent.parent / "particle-life-app_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from plgpu import GpuWorld, ParticleLifeAccelerator, Physics  # noqa: E402
from plgpu.batch import GpuBatch, WorldDesc  # noqa: E402
from plgpu.workloads import BLOB3D_RMAX, friction_of_half_life  # noqa: E402

FRICTION = friction_of_half_life(0.043)  # the reference's friction half-life
BETA = 0.3
BLOBS = 64


def _state(name, dim, n, types, rmax, steps, dist="uniform", sigma=0.0, wrap=True, dt=0.01, pinned=False):
    return dict(name=name, kind="state", dim=dim, n=n, types=types, rmax=rmax, steps=steps, dist=dist, sigma=sigma,
                wrap=wrap, dt=dt, pinned=pinned)


def listed():
    return [
        # The app as it starts: its default 10,000 particles, one update and
        # one snapshot per frame.  The smallest call: launches and the host.
        dict(name="frame_2d_10k", kind="frame", dim=2, n=10_000, types=7, rmax=0.02),
        # The same size run headless: the 10k benchmark configuration, with
        # many steps between looks.
        _state("steps_2d_10k", 2, 10_000, 6, 0.02, 200, dt=0.02),
        # A ragged mid-size world that has clustered, in the clamped box.
        _state("steps_2d_blobs_120k", 2, 120_011, 12, 0.008, 50, dist="blobs", sigma=0.03, wrap=False),
        # The headline configuration (1M particles, 8 types, 20 neighbours).
        _state("steps_2d_1m", 2, 1_000_000, 8, 0.0025, 20),
        # One step of it end to end with page-locked arrays.
        _state("e2e_2d_1m", 2, 1_000_000, 8, 0.0025, 1, pinned=True),
        # 3D, uniform, odd size, more than 16 types (matrix outside shared memory).
        _state("steps_3d_60k", 3, 60_001, 24, 0.05, 50),
        # 3D at the tests' size, 16 types, about 36 neighbours.
        _state("steps_3d_250k", 3, 250_000, 16, 0.0325, 20),
        # The 3D benchmark configuration: 4M particles in 64 blobs.
        _state("steps_3d_blobs_4m", 3, 4_000_000, 16, BLOB3D_RMAX, 8, dist="blobs", sigma=0.025),
        # A sweep: 16 worlds over the batched benchmark's sizes and radii.
        dict(name="sweep_2d_16", kind="sweep", dim=2, worlds=16, n_lo=1_000, n_hi=200_000, rmax_lo=0.005,
             rmax_hi=0.03, steps=100),
        # A 3D sweep of small and mid-size worlds.
        dict(name="sweep_3d_8", kind="sweep", dim=3, worlds=8, n_lo=2_000, n_hi=150_000, rmax_lo=0.03, rmax_hi=0.06,
             steps=30),
        # The 256 x 256 picture of a save.
        dict(name="image_40k", kind="image", dim=2, n=40_000, types=7, rmax=0.02, pixels=256),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _rmax_for(dim, n, k):
    r = math.sqrt(k / (math.pi * n)) if dim == 2 else (3 * k / (4 * math.pi * n)) ** (1 / 3)
    return min(r, 0.3)


def draw(rng):
    kind = rng.choice(["frame", "state", "state", "state", "sweep", "image"])
    dim = rng.choice([2, 3])
    if kind == "frame":
        n = _log_int(rng, 1_000, 50_000)
        return dict(kind=kind, dim=dim, n=n, types=rng.randint(3, 16), rmax=_rmax_for(dim, n, rng.uniform(10, 50)))
    if kind == "image":
        n = _log_int(rng, 1_000, 100_000)
        return dict(kind=kind, dim=2, n=n, types=rng.randint(3, 16), rmax=_rmax_for(2, n, rng.uniform(10, 50)),
                    pixels=rng.choice([256, 200, 512]))
    if kind == "sweep":
        lo = _log_int(rng, 500, 5_000)
        hi = _log_int(rng, 20_000, 150_000)
        r = (0.005, 0.03) if dim == 2 else (0.02, 0.05)
        return dict(kind=kind, dim=dim, worlds=rng.randint(2, 16), n_lo=lo, n_hi=hi,
                    rmax_lo=r[0] * rng.uniform(1.0, 1.5), rmax_hi=r[1], steps=rng.randint(10, 50))
    n = _log_int(rng, 1_000, 2_000_000)
    dist = rng.choice(["uniform", "uniform", "blobs"])
    k = rng.uniform(10, 50)
    sigma = rng.uniform(0.02, 0.05) if dist == "blobs" else 0.0
    rmax = _rmax_for(dim, n, k)
    if dist == "blobs":  # k neighbours in the blobs, not in the mean density
        rmax *= min(1.0, (k / max(_neighbours(dim, n, rmax, sigma), 1e-9)) ** (1 / dim))
    steps = max(1, min(200, _log_int(rng, 4, 200), int(2e7 / n)))
    types = rng.randint(17, 64) if rng.random() < 0.1 else rng.randint(3, 16)
    return dict(kind="state", dim=dim, n=n, types=types, rmax=rmax, steps=steps, dist=dist, sigma=sigma,
                wrap=rng.random() < 0.75, dt=rng.choice([0.005, 0.01, 0.02]), pinned=rng.random() < 0.25)


# ---- inputs ----


def _f32(a):
    return np.asarray(a, np.float32).astype(np.float64)


def _matrix(rng, types):
    return _f32(2 * rng.random((types, types)) - 1)


def _particles(rng, dim, n, types, dist="uniform", sigma=0.0):
    pos = np.zeros((n, 3))
    if dist == "blobs":
        centres = rng.random((BLOBS, dim), dtype=np.float32)
        p = rng.standard_normal((n, dim), dtype=np.float32) * np.float32(sigma)
        p += centres[rng.integers(0, BLOBS, n)]
        p -= np.floor(p)
        p[p >= 1.0] = 0.0
        pos[:, :dim] = p
    else:
        pos[:, :dim] = rng.random((n, dim), dtype=np.float32)
    vel = np.zeros((n, 3))
    vel[:, :dim] = rng.standard_normal((n, dim), dtype=np.float32) * np.float32(0.01)
    return pos, vel, rng.integers(0, types, n).astype(np.int32)


class _UniformPositions:
    """A position setter whose coordinates are FP32 values."""

    def __init__(self, rng, dim):
        self.rng, self.dim = rng, dim

    def set(self, position, type_, n_types):
        position[:] = 0.0
        position[: self.dim] = self.rng.random(self.dim, dtype=np.float32)


def _generator(seed):
    return np.random.Generator(np.random.Philox(seed))


def _physics(case, seed):
    p = Physics(ParticleLifeAccelerator(BETA), position_setter=_UniformPositions(_generator(seed + 1), case["dim"]),
                dim=case["dim"], seed=seed, initial_count=0)
    p.set_matrix_size(case["types"])
    p.settings.matrix.values[:] = _f32(p.settings.matrix.values)
    p.settings.rmax = case["rmax"]
    p.set_particle_count(case["n"])
    return p


def _sweep_worlds(case, seed):
    """Sizes and radii spread over their ranges (the seed does not move them), contents from the seed."""
    rng = _generator(seed)
    w = case["worlds"]
    out = []
    for k in range(w):
        f = k / max(w - 1, 1)
        n = int(round(case["n_lo"] * (case["n_hi"] / case["n_lo"]) ** f))
        g = ((k * 7) % w) / max(w - 1, 1)  # large and small radii over all sizes
        rmax = case["rmax_lo"] + (case["rmax_hi"] - case["rmax_lo"]) * g
        types = 3 + (k * 5) % 10
        pos, vel, typ = _particles(rng, case["dim"], n, types)
        out.append(WorldDesc(pos=pos, vel=vel, types=typ, matrix=_matrix(rng, types), rmax=rmax, friction=FRICTION,
                             dt=0.02, beta=BETA))
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("frame", "image"):
        p = _physics(case, seed)
        p.world  # the GPU world
        st = dict(kind=kind, physics=p)
        if kind == "image":
            pal = np.ones((case["types"], 4), np.float32)
            pal[:, :3] = _generator(seed + 2).random((case["types"], 3), dtype=np.float32)
            st.update(palette=pal, pixels=case["pixels"])
        return st
    if kind == "sweep":
        worlds = _sweep_worlds(case, seed)
        cells = sum(int(math.floor(1.0 / w.rmax)) ** case["dim"] for w in worlds)
        b = GpuBatch(case["dim"], sum(len(w.types) for w in worlds), len(worlds), cells)
        return dict(kind=kind, batch=b, worlds=worlds, ids=[], steps=case["steps"])
    rng = _generator(seed)
    n = case["n"]
    pos, vel, types = _particles(rng, case["dim"], n, case["types"], case["dist"], case["sigma"])
    out = [np.zeros((n, 3)), np.zeros((n, 3)), np.zeros(n, np.int32), np.zeros(n, np.int32)]
    if case["pinned"]:
        pos, vel, types, *out = [torch.from_numpy(a).pin_memory().numpy() for a in (pos, vel, types, *out)]
    w = GpuWorld(case["dim"], n)
    w.set_settings(case["rmax"], FRICTION, 1.0, case["dt"], beta=BETA, wrap=case["wrap"])
    w.set_matrix(_matrix(rng, case["types"]))
    return dict(kind=kind, world=w, pos=pos, vel=vel, types=types, out=tuple(out), steps=case["steps"])


def run(state):
    kind = state["kind"]
    if kind == "frame":
        p = state["physics"]
        p.update()
        return p.positions, p.velocities, p.types, p.ids
    if kind == "image":
        return state["physics"].thumbnail(state["palette"], state["pixels"])
    if kind == "sweep":
        b = state["batch"]
        state["ids"] = b.update(remove=state["ids"], add=state["worlds"])
        b.step(state["steps"])
        return [b.download(i) for i in state["ids"]]
    w = state["world"]
    w.upload(state["pos"], state["vel"], state["types"])
    return w.step_download(state["steps"], state["out"])


# ---- what a pass cannot do without ----


def _neighbours(dim, n, rmax, sigma):
    """Mean particles within rmax of a particle."""
    ball = math.pi * rmax**2 if dim == 2 else 4 / 3 * math.pi * rmax**3
    if not sigma:
        return n * ball
    blob = (4 * math.pi * sigma**2) ** (dim / 2)  # inverse mean density of a Gaussian blob seen from its members
    return n * ball * (1 / BLOBS / max(blob, 1e-30) + (1 - 1 / BLOBS))


def work(case):
    """bytes: the state read from and written to the host arrays (or the
    picture) once.  flops: per step, for every interacting pair its distance,
    force and accumulation (2D 19, 3D 24)."""
    kind, dim = case["kind"], case["dim"]
    pair = 19 if dim == 2 else 24
    if kind == "image":
        return dict(bytes=16 * case["n"] + 4 * case["pixels"] ** 2, flops=0)
    if kind == "frame":
        n = case["n"]
        return dict(bytes=56 * n, flops=pair * n * _neighbours(dim, n, case["rmax"], 0))
    if kind == "sweep":
        ws = _sweep_sizes(case)
        return dict(bytes=sum(108 * n for n, _ in ws),
                    flops=case["steps"] * pair * sum(n * _neighbours(dim, n, r, 0) for n, r in ws))
    n = case["n"]
    return dict(bytes=108 * n, flops=case["steps"] * pair * n * _neighbours(dim, n, case["rmax"], case["sigma"]))


def _sweep_sizes(case):
    w, out = case["worlds"], []
    for k in range(w):
        f = k / max(w - 1, 1)
        g = ((k * 7) % w) / max(w - 1, 1)
        out.append((int(round(case["n_lo"] * (case["n_hi"] / case["n_lo"]) ** f)),
                    case["rmax_lo"] + (case["rmax_hi"] - case["rmax_lo"]) * g))
    return out


# ---- 64-bit values ----


def _exact_step(dim, pos, vel, types, matrix, rmax, friction, force, dt, wrap):
    """One update in float64: particles in the stable order of their cells, forces from all particles
    within rmax, then velocity and position."""
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    x = torch.from_numpy(pos[:, :dim].copy()).to(dev)
    v = torch.from_numpy(vel[:, :dim].copy()).to(dev)
    t = torch.from_numpy(types.astype(np.int64)).to(dev)
    m = torch.from_numpy(np.ascontiguousarray(matrix)).to(dev)
    n, nx = x.shape[0], int(math.floor(1 / rmax))
    c = (x / rmax).to(torch.int64).clamp_(max=nx - 1)
    mult = torch.tensor([nx**k for k in range(dim)], device=dev)
    key = (c * mult).sum(1)
    order = torch.argsort(key, stable=True)
    x, v, t, c, key = x[order], v[order], t[order], c[order], key[order]
    start = torch.searchsorted(key, torch.arange(nx**dim + 1, device=dev))
    acc = torch.zeros_like(x)
    offsets = torch.cartesian_prod(*[torch.tensor([-1, 0, 1], device=dev)] * dim)
    # Targets by the size of their largest neighbour cell, in slices of a bounded number of pairs.
    size = start[1:] - start[:-1]
    for off in offsets:
        cell = c + off
        inside = ((cell >= 0) & (cell < nx)).all(1)
        nb = (cell.remainder(nx) * mult).sum(1)
        cnt = size[nb]
        if not wrap:
            cnt = torch.where(inside, cnt, torch.zeros_like(cnt))
        by = torch.argsort(cnt)
        sizes = cnt[by].cpu().numpy()
        lo = int(np.searchsorted(sizes, 1))
        while lo < n:
            hi = min(n, lo + 8192)
            while hi < n and (hi - lo) * int(sizes[hi - 1]) < 4_000_000:
                hi = min(n, 2 * hi - lo)
            i = by[lo:hi]
            k = torch.arange(int(sizes[hi - 1]), device=dev)
            j = start[nb[i]][:, None] + k[None, :]
            ok = (k[None, :] < cnt[i][:, None]) & (j != i[:, None])
            j = j.clamp(max=n - 1)
            d = x[j] - x[i][:, None, :]
            if wrap:
                d = torch.where(d < -0.5, d + 1, torch.where(d >= 0.5, d - 1, d))
            d2 = (d * d).sum(2)
            ok &= (d2 != 0) & (d2 <= rmax * rmax)
            r = torch.where(ok, d2, torch.ones_like(d2)).sqrt() / rmax
            a = m[t[i][:, None], t[j]]
            f = torch.where(r < BETA, r / BETA - 1, a * (1 - (1 + BETA - 2 * r).abs() / (1 - BETA)))
            g = torch.where(ok, f / (r * rmax), torch.zeros_like(f))
            acc[i] += (d * g[:, :, None]).sum(1)
            lo = hi
    v = v * friction ** (60 * dt) + acc * (rmax * force * dt)
    x = x + v * dt
    x = x - x.floor() if wrap else x.clamp(0, 1)
    full = lambda a: torch.nn.functional.pad(a, (0, 3 - dim)).cpu().numpy()  # noqa: E731
    return full(x), full(v), t.cpu().numpy().astype(np.int32), order.cpu().numpy().astype(np.int32)


def exact(case, seed):
    """One step has 64-bit values.  After several, the two states' cell orders have parted here and there (a
    particle within rounding of a cell's edge), so they have none to be held against; pictures are bytes."""
    if case["kind"] == "frame":
        p = _physics(case, seed)
        s = p.settings
        return _exact_step(case["dim"], p.positions, p.velocities, p.types, s.matrix.as_array(), s.rmax, s.friction,
                           s.force, s.dt, s.wrap)
    if case["kind"] == "state" and case["steps"] == 1:
        rng = _generator(seed)
        pos, vel, types = _particles(rng, case["dim"], case["n"], case["types"], case["dist"], case["sigma"])
        return _exact_step(case["dim"], pos, vel, types, _matrix(rng, case["types"]), case["rmax"], FRICTION, 1.0,
                           case["dt"], case["wrap"])
    return None
