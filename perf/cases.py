"""The work that a user of the engine has it do, as timed cases.

A case is one pass of a program that keeps its particles in host memory and
hands them to the engine: upload, a few time steps, download (or an export
snapshot, or a differentiable trajectory forward and backward).  Scenes are
the lattice scenes of mps_gb300.scenes (dam break, hydrostatic tank, shaken
column, a 3-D tank) with a seeded compression, jitter and velocity
field, so that pressures and velocities are of the size that a running
simulation has, and not those of a lattice at rest.

exact() is the same step written with torch in 64 bits (neighbour pairs from a
sorted cell grid, CG with one residual correction, autograd for the adjoint),
independent of the engine.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from mps_gb300 import FP64, MIXED, Engine, scenes
from mps_gb300.engine import Batch, Trajectory

GHOST, FLUID, WALL, DUMMY = scenes.GHOST, scenes.FLUID, scenes.WALL, scenes.DUMMY


# Relative residual of the mixed solves (the default is 1e-10, a batch's 1e-8): the FP32 sums that
# follow a solve round another way where pressures differ in their tenth digit, so that only
# tighter solves give results that can be told apart from a change of the step itself.
TOL = 1e-12


def listed():
    return [
        # the smallest scene of the smoke test, stepped one call at a time: latency of a step
        dict(name="column_150_fp64", kind="steps", scene="dam", precision="fp64", cols=10, rows=15,
             l0=0.02, steps=4, call="step"),
        # the 1,250-particle dam break (tank 1.0 x 0.6 m), the reference's own CPU-sized run
        dict(name="dam_1250_fp64", kind="steps", scene="dam", precision="fp64", cols=25, rows=50,
             l0=0.01, steps=5, call="report"),
        # the same scene with the mixed solver, single steps as an interactive program takes them
        dict(name="dam_1250_mixed", kind="steps", scene="dam", precision="mixed", cols=25, rows=50,
             l0=0.01, steps=5, call="step"),
        # a validation-sized FP64 run, odd sizes
        dict(name="hydro_20k_fp64", kind="steps", scene="hydro", precision="fp64", cols=143, rows=141,
             l0=2.5e-3, steps=2, call="report"),
        # the driver loop between two exports: steps, an export step, the snapshot
        dict(name="dam_45k_mixed_export", kind="steps", scene="dam", precision="mixed", cols=151, rows=299,
             l0=1.7e-3, steps=5, call="export"),
        # a collision-heavy column
        dict(name="shaken_100k_mixed", kind="steps", scene="shaken", precision="mixed", cols=225, rows=450,
             l0=1e-3, steps=3, call="report"),
        # a 3-D tank of water (Jacobi-preconditioned mixed solver, 27-cell sweeps)
        dict(name="box3d_9k_mixed", kind="steps", scene="box", precision="mixed", cols=21, rows=20,
             l0=0.01, steps=3, call="report"),
        # the benchmark's million-particle dam break
        dict(name="dam_1m_mixed", kind="steps", scene="dam", precision="mixed", cols=707, rows=1414,
             l0=0.5 / 707, steps=4, call="report"),
        # the two-million-particle FP64 dam break
        dict(name="dam_2m_fp64", kind="steps", scene="dam", precision="fp64", cols=1000, rows=2000,
             l0=5e-4, steps=1, call="step"),
        # 64 uneven scenes of 2,000 - 60,000 fluid particles in one batch
        dict(name="batch_64", kind="batch", count=64, sizes=1, low=2000, high=60000, steps=3),
        # differentiable trajectories: a small one and the 25,600-particle tank
        dict(name="adjoint_1600", kind="adjoint", cols=40, rows=40, l0=0.01, steps=10, every=5),
        dict(name="adjoint_25600", kind="adjoint", cols=160, rows=160, l0=2.5e-3, steps=4, every=2),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["steps"] * 8 + ["batch", "adjoint"])
    l0 = _log(rng, 5e-4, 2e-2)
    if kind == "batch":
        lo = int(_log(rng, 500, 8000))
        return dict(kind="batch", count=rng.randint(3, 48), sizes=rng.randint(2, 1 << 20), low=lo,
                    high=lo + int(_log(rng, 1000, 50000)), steps=rng.randint(1, 4))
    if kind == "adjoint":
        nf, aspect = _log(rng, 200, 25000), rng.uniform(0.6, 1.7)
        steps = rng.randint(2, 5)
        return dict(kind="adjoint", cols=max(8, round(math.sqrt(nf / aspect))),
                    rows=max(8, round(math.sqrt(nf * aspect))), l0=l0, steps=steps, every=rng.randint(1, steps))
    scene = rng.choice(["dam"] * 5 + ["hydro"] * 3 + ["shaken", "box"])
    precision = rng.choice(["mixed", "mixed", "fp64"])
    if scene == "box":
        cols = rng.randint(5, 26)
        return dict(kind="steps", scene=scene, precision=precision, cols=cols, rows=rng.randint(5, 24),
                    l0=max(l0, 5e-3), steps=rng.randint(1, 4), call=rng.choice(["step", "report", "export"]))
    top = {"mixed": 9e5, "fp64": 2e5}[precision]
    nf, aspect = _log(rng, 100, top if scene != "shaken" else 1e5), rng.uniform(0.5, 2.2)
    steps = rng.randint(1, 5 if precision == "mixed" or nf < 3e4 else 2)
    return dict(kind="steps", scene=scene, precision=precision, cols=max(6, round(math.sqrt(nf / aspect))),
                rows=max(6, round(math.sqrt(nf * aspect))), l0=l0, steps=steps,
                call=rng.choice(["step", "report", "report", "export"]))


# ------------------------------------------------------------------ inputs


def _box(n, h, l0):
    """An open 3-D tank (one wall and two dummy layers, y up) filled to height h."""
    r, ry = np.arange(-3, n + 3), np.arange(-3, h + 2)
    ix, iy, iz = (a.ravel() for a in np.meshgrid(r, ry, r, indexing="ij"))
    deep = np.max([-1 - ix, ix - n, -1 - iz, iz - n, -1 - iy], axis=0)  # < 0: in the tank
    t = np.where(deep < 0, FLUID, np.where(deep == 0, WALL, DUMMY)).astype(np.int32)
    keep = (deep >= 0) | (iy < h)
    pos = np.stack([(a[keep] + 0.5) * l0 for a in (ix, iy, iz)], 1)
    m = 8 * l0
    prm = scenes.baseline_physics(l0, 0.1 * l0, (-m, -m, -m), (n * l0 + m, h * l0 + 2 * m, n * l0 + m))
    prm["dim"] = 3
    return prm, pos, np.zeros_like(pos), t[keep]


def _deform(scene, size, rng):
    """The fluid compressed vertically until the source term relaxation (n - n0) / (n0 dt^2)
    makes up for the free surface and gives a pressure of the order of rho g H, jittered by 0.01 l0,
    with a cellular velocity field of ~0.5 m/s and 5 mm/s of noise."""
    prm, pos, vel, t = scene
    l0, d = prm["particle_distance"], 3 if prm["dim"] == 3 else 2
    f = np.flatnonzero(t == FLUID)
    x = pos[f] / np.asarray(size)
    new, v = pos[f].copy(), np.zeros((len(f), 3))
    strain = rng.uniform(0.7, 1.3) * 8 * 9.81 * prm["dt"] ** 2 / (prm["relaxation"] * size[1])
    new[:, 1] -= strain * new[:, 1]
    for _ in range(3):
        k, u = rng.integers(1, 4, 2), rng.uniform(-0.4, 0.4)
        (s0, s1), (c0, c1) = ([fn(math.pi * k[a] * x[:, a]) for a in (0, 1)] for fn in (np.sin, np.cos))
        v[:, 0] += u * s0 * c1
        v[:, 1] -= u * (k[0] * size[1]) / (k[1] * size[0]) * c0 * s1
    new[:, :d] += rng.uniform(-0.01, 0.01, (len(f), d)) * l0
    v[:, :d] += rng.normal(0, 0.005, (len(f), d))
    pos, vel = pos.copy(), vel.copy()
    pos[f], vel[f] = new, v
    return prm, pos, vel, t


def _scene(case, seed):
    rng = np.random.default_rng(seed)
    if case["kind"] == "batch":
        out = []
        for prm, pos, vel, t in scenes.batch_scenes(case["sizes"], case["count"], (case["low"], case["high"])):
            f = pos[t == FLUID]
            l0 = prm["particle_distance"]
            out.append(_deform((prm, pos, vel, t), (f[:, 0].max() + l0 / 2, f[:, 1].max() + l0 / 2, 1.0), rng))
        return out
    l0, nx, ny = case["l0"], case["cols"], case["rows"]
    w, h = nx * l0, ny * l0
    scene = case.get("scene", "hydro")
    if scene == "box":
        return _deform(_box(nx, ny, l0), (w, h, w), rng)
    if scene == "hydro":
        s = scenes.hydrostatic(l0, size=(w, h), dt=0.1 * l0, margin=20 * l0)
    else:
        s = scenes.dam_break(l0, tank=(4 * w, math.ceil(1.2 * ny) * l0), column=(w, h), dt=0.1 * l0,
                             margin=20 * l0)
    if scene == "shaken":
        return scenes.shaken(s, seed=int(rng.integers(1 << 30)))
    return _deform(s, (w, h, 1.0), rng)


def _pinned(shape, dtype=torch.float64):
    return torch.zeros(shape, dtype=dtype, pin_memory=torch.cuda.is_available()).numpy()


def _host_state(scene):
    """A program's particle arrays: inputs and results, in pinned memory."""
    _, pos, vel, t = scene
    n = len(t)
    inp = dict(pos=_pinned((n, 3)), vel=_pinned((n, 3)), types=_pinned(n, torch.int32))
    inp["pos"][:], inp["vel"][:], inp["types"][:] = pos, vel, t
    res = dict(pos=_pinned((n, 3)), vel=_pinned((n, 3)), pressure=_pinned(n),
               types=_pinned(n, torch.int32), bc=_pinned(n, torch.int32))
    return inp, res


def prepare(case, seed):
    scene = _scene(case, seed)
    if case["kind"] == "batch":
        # the scenes' particles one after another in one set of arrays
        inp, res = _host_state((None,) + tuple(np.concatenate([s[q] for s in scene]) for q in (1, 2, 3)))
        at = np.cumsum([0] + [len(s[3]) for s in scene])
        part = [{k: v[a:b] for k, v in inp.items()} for a, b in zip(at, at[1:])]
        into = [{k: v[a:b] for k, v in res.items()} for a, b in zip(at, at[1:])]
        return dict(case=case, batch=Batch(scene, tol=TOL), inp=part, into=into, res=res)
    if case["kind"] == "adjoint":
        prm, pos, vel, t = scene
        rng = np.random.default_rng(seed + 1)
        e = Engine(prm, pos, vel, t, precision=FP64)
        taps = scenes.wall_taps(pos, t, prm["particle_distance"], min(16, case["cols"]))
        s, target = case["steps"], rng.normal(0, 1, (2,) + pos.shape) * [1, 1, 0]
        return dict(case=case, vel=vel, trajectory=Trajectory(e, s, case["every"], taps),
                    d_sensor=rng.normal(0, 1e-3, (s, len(taps))), d_pos=target[0], d_vel=target[1])
    inp, res = _host_state(scene)
    e = Engine(*scene) if case["precision"] == "fp64" else Engine(*scene, precision=MIXED, tol=TOL)
    return dict(case=case, engine=e, inp=inp, res=res)


def run(s):
    case, k = s["case"], s["case"]["steps"]
    if case["kind"] == "batch":
        b = s["batch"]
        for i, inp in enumerate(s["inp"]):
            b.scene(i).upload(**inp)
        b.step(k)
        for i, into in enumerate(s["into"]):
            b.scene(i).download_into(**into)
        return s["res"]
    if case["kind"] == "adjoint":
        t = s["trajectory"]
        sensor, pos, vel = t.forward(vel0=s["vel"])
        gpos, gvel, gg = t.backward(s["d_sensor"], s["d_pos"], s["d_vel"])
        return dict(sensor=sensor, pos=pos, vel=vel, d_pos0=gpos, d_vel0=gvel, d_gravity=gg)
    e = s["engine"]
    e.upload(**s["inp"])
    if case["call"] == "export":
        e.run_report(k - 1)
        e.step(export=True)
        e.export_begin()
        return e.export_snapshot()
    if case["call"] == "step":
        for _ in range(k):
            e.step()
    else:
        e.run_report(k)
    e.download_into(**s["res"])
    return s["res"]


def work(case):
    """Particles in (52 B) and out (64 B); per step and pair of neighbours the weights,
    the viscosity, matrix and gradient terms once, ~60 operations."""
    if case["kind"] == "batch":
        n = case["count"] * 0.5 * (case["low"] + case["high"])
    else:
        n = case["cols"] * case["rows"] * (case["cols"] if case.get("scene") == "box" else 1)
    pairs = 120 if case.get("scene") == "box" else 28
    both = 3 if case["kind"] == "adjoint" else 1
    return {"bytes": 116.0 * n * both, "flops": 60.0 * n * pairs * case["steps"] * both}


# ------------------------------------------------- the step in 64-bit torch


def _lattice_sums(dim, l0, re):
    r = np.arange(-4, 5) * l0
    z = r if dim == 3 else np.zeros(1)
    d = np.sqrt(sum(a * a for a in np.meshgrid(r, r, z, indexing="ij"))).ravel()
    d = d[(d > 0) & (d < re)]
    w = re / d - 1
    return w.sum(), (d * d * w).sum() / w.sum()


def _pairs(pos, ghost, lo, re):
    """All ordered pairs (i, j) nearer than re, from a grid of cells of edge re."""
    pos = pos.detach()
    dim = pos.shape[1]
    cell = ((pos - lo) / re).floor().long() + 2
    m = [int(v) + 3 for v in cell.max(0).values]
    cell[ghost] = 0
    key = cell[:, 0] * m[1] + cell[:, 1]
    if dim == 3:
        key = key * m[2] + cell[:, 2]
    skey, order = key.sort()
    around = [(a,) for a in (-1, 0, 1)] if dim == 2 else [(a, b) for a in (-1, 0, 1) for b in (-1, 0, 1)]
    found = []
    for c0 in range(0, len(pos), 1 << 18):
        rows = torch.arange(c0, min(c0 + (1 << 18), len(pos)), device=pos.device)
        rows = rows[~ghost[rows]]
        for o in around:
            mid = key[rows] + (o[0] * m[1] if dim == 2 else (o[0] * m[1] + o[1]) * m[2])
            first = torch.searchsorted(skey, mid - 1)
            count = torch.searchsorted(skey, mid + 1, right=True) - first
            i = rows.repeat_interleave(count)
            j = torch.arange(len(i), device=pos.device) - (count.cumsum(0) - count - first).repeat_interleave(count)
            j = order[j]
            near = (i != j) & ((pos[i] - pos[j]).square().sum(1).sqrt() < re)
            found.append((i[near], j[near]))
    return torch.cat([f[0] for f in found]), torch.cat([f[1] for f in found])


def _cg(A, inv, b):
    """A x = b: Jacobi CG to 1e-13, then its residual's own solve added."""
    x = torch.zeros_like(b)
    for tol in (1e-13, 1e-7):
        r = b - A @ x
        stop = tol * float(b.norm() if tol < 1e-10 else r.norm())
        if stop == 0:
            return x
        d, z = torch.zeros_like(b), inv * r
        p, rz = z.clone(), r @ z
        for k in range(40000):
            q = A @ p
            a = rz / (p @ q)
            d += a * p
            r -= a * q
            if k % 20 == 19 and float(r.norm()) <= stop:
                break
            z = inv * r
            new = r @ z
            p = z + (new / rz) * p
            rz = new
        x = x + d
    return x


class _Solve(torch.autograd.Function):
    """x of (diag, off on the pattern (i, j)) x = b over m unknowns; A is symmetric."""

    @staticmethod
    def forward(ctx, i, j, off, diag, b):
        m = len(b)
        at = torch.arange(m, device=b.device)
        row, col, val = torch.cat([i, at]), torch.cat([j, at]), torch.cat([off, diag])
        o = torch.argsort(row * m + col)
        ptr = torch.zeros(m + 1, dtype=torch.long, device=b.device)
        ptr[1:] = torch.bincount(row, minlength=m).cumsum(0)
        A = torch.sparse_csr_tensor(ptr, col[o], val[o], (m, m))
        x = _cg(A, 1 / diag, b)
        ctx.A, ctx.inv = A, 1 / diag
        ctx.save_for_backward(i, j, x)
        return x

    @staticmethod
    def backward(ctx, g):
        i, j, x = ctx.saved_tensors
        lam = _cg(ctx.A, ctx.inv, g)
        return None, None, -lam[i] * x[j], -lam * x, lam


def _collide(prm, pos, vel, t, i, j, dist, lo, re):
    """The collision pass: candidates by particle, in the order of its cell sweep, one after another."""
    cd = prm["collision_distance"]
    c = (dist < cd) & (t[i] == FLUID) & ((t[j] != FLUID) | (j < i))
    if not bool(c.any()):
        return pos, vel
    i, j, dist = i[c], j[c], dist[c]
    cell = ((pos[j] - lo) / re).floor().long().cpu().numpy()
    i, j, dist = (v.cpu().numpy() for v in (i, j, dist))
    order = np.lexsort((j, *(cell[:, a] for a in reversed(range(cell.shape[1]))), i))
    x, v, ty = pos.cpu().numpy(), vel.cpu().numpy(), t.cpu().numpy()
    for a, b, d in zip(i[order].tolist(), j[order].tolist(), dist[order].tolist()):
        ia, ib = 1 / prm["density"], (1 / prm["density"] if ty[b] == FLUID else 0.0)
        red = 1 / (ia + ib)
        e = x[b] - x[a]
        e = e / math.sqrt(float(e @ e))
        rel = float((v[b] - v[a]) @ e)
        if rel < 0:
            imp, push = -(1 + prm["restitution"]) * rel * red, (cd - d) * red
            v[a] -= imp * ia * e
            v[b] += imp * ib * e
            x[a] -= push * ia * e
            x[b] += push * ib * e
    return torch.from_numpy(x).to(pos.device), torch.from_numpy(v).to(pos.device)


def _step(prm, g, pos, vel, t):
    """One time step on float64 tensors (n, dim): new positions, velocities, types, and the pressure."""
    n, dim = pos.shape
    dt, rho = prm["dt"], prm["density"]
    re_p, re_v, re_s = prm["re_pressure"], prm["re_viscosity"], prm["re_surface"]
    re = max(re_p, re_v, re_s)
    (n0p, lamp), (n0v, lamv), (n0s, _) = (_lattice_sums(prm["dim"], prm["particle_distance"], r)
                                          for r in (re_p, re_v, re_s))
    lo, hi = (torch.tensor(prm[q][:dim], dtype=pos.dtype, device=pos.device) for q in ("domain_min", "domain_max"))

    def add(i, v):
        return torch.zeros((n,) + v.shape[1:], dtype=v.dtype, device=v.device).index_add(0, i, v)

    def length(i, j, x):
        return (x[j] - x[i]).square().sum(1).sqrt()

    def inside(x, t):
        out = ((x < lo) | (x > hi)).any(1) & (t == FLUID)
        return torch.where(out, torch.full_like(t, GHOST), t)

    # explicit part
    fluid = (t == FLUID)[:, None]
    i, j = _pairs(pos, t == GHOST, lo, re)
    k = t[i] == FLUID
    i, j = i[k], j[k]
    d = length(i, j, pos)
    k = d < re_v
    i, j, d = i[k], j[k], d[k]
    lap = add(i, (vel[j] - vel[i]) * (re_v / d - 1)[:, None])
    acc = g + lap * (prm["kinematic_viscosity"] * 2 * prm["dim"] / (n0v * lamv))
    vel = torch.where(fluid, vel + acc * dt, vel)
    pos = torch.where(fluid, pos + vel * dt, pos)
    t = inside(pos, t)
    # collisions
    if not pos.requires_grad:
        i, j = _pairs(pos, t == GHOST, lo, re)
        pos, vel = _collide(prm, pos, vel, t, i, j, length(i, j, pos), lo, re)
    # boundary condition, source, matrix
    i, j = _pairs(pos, t == GHOST, lo, re)
    d = length(i, j, pos)
    s = d.detach() < re_s
    ns = add(i[s], re_s / d.detach()[s] - 1)
    ignored = (t == GHOST) | (t == DUMMY)
    surface = ~ignored & (ns < prm["surface_threshold"] * n0s)
    inner = ~ignored & ~surface
    k = d.detach() < re_p
    i, j, d = i[k], j[k], d[k]
    w = re_p / d - 1
    src = prm["relaxation"] / (dt * dt) * (add(i, w) - n0p) / n0p
    flag, before = surface.clone(), -1
    while (now := int(flag.sum())) != before:
        before = now
        for _ in range(16):
            flag[j[flag[i]]] = True
    k = inner[i] & ~ignored[j]
    a = (2 * prm["dim"] / (lamp * n0p)) / rho * w[k]
    diag = add(i[k], a) + prm["compressibility"] / (dt * dt)
    diag = torch.where(flag, diag, 2 * diag)
    u = inner.nonzero()[:, 0]
    at = torch.zeros(n, dtype=torch.long, device=pos.device)
    at[u] = torch.arange(len(u), device=pos.device)
    both = inner[j[k]]
    x = _Solve.apply(at[i[k]][both], at[j[k]][both], -a[both], diag[u], src[u])
    p = torch.zeros(n, dtype=pos.dtype, device=pos.device).index_put((u,), x).clamp(min=0)
    # minimum pressure, gradient, move
    k = (t[i] == FLUID) & (t[j] != DUMMY)
    i, j, d, w = i[k], j[k], d[k], w[k]
    low = p.scatter_reduce(0, i, p[j], "amin")
    grad = add(i, (pos[j] - pos[i]) * ((p[j] - low[i]) * w / (d * d))[:, None]) * (prm["dim"] / n0p)
    acc = -grad / rho
    fluid = (t == FLUID)[:, None]
    vel = torch.where(fluid, vel + acc * dt, vel)
    pos = torch.where(fluid, pos + acc * dt * dt, pos)
    return pos, vel, inside(pos, t), p, surface


def _march(scene, steps, grad=False):
    prm, pos, vel, t = scene
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    dim = prm["dim"]
    x0, v0, g = (torch.tensor(np.asarray(a, np.float64)[..., :dim], device=dev, requires_grad=grad)
                 for a in (pos, vel, prm["gravity"]))
    x, v, t, taps = x0, v0, torch.tensor(t, device=dev), []
    for _ in range(steps):
        x, v, t, p, surface = _step(prm, g, x, v, t)
        taps.append(p)
    return (x0, v0, g), x, v, t, taps, surface


def _full(a, rest=0.0):
    """(n, dim) -> (n, 3) on the host."""
    a = a.detach().cpu().numpy()
    out = np.full(a.shape[:-1] + (3,), rest)
    out[..., :a.shape[-1]] = a
    return out


def exact(case, seed):
    scene = _scene(case, seed)
    if case["kind"] == "adjoint":
        prm, pos, _, t = scene
        rng = np.random.default_rng(seed + 1)
        taps = scenes.wall_taps(pos, t, prm["particle_distance"], min(16, case["cols"]))
        target = rng.normal(0, 1, (2,) + pos.shape)
        dsens = torch.tensor(rng.normal(0, 1e-3, (case["steps"], len(taps))))
        (x0, v0, g), x, v, _, ps, _ = _march(scene, case["steps"], grad=True)
        sensor = torch.stack([p[torch.tensor(taps.astype(np.int64), device=p.device)] for p in ps])
        dx, dv = (torch.tensor(a[:, :2], device=x.device) for a in target)
        ((sensor * dsens.to(x.device)).sum() + (x * dx).sum() + (v * dv).sum()).backward()
        return dict(sensor=sensor.detach().cpu().numpy(), pos=_full(x), vel=_full(v), d_pos0=_full(x0.grad),
                    d_vel0=_full(v0.grad), d_gravity=_full(g.grad))
    with torch.no_grad():
        if case["kind"] == "batch":
            out = [_march(s, case["steps"]) for s in scene]
            return dict(pos=np.concatenate([_full(o[1]) for o in out]), vel=np.concatenate([_full(o[2]) for o in out]),
                        pressure=np.concatenate([o[4][-1].cpu().numpy() for o in out]))
        prm = scene[0]
        _, x, v, t, ps, surface = _march(scene, case["steps"])
        res = dict(pos=_full(x), vel=_full(v), pressure=ps[-1].cpu().numpy())
        if case["call"] == "export":
            dim = prm["dim"]
            lo = torch.tensor(prm["domain_min"][:dim], dtype=x.dtype, device=x.device)
            i, j = _pairs(x, t == GHOST, lo, prm["re_pressure"])
            w = prm["re_pressure"] / (x[j] - x[i]).square().sum(1).sqrt() - 1
            nd = torch.zeros(len(x), dtype=x.dtype, device=x.device).index_add(0, i, w)
            nd /= _lattice_sums(dim, prm["particle_distance"], prm["re_pressure"])[0]
            res["ndr"] = torch.where(surface, torch.zeros_like(nd), nd).cpu().numpy()
        return res
