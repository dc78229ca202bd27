"""The split sweeps (one warp per slot range, up to 20,000 particles) give the bits of one
thread per particle, in both precisions: the terms are added in list order.

Viscosity: a scene without pressure (relaxation 0: no source), so that the step's
velocities are those of the explicit part (and the collisions), against the same scene
above the line.  Pressure gradient: fluid at rest without gravity, so that the velocity
after the step is the gradient's; against the sums in numpy in list order from the
engine's own pressures, on both sides of the line.
"""
import numpy as np
import pytest

from gpu_util import engine_or_skip
from mps_gb300 import scenes
from test_gpu_sweep_split import L0, LINE, above_the_line, box, planar

pytestmark = pytest.mark.gpu
f4 = np.float32


def still(scene):
    """No source, and a viscosity that changes velocities of 0.1 m/s by some per cent."""
    prm, pos, vel, t = scene
    return dict(prm, relaxation=0.0, kinematic_viscosity=0.02), pos, vel, t


@pytest.mark.parametrize("scene", [planar(5, 3), planar(40, 30), planar(135, 125), box(3), box(12), box(27),
                                   box(14, 0.8)],
                         ids=["p5x3", "p40x30", "p135x125", "b3", "b12", "b27", "bdense"])
def test_viscosity_bits(scene):
    m = engine_or_skip()
    scene = still(scene)
    n = len(scene[3])
    assert n <= LINE
    for prec in (m.FP64, m.MIXED):
        got = []
        for s in (scene, above_the_line(scene)):
            e = m.Engine(*s, precision=prec)
            e.step()
            got.append(e.state())
            e.close()
        a, b = got
        assert not a["pressure"].any() and not b["pressure"].any()
        assert np.max(np.abs(a["vel"] - scene[2])) > 1e-4
        assert np.array_equal(a["vel"], b["vel"][:n])
        assert np.array_equal(a["pos"], b["pos"][:n])


def at_rest(scene, squeeze, seed):
    prm, pos, vel, t = scene
    pos, rng = pos.copy(), np.random.default_rng(seed)
    f, d = t == scenes.FLUID, 3 if prm["dim"] == 3 else 2
    pos[f, :d] += rng.uniform(-0.1, 0.1, (f.sum(), d)) * L0
    pos[f, 1] *= squeeze
    prm = dict(prm, gravity=[0.0, 0.0, 0.0], collision_distance=0.2 * L0)
    return prm, pos, np.zeros_like(vel), t


def n0_of(dim, re):
    r = range(-4, 5)
    n0 = 0.0
    for ix in r:
        for iy in r:
            for iz in (r if dim == 3 else (0,)):
                if ix or iy or iz:
                    x, y, z = L0 * ix, L0 * iy, L0 * iz
                    dist = np.sqrt((x * x + y * y) + z * z)
                    n0 += re / dist - 1.0 if dist < re else 0.0
    return n0


def gradient(scene, p, off, nb, dist, mixed):
    """Velocities after the step, by list column; p: the pressures it ended with."""
    prm, pos, _, t = scene
    n, re, is3 = len(t), prm["re_pressure"], prm["dim"] == 3
    cnt = np.diff(off)
    q = off[:-1, None] + np.minimum(np.arange(cnt.max()), np.maximum(cnt - 1, 0)[:, None])
    q = np.minimum(q, len(nb) - 1)
    J, D = nb[q], dist[q]
    on = (np.arange(cnt.max()) < cnt[:, None]) & (D < re) & (t[J] != scenes.DUMMY)
    pmin = np.minimum(p, np.min(np.where(on, p[J], np.inf), axis=1))
    scale = float(prm["dim"]) / n0_of(prm["dim"], re)
    rho, dt = prm["density"], prm["dt"]
    v = np.zeros((n, 3))
    if mixed:
        fd = D.astype(f4)
        if is3:
            dp = (p[J] - pmin[:, None]).astype(f4)
        else:
            hi, mh = p.astype(f4), pmin.astype(f4)
            lo, ml = (p - hi).astype(f4), (pmin - mh).astype(f4)
            dp = (hi[J] - mh[:, None]) + (lo[J] - ml[:, None])
        coef = dp * (f4(re) / fd - f4(1)) / (fd * fd)
        sc = -f4(scale) / f4(rho)
    for d in range(3 if is3 else 2):
        x = pos[:, d]
        if mixed:
            if is3:
                dx = (x[J] - x[:, None]).astype(f4)
            else:
                h = x.astype(f4)
                l = (x - h).astype(f4)
                dx = (h[J] - h[:, None]) + (l[J] - l[:, None])
            s = np.zeros(n, f4)
            for c in range(J.shape[1]):  # (FP64's second rounding differs once in 2^29)
                s = np.where(on[:, c], (np.float64(dx[:, c]) * coef[:, c] + np.float64(s)).astype(f4), s)
            a = np.float64(s * sc)
        else:
            s = np.zeros(n)
            w, d2 = re / D - 1.0, D * D
            terms = ((x[J] - x[:, None]) * (p[J] - pmin[:, None])) * w / d2
            for c in range(J.shape[1]):
                s = s + np.where(on[:, c], terms[:, c], 0.0)
            a = (-1.0 * (s * scale)) / rho
        v[:, d] = np.where(t == scenes.FLUID, a * dt, 0.0)
    return v


@pytest.mark.parametrize("scene", [at_rest(planar(40, 30), 0.97, 1), at_rest(planar(130, 120), 0.99, 2),
                                   at_rest(box(12, 0.9), 1.0, 3), at_rest(box(26, 0.95), 1.0, 4)],
                         ids=["p40x30", "p130x120", "b12", "b26"])
@pytest.mark.parametrize("above", [False, True])
def test_gradient_bits(scene, above):
    m = engine_or_skip()
    n = len(scene[3])
    for prec in (m.FP64, m.MIXED):
        s = above_the_line(scene) if above else scene
        e = m.Engine(*s, precision=prec)
        e.step()
        got, (off, nb, dist) = e.state(), e.neighbors()
        e.close()
        want = gradient(s, got["pressure"], off, nb, dist, prec == m.MIXED)
        assert (got["pressure"] > 0).sum() > 100
        moved = np.abs(got["vel"][:n]).max(axis=1) > 0
        assert moved.sum() > 100
        assert np.array_equal(got["vel"][:n], want[:n])
