"""The sweeps with one warp per slot range (up to 20,000 particles) against those
with one thread per particle: a scene, and the same scene with isolated dummies far
away that put it above the line.  FP64: lists, distances, sources, flags and collision
pairs are exact in both forms, so they are identical.  Mixed: the forms add FP32
terms in another order, some hundred of them at 6e-8 each, which partly cancel:
1e-5 of the step's largest displacement, and 1e-9 m; the solves stop at a relative
residual of 1e-10 (pressures: 1e-6).
"""
import numpy as np
import pytest

from gpu_util import engine_or_skip, rel_l2
from mps_gb300 import scenes

pytestmark = pytest.mark.gpu
LINE = 20000
L0 = 0.01


def planar(cols, rows):
    return scenes.shaken(scenes.hydrostatic(L0, size=(cols * L0, rows * L0), dt=0.1 * L0, margin=8 * L0), jitter=0.3)


def box(side, squeeze=1.0):
    """A jittered cube of fluid in a domain of its own, y up; squeeze < 1: denser."""
    g = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)
    rng = np.random.default_rng(side)
    pos = (g + 0.5 + rng.uniform(-0.1, 0.1, g.shape)) * L0 * squeeze
    m = 8 * L0
    prm = scenes.baseline_physics(L0, 0.1 * L0, (-m, -m, -m), (side * L0 + m,) * 3)
    prm["dim"] = 3
    return prm, pos, rng.normal(0.0, 0.1, pos.shape), np.full(len(pos), scenes.FLUID, np.int32)


def above_the_line(scene):
    """The scene first, then isolated dummies in a domain that grows along x only (cell
    keys are x-major: the scene's cells keep theirs)."""
    prm, pos, vel, t = scene
    prm = dict(prm, domain_max=list(prm["domain_max"]))
    k = np.arange(max(LINE + 1 - len(t), 1))
    lo, hi = np.asarray(prm["domain_min"]), np.asarray(prm["domain_max"])
    per = int((hi[1] - lo[1] - 8 * L0) / (4 * L0))
    far = np.zeros((len(k), 3))
    far[:, 0] = hi[0] + (4 + 4 * (k // per)) * L0
    far[:, 1] = lo[1] + (4 + 4 * (k % per)) * L0
    prm["domain_max"][0] = far[:, 0].max() + 8 * L0
    return (prm, np.concatenate([pos, far]), np.concatenate([vel, 0 * far]),
            np.concatenate([t, np.full(len(k), scenes.DUMMY, np.int32)]))


@pytest.mark.parametrize("scene", [planar(1, 1), planar(5, 3), planar(40, 30), planar(135, 125), box(1), box(3), box(12),
                                   box(27), box(14, 0.8)],
                         ids=["p1", "p5x3", "p40x30", "p135x125", "b1", "b3", "b12", "b27", "dense"])
def test_same_as_one_thread_per_particle(scene):
    m = engine_or_skip()
    n = len(scene[3])
    assert n <= LINE
    for prec in (m.FP64, m.MIXED):
        got = []
        for s in (scene, above_the_line(scene)):
            e = m.Engine(*s, precision=prec)
            e.step()
            got.append((e.state(), e.neighbors(), e.system()[0], e.collisions()))
            e.close()
        (a, la, sa, ca), (b, lb, sb, cb) = got
        # the step's last move takes particles of the dense box out of the scene's own domain
        out = b["pos"][:n, 0] > scene[0]["domain_max"][0]
        assert np.array_equal(a["type"], np.where(out, scenes.GHOST, b["type"][:n]))
        for key in ("bc", "dirichlet"):
            assert np.array_equal(a[key], b[key][:n]), key
        assert np.array_equal(la[0], lb[0][:n + 1])
        last = la[0][-1]
        assert np.array_equal(la[1], lb[1][:last])
        assert np.array_equal(ca[0], cb[0]) and np.array_equal(ca[1], cb[1])
        if prec == m.FP64:
            assert np.array_equal(la[2], lb[2][:last])
            assert np.array_equal(sa, sb[:n])
            assert np.array_equal(ca[2], cb[2])
        else:
            moved = np.max(np.abs(a["pos"] - scene[1]))
            assert np.max(np.abs(a["pos"] - b["pos"][:n])) < 1e-9 + 1e-5 * moved
            assert rel_l2(b["pressure"][:n], a["pressure"]) < 1e-6 or not a["pressure"].any()
