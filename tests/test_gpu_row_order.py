"""The mixed solver's operator rows without the compact form (3-D scenes) add their
entries one after another in the order of the neighbour list, whatever number of warps
shares a row: two inner iterations from a zero start, against the same iterations in
numpy.  Element by element the iteration is FP32 with fused multiply-adds (made here
in FP64, whose second rounding differs once in 2^29), and its scalars come from FP32
sums exact to 2^-44, here FP64 sums; so x32 has the same bits, and x = ||b|| x32
agrees to the rounding of ||b||: 1e-12 of the largest.  Sums in another order differ
by 6e-8 of a row's terms.
"""
import numpy as np
import pytest

from gpu_util import engine_or_skip
from mps_gb300 import scenes
from test_gpu_sweep_split import L0, box

pytestmark = pytest.mark.gpu
f4, f8 = np.float32, np.float64


def fma(a, b, c):
    return (f8(a) * f8(b) + f8(c)).astype(f4)


def two_iterations(e, n, prm):
    src, rp, col, val = e.system()
    off, nb, dist = e.neighbors()
    state = e.state()
    re = prm["re_pressure"]
    A = {}
    diag = np.zeros(n)
    for i in range(n):
        for q in range(rp[i], rp[i + 1]):
            A[i, col[q]] = val[q]
        diag[i] = A.get((i, i), 0.0)
    rows = [[j for j, d in zip(nb[off[i]:off[i + 1]], dist[off[i]:off[i + 1]]) if d < re and (i, j) in A]
            if diag[i] > 0 else [] for i in range(n)]
    width = max(map(len, rows))
    J = np.array([r + [i] * (width - len(r)) for i, r in enumerate(rows)], dtype=np.int64)
    V = np.array([[A[i, j] for j in r] + [0.0] * (width - len(r)) for i, r in enumerate(rows)]).astype(f4)
    on = diag > 0
    assert state["dirichlet"][:n][on].all() and width > 32
    # the row sum: the terms of the neighbours without an unknown (surface particles here)
    i0 = int(np.flatnonzero(on)[0])
    j0 = rows[i0][0]
    c = -A[i0, j0] / (re / dist[off[i0] + list(nb[off[i0]:off[i0 + 1]]).index(j0)] - 1.0)
    rsum = np.full(n, prm["compressibility"] / prm["dt"] ** 2)
    for i in np.flatnonzero(on):
        rsum[i] += sum(c * (re / d - 1.0) for j, d in zip(nb[off[i]:off[i + 1]], dist[off[i]:off[i + 1]])
                       if d < re and (i, j) not in A)
    rsum = rsum.astype(f4)
    inv = np.where(on, 1.0 / np.where(on, diag, 1.0), 1.0).astype(f4)
    norm = np.sqrt(np.sum(src[:n] ** 2))
    r = src[:n].astype(f4) * f4(1.0 / norm)
    x, p, s = np.zeros(n, f4), np.zeros(n, f4), np.zeros(n, f4)
    u = inv * r
    beta, alpha, gamma_old = f4(0), f4(0), f4(1)
    for k in range(2):
        o = np.zeros(n, f4)
        for m in range(width):
            o = fma(V[:, m], u[J[:, m]] - u, o)
        w = np.where(on, fma(rsum, u, o), f4(0))
        gamma, delta = f4(np.sum(f8(r) * u)), f4(np.sum(f8(w) * u))
        if k == 0:
            alpha = gamma / delta
        else:
            beta = gamma / gamma_old
            alpha = gamma / (delta - beta * gamma / alpha)
        gamma_old = gamma
        p, s = fma(beta, p, u), fma(beta, s, w)
        x, r = fma(alpha, p, x), fma(-alpha, s, r)
        u = inv * r
    return norm * f8(x)


def filled(scene, count):
    """The scene first, then isolated dummies up to `count` particles, beyond the scene along x."""
    prm, pos, vel, t = scene
    prm = dict(prm, domain_max=list(prm["domain_max"]))
    k = np.arange(count - len(t))
    if not len(k):
        return scene
    per = 12
    prm["domain_max"][1] = max(prm["domain_max"][1], prm["domain_min"][1] + 4 * (per + 2) * L0)
    far = np.zeros((len(k), 3))
    far[:, 0] = prm["domain_max"][0] + (4 + 4 * (k // per)) * L0
    far[:, 1] = prm["domain_min"][1] + (4 + 4 * (k % per)) * L0
    prm["domain_max"][0] = far[:, 0].max() + 8 * L0
    return (prm, np.concatenate([pos, far]), np.concatenate([vel, 0 * far]),
            np.concatenate([t, np.full(len(k), scenes.DUMMY, np.int32)]))


def check(e, n, prm, p):
    x = np.maximum(two_iterations(e, n, prm), 0.0)
    assert (x > 0).sum() > 100
    assert np.max(np.abs(p[:n] - x)) <= 1e-12 * x.max()


# eight, four and two warps per slice of 32 rows, and one
@pytest.mark.parametrize("count", [1000, 25000, 50000, 90000])
def test_rows_add_in_list_order(count):
    m = engine_or_skip()
    from mps_gb300.engine import MPS_ERR_NOT_CONVERGED, MpsError

    scene = box(10, 0.9)
    e = m.Engine(*filled(scene, count), precision=m.MIXED, max_iter=2)
    with pytest.raises(MpsError) as ex:
        e.step()
    assert ex.value.code == MPS_ERR_NOT_CONVERGED
    check(e, len(scene[3]), scene[0], e.state()["pressure"])
    e.close()


@pytest.mark.parametrize("block,alpha", [(256, 0.0), (256, 3.0), (512, 1.25), (1024, 0.0), (1024, 3.0)])
def test_rows_of_a_batch_add_in_list_order(block, alpha):
    """A 3-D scene beside a planar one and a larger one (alpha: the blocks' shares, down to
    one block for the first scene)."""
    m = engine_or_skip()
    from mps_gb300.engine import MpsError

    some = [box(10, 0.9), scenes.hydrostatic(L0, size=(0.3, 0.2), dt=0.1 * L0, margin=8 * L0), box(20, 0.9)]
    b = m.Batch(some, max_iter=2)
    b.set_launch(block, alpha)
    with pytest.raises(MpsError):
        b.step()
    e = b.scene(0)
    check(e, len(some[0][3]), some[0][0], e.state()["pressure"])
    b.close()
