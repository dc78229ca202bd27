"""The solves of small scenes with positive pressures: blocks of fluid squeezed to 0.94 of
the particle distance, of 25 to 9,000 particles, on both sides of a slice (32 rows), of the
one-cluster FP64 form's line (4,000 rows), of the mixed cluster's (8,000) and of one slice
per block (152 slices).  Against a sparse direct solve of the assembled system, with the
tolerances of the larger scenes' tests: 1e-9 for FP64 (condition numbers up to 1e4 here),
1e-6 for the mixed solver's relative residual of 1e-10.
"""
import numpy as np
import pytest

from gpu_util import engine_or_skip, rel_l2
from mps_gb300 import scenes

pytestmark = pytest.mark.gpu
L0 = 0.01


def block(n):
    side = int(np.ceil(np.sqrt(n)))
    g = np.stack(np.meshgrid(np.arange(side), np.arange(side), indexing="ij"), -1).reshape(-1, 2)[:n]
    pos = np.zeros((n, 3))
    pos[:, :2] = (g + 0.5) * L0 * 0.94
    m = 8 * L0
    prm = scenes.baseline_physics(L0, 0.1 * L0, (-m, -m, 0.0), (side * L0 + m, side * L0 + m, 0.0))
    return prm, pos, np.zeros_like(pos), np.full(n, scenes.FLUID, np.int32)


@pytest.mark.parametrize("n", [25, 31, 32, 33, 64, 100, 513, 2000, 3999, 4000, 4001, 4864, 4865, 8000, 8001, 9000])
def test_positive_pressures(n):
    m = engine_or_skip()
    sp = pytest.importorskip("scipy.sparse")
    from scipy.sparse.linalg import spsolve

    for prec, tol in ((m.FP64, 1e-9), (m.MIXED, 1e-6)):
        e = m.Engine(*block(n), precision=prec)
        e.step()
        src, rp, col, val = e.system()
        p = e.state()["pressure"]
        e.close()
        rows = np.flatnonzero(np.diff(rp) > 0)
        A = sp.csr_matrix((val, col, rp), shape=(n, n))[rows][:, rows].tocsc()
        x = np.zeros(n)
        x[rows] = spsolve(A, src[rows])
        assert len(rows) > 0 and x.max() > 0 and (x[rows] > 0).mean() > 0.5
        assert rel_l2(p, np.maximum(x, 0.0)) < tol
