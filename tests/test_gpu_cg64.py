"""The FP64 pressure solve (cg64.cu) over its row distributions: one partial
slice, one slice per block, several resident slices per block, streamed rows
(512 and 1024 threads), and a grid whose windows no longer fit (gathered).

Tolerances: CG in FP64 on these matrices (condition number up to ~1e6 for the
deepest tank) leaves an error of at most ~1e6 * 2^-52 = 2e-10 relative; 1e-9 is
asked for.  The mixed solver stops at a relative residual of 1e-10; on the
shallow wide tank (condition number ~1e4) the pressures agree to 1e-6.
"""
import numpy as np
import pytest

from gpu_util import engine_or_skip, rel_l2
from mps_gb300 import scenes

pytestmark = pytest.mark.gpu


def compressed_tank(cols, rows, strain=1e-3, l0=0.01):
    prm, pos, vel, t = scenes.hydrostatic(l0, size=(cols * l0, rows * l0), dt=0.1 * l0, margin=10 * l0)
    fluid = t == scenes.FLUID
    pos[fluid, 1] *= 1.0 - strain
    return prm, pos, vel, t


@pytest.mark.parametrize("cols,rows", [(2, 2), (3, 5), (7, 16), (30, 31), (64, 75), (150, 141), (240, 250), (1400, 110)])
def test_pressure_solves_the_assembled_system(cols, rows):
    m = engine_or_skip()
    sp = pytest.importorskip("scipy.sparse")
    from scipy.sparse.linalg import spsolve

    prm, pos, vel, t = compressed_tank(cols, rows)
    e = m.Engine(prm, pos, vel, t)
    e.step()
    src, rp, col, val = e.system()
    p = e.state()["pressure"]
    e.close()
    n = len(t)
    A = sp.csr_matrix((val, col, rp), shape=(n, n))
    rows_in = np.flatnonzero(np.diff(rp) > 0)
    x = np.zeros(n)
    if len(rows_in):
        x[rows_in] = spsolve(A[rows_in][:, rows_in].tocsc(), src[rows_in])
    assert rel_l2(p, np.maximum(x, 0.0)) < 1e-9


@pytest.mark.parametrize("cols", [72000, 110000])
def test_wide_tank_against_mixed(cols):
    """~3.3M rows: windows close to the shared memory; ~4.6M: gathered."""
    m = engine_or_skip()
    scene = compressed_tank(cols, 38, strain=2e-3)
    got = []
    for prec in (m.FP64, m.MIXED):
        e = m.Engine(*scene, precision=prec)
        e.step()
        got.append(e.state())
        e.close()
    assert got[0]["pressure"].max() > 0
    assert np.array_equal(got[0]["bc"], got[1]["bc"])
    assert rel_l2(got[1]["pressure"], got[0]["pressure"]) < 1e-6
