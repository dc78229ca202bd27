"""The mixed solver's split V-cycle over its forms: one cluster (every level in
every block's shared memory), grid-wide with shared coarse levels, patches that
do not fit and live in global memory (two bodies of water at the ends of a very
wide domain), and the streaming form above 150,000 rows.  Against the FP64 solver
from the same state: the mixed solve stops at a relative residual of 1e-10 and
its FP32 sums round at 6e-8, so pressures agree to 1e-6 and surface flags are
identical.
"""
import numpy as np
import pytest

from gpu_util import engine_or_skip, rel_l2
from mps_gb300 import scenes

pytestmark = pytest.mark.gpu


def column(cols, rows, l0=0.01, gap=0):
    """A compressed column in its tank; gap > 0: a second one `gap` particle distances to the right."""
    prm, pos, vel, t = scenes.hydrostatic(l0, size=(cols * l0, rows * l0), dt=0.1 * l0, margin=12 * l0)
    pos[t == scenes.FLUID, 1] *= 0.998
    if gap:
        other = pos + [gap * l0, 0.0, 0.0]
        pos, vel, t = np.concatenate([pos, other]), np.concatenate([vel, vel]), np.concatenate([t, t])
        prm["domain_max"][0] += gap * l0
        prm["domain_max"][1] += gap * l0  # the empty cells above count as well
    return prm, pos, vel, t


@pytest.mark.parametrize("cols,rows,gap", [(3, 4, 0), (40, 31, 0), (150, 145, 0), (160, 150, 0), (20, 25, 600),
                                           (60, 50, 4500), (330, 200, 0), (640, 480, 0)])
def test_against_fp64(cols, rows, gap):
    m = engine_or_skip()
    scene = column(cols, rows, gap=gap)
    got = []
    for prec in (m.FP64, m.MIXED):
        e = m.Engine(*scene, precision=prec)
        for _ in range(2):
            e.step()
        got.append(e.state())
        e.close()
    a, b = got
    assert a["pressure"].max() > 0 or cols < 10
    assert np.array_equal(a["bc"], b["bc"]) and np.array_equal(a["type"], b["type"])
    assert rel_l2(b["pressure"], a["pressure"]) < 1e-6
    assert rel_l2(b["pos"], a["pos"]) < 1e-9
