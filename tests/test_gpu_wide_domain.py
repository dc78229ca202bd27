"""Planar mixed solves in domains of more than 32,767 and 65,536 cells along an axis: two
bodies of water at its ends, in each form of the solve whose blocks keep their cells'
stencils in shared memory.  Against the FP64 solver from the same state, with the
tolerances of the split cycle's test (solves to 1e-10, FP32 sums at 6e-8: pressures
agree to 1e-6, flags are identical).
"""
import numpy as np
import pytest

from gpu_util import engine_or_skip, rel_l2
from mps_gb300 import scenes

pytestmark = pytest.mark.gpu
L0 = 0.01


def bodies(cols, rows, gap, axis):
    """A compressed column in its tank, and a second one `gap` particle distances along axis."""
    prm, pos, vel, t = scenes.hydrostatic(L0, size=(cols * L0, rows * L0), dt=0.1 * L0, margin=12 * L0)
    pos[t == scenes.FLUID, 1] *= 0.998
    other = pos.copy()
    other[:, axis] += gap * L0
    prm["domain_max"][axis] += gap * L0
    return prm, np.concatenate([pos, other]), np.concatenate([vel, vel]), np.concatenate([t, t])


def step_of(m, scene, prec):
    e = m.Engine(*scene, precision=prec)
    e.step()
    out = e.state()
    e.close()
    return out


def agree(a, b):
    assert a["pressure"].max() > 0
    assert np.array_equal(a["bc"], b["bc"]) and np.array_equal(a["type"], b["type"])
    assert rel_l2(b["pressure"], a["pressure"]) < 1e-6


# 33,901 and 67,772 cells in x, 66,160 in y; above 150,000 rows the streaming form
@pytest.mark.parametrize("cols,rows,gap,axis", [(60, 50, 105000, 0), (60, 50, 210000, 0), (60, 50, 205000, 1),
                                                (280, 280, 105000, 0)])
def test_against_fp64(cols, rows, gap, axis):
    m = engine_or_skip()
    scene = bodies(cols, rows, gap, axis)
    agree(step_of(m, scene, m.FP64), step_of(m, scene, m.MIXED))


@pytest.mark.parametrize("block", [256, 1024])
def test_batch(block):
    m = engine_or_skip()
    some = [bodies(40, 30, 105000, 0), bodies(30, 40, 205000, 1), bodies(30, 20, 50, 0)]
    b = m.Batch(some, tol=1e-10)
    b.set_launch(block, 1.0)
    b.step()
    for s, scene in enumerate(some):
        agree(step_of(m, scene, m.FP64), b.scene(s).state())
    b.close()
