"""The symmetry fingerprint of a step sees an asymmetric matrix: a block of fluid so dense
that the neighbour lists overflow, each particle's list without the last of its
neighbours, makes a matrix whose entries lack their transposes.  The step reports the
overflow (MPS_ERR_CAPACITY comes first), and its skipped solve (relative residual -1,
no iterations) shows that the fingerprint was not zero: in the assembly for the FP64
solver, in the operator's setup for the mixed one.
"""
import ctypes as C

import numpy as np
import pytest

from gpu_util import engine_or_skip
from mps_gb300 import scenes

pytestmark = pytest.mark.gpu
L0 = 0.01


def block(scale, side=24):
    g = np.stack(np.meshgrid(np.arange(side), np.arange(side), indexing="ij"), -1).reshape(-1, 2)
    pos = np.zeros((len(g), 3))
    pos[:, :2] = (g + 0.5) * L0
    m = 8 * L0
    prm = scenes.baseline_physics(L0, 0.1 * L0, (-m, -m, 0.0), (side * L0 + m, side * L0 + m, 0.0))
    prm["collision_distance"] = 0.1 * L0
    t = np.full(len(g), scenes.FLUID, np.int32)
    return (prm, pos, np.zeros_like(pos), t), pos * [scale, scale, 0.0]


@pytest.mark.parametrize("precision", ["FP64", "MIXED"])
@pytest.mark.parametrize("scale,overflows", [(0.9, False), (0.6, True)])
def test_step_fingerprint(precision, scale, overflows):
    m = engine_or_skip()
    from mps_gb300 import engine

    scene, dense = block(scale)
    e = m.Engine(*scene, precision=getattr(m, precision))
    e.upload(pos=dense)
    st = engine.MpsStepStats()
    rc = engine.load().mps_step(e._h, 0, C.byref(st))
    assert rc == (engine.MPS_ERR_CAPACITY if overflows else engine.MPS_OK)
    assert st.max_neighbors > 64 if overflows else st.max_neighbors <= 64
    assert (st.cg_relative_residual == -1.0 and st.cg_iterations == 0) == overflows
    if not overflows:
        assert st.cg_iterations > 0
    e.close()
