"""The default weights of the additive multigrid modes are omega 1.0 and scale 1.4 on every
level: a step with the defaults gives the bits of one with those weights set.  (Another
scale between the cell levels takes fewer iterations, but another path to the solution:
single velocities then move by up to 7e-8 through the FP32 gradient.)"""
import numpy as np
import pytest

from gpu_util import engine_or_skip
from mps_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [1, 3, 4])
@pytest.mark.parametrize("cols,rows", [(40, 30), (150, 145)])
def test_defaults(mode, cols, rows):
    m = engine_or_skip()
    prm, pos, vel, t = scenes.hydrostatic(0.01, size=(cols * 0.01, rows * 0.01), margin=0.1)
    pos[t == scenes.FLUID, 1] *= 0.998
    got = []
    for weights in ((), (1.0, 1.4)):
        e = m.Engine(prm, pos, vel, t, precision=m.MIXED)
        e.set_multigrid(mode, *weights)
        for _ in range(2):
            st = e.step()
        got.append((e.state(), st["cg_iterations"]))
        e.close()
    (a, ia), (b, ib) = got
    assert a["pressure"].max() > 0 and ia == ib
    for key in ("pressure", "pos", "vel"):
        assert np.array_equal(a[key], b[key]), key
