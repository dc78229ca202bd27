"""More collision pairs than the engine's table of 4 per particle holds: the step reports
MPS_ERR_CAPACITY, applies none and reads no pair that was never written, in both orders
of application; a scene that fits runs afterwards."""
import numpy as np
import pytest

from gpu_util import engine_or_skip
from test_gpu_sweep_split import L0, box

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("serial", [False, True])
@pytest.mark.parametrize("side,cd", [(12, 1.6), (12, 2.3), (30, 2.3)])
def test_overflow_is_reported(side, cd, serial):
    m = engine_or_skip()
    from mps_gb300 import engine

    prm, pos, vel, t = box(side)
    prm["collision_distance"] = cd * L0  # 8 to 21 pairs per particle
    e = m.Engine(prm, pos, vel, t, precision=m.FP64)
    e.set_collisions(serial)
    for _ in range(2):
        with pytest.raises(engine.MpsError) as ex:
            e.step()
        assert ex.value.code == engine.MPS_ERR_CAPACITY
    s = e.state()
    assert np.isfinite(s["pos"]).all()
    e.close()
    # no collisions: as with a distance that no pair is within
    e = m.Engine(dict(prm, collision_distance=0.1 * L0), pos, vel, t, precision=m.FP64)
    for _ in range(2):
        e.step()
    assert len(e.collisions()[0]) == 0
    assert np.array_equal(e.state()["pos"], s["pos"])
    e.close()
