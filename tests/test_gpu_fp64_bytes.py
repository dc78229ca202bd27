"""solve_bytes of the FP64 solver counts what its kernel streams: per iteration 10 bytes per
stored off-diagonal entry (FP64 value, 16-bit index) and 80 per row, once 10 and 56."""
import pytest

from gpu_util import engine_or_skip
from mps_gb300 import scenes

pytestmark = pytest.mark.gpu


def test_fp64_bytes():
    m = engine_or_skip()
    prm, pos, vel, t = scenes.hydrostatic(0.01, size=(0.6, 0.5), margin=0.1)
    pos[t == scenes.FLUID, 1] *= 0.998
    e = m.Engine(prm, pos, vel, t)
    st = e.step()
    e.close()
    nnz, n, it = st["nnz_offdiag"], len(t), st["cg_iterations"]
    assert it > 0 and nnz > 0
    assert st["solve_bytes"] == it * (10 * nnz + 80 * n) + 10 * nnz + 56 * n
