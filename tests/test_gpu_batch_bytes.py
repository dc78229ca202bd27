"""solve_bytes of a batch counts the arrangement that its blocks ran: 1,024-thread blocks
the overlapped one (as a single engine's mode 1), smaller ones the plain one (mode 4).
The model is linear in the iterations; its other terms are taken off as the engine adds
them (17 B per entry and 64 B per row of setup; 12 B per entry and 36 B per row and
FP64 residual), so the rest per iteration is the same number for the same scene."""
import pytest

from gpu_util import engine_or_skip
from mps_gb300 import scenes

pytestmark = pytest.mark.gpu


def per_iteration(st, n):
    nnz = st["nnz_offdiag"]
    rest = 17 * nnz + 64 * n + (st["refinements"] + 1) * (12 * nnz + 36 * n)
    assert st["cg_iterations"] > 0
    return (st["solve_bytes"] - rest) / st["cg_iterations"]


@pytest.mark.parametrize("block,mode", [(256, 4), (512, 4), (1024, 1)])
def test_batch_counts_its_own_arrangement(block, mode):
    m = engine_or_skip()
    some = []
    for cols, rows in ((40, 30), (25, 50)):
        prm, pos, vel, t = scenes.hydrostatic(0.01, size=(cols * 0.01, rows * 0.01), margin=0.1)
        pos[t == scenes.FLUID, 1] *= 0.998
        some.append((prm, pos, vel, t))
    b = m.Batch(some)
    b.set_launch(block, 1.0)
    stats, _ = b.step()
    for st, scene in zip(stats, some):
        e = m.Engine(*scene, precision=m.MIXED, tol=1e-8)
        e.set_multigrid(mode)
        want = per_iteration(e.step(), len(scene[3]))
        e.close()
        assert per_iteration(st, len(scene[3])) == pytest.approx(want, rel=1e-12)
    b.close()
