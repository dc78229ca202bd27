"""The FP64 solve's exchange between blocks, polled by every block, gives up in every block
with the timeout status when a member's slot is never written, and the context stays
usable.  The failure is made on the host side of the wait (a member count that no launch
completes); nothing faults."""
import pytest

from golden_cases import load
from gpu_util import engine_or_skip

pytestmark = pytest.mark.gpu


def test_exchange_gives_up_and_context_survives():
    m = engine_or_skip()
    from mps_gb300.engine import selftest_wait_limit

    rc, gave_up, seconds = selftest_wait_limit(exchange=True)
    assert rc == 0 and gave_up == 8, (rc, gave_up)
    assert seconds < 10.0
    g = load("dambreak_l0_01")
    e = m.Engine(g["params"], g["pos0"], g["vel0"], g["type0"], precision=m.FP64)
    assert e.step()["status"] == 0
    e.close()
