"""A plan whose rollout was left before its last step (an exception between two advances, an
environment reset): the next rollout on it is the same bits as on a fresh plan, in the node-step
kernel and in separate ones, and the flags of the one left stay."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from microcosmos_b200 import baseline_config, scenarios  # noqa: E402
from microcosmos_b200.engine import Actuation, DeviceState, Plan  # noqa: E402


@pytest.mark.parametrize("over", [dict(), dict(enable_fluid=False), dict(enable_steric=False)])
@pytest.mark.parametrize("cluster", [0, 1])
def test_begin_after_a_rollout_that_was_left(cluster, over):
    sc = scenarios.make_scenario(128, 128, 2, 16, seed=5, amp=0.3, period=20.0)
    plan = Plan.for_states([DeviceState.from_scenario(sc)], [baseline_config(**over)], [0.01], ib_cluster=cluster)

    def begin(state):
        plan.begin([state], [Actuation.from_scenario(sc)])
        return state

    def whole():
        st = begin(DeviceState.from_scenario(sc))
        plan.advance(5, last=True)
        plan.end()
        return st

    want = whole()
    left = DeviceState.from_scenario(sc)
    left.velocity[3] = float("nan")
    begin(left)
    plan.advance(3)
    flags = plan.read_flags()
    for _ in range(2):
        got = whole()
        assert plan.read_flags() == flags and flags[0] & 1
        for k in ("position", "velocity", "theta", "f_grid", "steric"):
            assert torch.equal(getattr(got, k).view(torch.int32), getattr(want, k).view(torch.int32)), k
