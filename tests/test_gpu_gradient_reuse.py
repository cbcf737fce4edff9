"""A gradient plan that is kept: short rollouts launch the kernels of their first gradient directly
and those of later ones by graphs.  Every gradient is the same bits; and graphs are launched from the
second on, at the step counts on both sides of where the first would already use them."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from microcosmos_b200 import baseline_config, scenarios  # noqa: E402
from microcosmos_b200.autodiff import GradPlan  # noqa: E402
from microcosmos_b200.engine import Actuation, DeviceState  # noqa: E402


def graph_launches(call):
    """Graph launches that the profiler saw in a call (None where it sees no launches at all), its result."""
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as prof:
        result = call()
        torch.cuda.synchronize()
    launches = [e for e in prof.key_averages() if "Launch" in e.key]
    return sum(e.count for e in launches if "GraphLaunch" in e.key) if launches else None, result


# 2 x 16 nodes: with the node-step kernel, 20 x 40: without
@pytest.mark.parametrize("steps,filaments,nodes", [(1, 2, 16), (16, 20, 40), (17, 2, 16), (64, 20, 40), (65, 2, 16)])
def test_gradients_of_a_kept_plan(steps, filaments, nodes):
    sc = scenarios.make_scenario(96, 80, filaments, nodes, seed=steps, amp=0.3, period=20.0)
    act = Actuation.from_scenario(sc)
    plan = GradPlan(sc.H, sc.W, sc.N, sc.pairs, sc.bending_pairs, baseline_config(), 0.01, steps)
    seed = torch.zeros((sc.N, 2), device="cuda")
    seed[:, 0] = 1.0 / sc.N
    first = None
    for k in range(3):
        st = DeviceState.from_scenario(sc)
        fwd, _ = graph_launches(lambda: plan.forward(st, act))
        bwd, grads = graph_launches(lambda: plan.backward(seed))
        got = {"x": st.position, "f": st.f_grid, **grads}
        first = first or got
        for name in first:
            assert torch.equal(got[name].view(torch.int32), first[name].view(torch.int32)), (k, name)
        if fwd is not None and bwd is not None:
            assert (fwd > 0) == (k > 0 or steps > 64), (k, fwd)
            assert (bwd > 0) == (k > 0 or steps > 16), (k, bwd)
    plan.close()
