"""Touched cells listed from the lattice's counters (plans whose populations exceed the L2, rollouts with
contributions for a third of their cells or more) against the list made by the stencil kernel: rollouts
beside a large lattice, which takes the plan over the line, and the same ones alone.  Every sum runs
in the order of the contributions, so the bits are the same.  Lattices whose cells are and are not
multiples of a thread's 8 and a CTA's 2,048; both stencil kernels; a rollout below the third."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from microcosmos_b200 import baseline_config, scenarios  # noqa: E402
from microcosmos_b200.engine import Actuation, DeviceState, Plan  # noqa: E402


def rollouts(scs, cfg, steps=3):
    states = [DeviceState.from_scenario(sc) for sc in scs]
    acts = [Actuation.from_scenario(sc) for sc in scs]
    plan = Plan.for_states(states, [cfg] * len(scs), [0.01] * len(scs))
    plan.rollout(states, steps, actuations=acts)
    plan.profile(True)
    plan.profile_reset()
    plan.rollout(states, 1, actuations=acts, use_graph=False)
    return states, plan.profile_read()["ib_list"][1]


@pytest.mark.parametrize("kernel", [1, 3, 4, 5])
def test_same_bits_as_the_stencil_kernels_list(kernel):
    sizes = [(64, 64, 20, 30), (33, 51, 10, 60), (45, 45, 30, 20), (128, 96, 40, 100), (67, 31, 9, 77), (200, 160, 4, 25)]
    scs = [scenarios.make_scenario(H, W, F, n, seed=i, amp=0.3, period=20.0) for i, (H, W, F, n) in enumerate(sizes)]
    large = scenarios.make_scenario(1344, 1344, 30, 40, seed=9, amp=0.3, period=20.0)  # 1.8 M cells
    cfg = baseline_config(ibm_kernel_size=kernel)
    alone, listed = rollouts(scs, cfg)
    assert listed == 0
    beside, listed = rollouts(scs + [large], cfg)
    assert listed == 1
    for a, b in zip(alone, beside):
        for k in ("position", "velocity", "theta", "f_grid", "fluid_velocity", "steric"):
            assert torch.equal(getattr(a, k).view(torch.int32), getattr(b, k).view(torch.int32)), k
