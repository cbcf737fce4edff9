"""Plans of more chain rods than are run by four warps each at once (6 x 148): every rod then takes the
warps that its nodes need.  A plan of copies of a few rollouts against those rollouts in small plans:
the same bits; and the cost: a launch of 4,000 short rods against one of 400, which all fit at once."""
import dataclasses

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from microcosmos_b200 import COSSERAT_SCHEME, baseline_config, scenarios  # noqa: E402
from microcosmos_b200.engine import Actuation, DeviceState, Plan  # noqa: E402

COSSERAT = dataclasses.replace(COSSERAT_SCHEME, dt=0.01, stiffness_stretch=10000.0, stiffness_shear=10000.0)
OFF = dict(enable_fluid=False, enable_steric=False)


def rollout(scs, cfg, copies, steps=3):
    """`copies` of the rollouts in one plan of separate kernels (an IB layout asked for keeps it there)."""
    states = [DeviceState.from_scenario(sc) for sc in scs * copies]
    acts = [Actuation.from_scenario(sc) for sc in scs * copies]
    plan = Plan.for_states(states, [cfg] * len(states), [0.01] * len(states), ib_cluster=1)
    plan.rollout(states, steps, actuations=acts)
    return plan, states, acts


@pytest.mark.parametrize("solver", ["pbd", "cosserat"])
@pytest.mark.parametrize("nodes", [12, 32, 33, 64, 100])
def test_many_rods_are_the_same_bits(nodes, solver):
    cfg = dataclasses.replace(baseline_config() if solver == "pbd" else COSSERAT, **OFF)
    scs = [scenarios.make_scenario(160, 144, 45, nodes, seed=s, amp=0.3, period=20.0) for s in (1, 2)]
    _, few, _ = rollout(scs, cfg, 1)
    _, many, _ = rollout(scs, cfg, 12)  # 1,080 rods
    for i, st in enumerate(many):
        for k in ("position", "velocity", "theta"):
            assert torch.equal(getattr(st, k).view(torch.int32), getattr(few[i % 2], k).view(torch.int32)), (i, k)


def test_cost_of_many_short_rods():
    """400 rods run at once; 4,000 of one warp each fill the SMs' 64 warp places once (9,472), and take
    at most three times as long (2.1 measured; 4.4 while only 4 CTAs fitted on an SM)."""
    us = []
    for copies in (1, 10):
        sc = scenarios.make_scenario(256, 256, 400, 32, seed=3, amp=0.3, period=20.0)
        plan, states, acts = rollout([sc], baseline_config(**OFF), copies)
        plan.profile(True)
        plan.profile_reset()
        plan.rollout(states, 8, actuations=acts, use_graph=False)
        ms, launches = plan.profile_read()["chain"]
        us.append(ms / launches * 1e3)
    assert us[1] < 3 * us[0], us
