"""Steps whose kernels are launched chained (each waits for the one before inside the kernel) against
the same steps with the kernels timed one at a time (no chained launch, no second stream): the same
bits in every state array.  Over what the chain is made of: kernel sizes 2 to 5 points, plans with
and without fluid and steric field, rods of one and several warps, trees, no iterations, rollouts
of different forcing rounds in one plan, filters of both families, one and many advances, and a
node grid beyond the size up to which launches are chained."""
import dataclasses

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from microcosmos_b200 import baseline_config, scenarios  # noqa: E402
from microcosmos_b200.engine import Actuation, DeviceState, Plan  # noqa: E402


def run(scs, cfgs, steps, profile):
    states = [DeviceState.from_scenario(sc) for sc in scs]
    plan = Plan.for_states(states, cfgs, [0.01] * len(scs))
    plan.profile(profile)
    plan.rollout(states, steps, actuations=[Actuation.from_scenario(sc) for sc in scs])
    return [st.host() for st in states]


def check(scs, cfgs, steps=5):
    for got, want in zip(run(scs, cfgs, steps, False), run(scs, cfgs, steps, True)):
        for k in want:
            if isinstance(want[k], np.ndarray):
                assert got[k].tobytes() == want[k].tobytes(), k


def scenario(H, W, filaments, nodes, seed):
    return scenarios.make_scenario(H, W, filaments, nodes, seed=seed, amp=0.3, period=20.0)


# 20 x 24 points and more: beyond the node-step kernel
@pytest.mark.parametrize("kernel", [2, 3, 4, 5])
@pytest.mark.parametrize("sides", [(128, 128), (96, 128), (90, 70)])
def test_one_rollout(sides, kernel):
    check([scenario(*sides, 20, 24, kernel)], [baseline_config(ibm_kernel_size=kernel)])


@pytest.mark.parametrize("off", ["enable_fluid", "enable_steric"])
def test_without(off):
    check([scenario(128, 128, 24, 40, 3)], [baseline_config(**{off: False})])


@pytest.mark.parametrize("cycles", [0, 1, 21])
def test_iteration_counts(cycles):
    check([scenario(128, 160, 20, 33, 5)], [baseline_config(cycles_per_step=cycles)])


@pytest.mark.parametrize("steps", [1, 2, 3, 8])
def test_uneven_batch(steps):
    scs = [scenario(64, 64, 9, 60, 1), scenario(96, 128, 3, 100, 2), scenario(128, 128, 1, 7, 3)]
    base = baseline_config()
    check(scs, [base, dataclasses.replace(base, ibm_iterations=2), base], steps)


def test_beyond_the_chained_grid():
    scs = [scenario(128, 128, 40, 64, s) for s in range(64)]
    check(scs, [baseline_config()] * 64, 3)
