"""Chain rods at the sizes where the chain kernel changes shape (one warp up to 32 nodes, then
22 nodes per warp, 256 at most) and at iteration counts around its chunk of 20, against the
float32 oracle: the rods alone (no fluid, no steric field).

Tolerance: the bar of test_gpu_parity.py for positions and angles, rel-L2 <= 1e-5; every
operation but the sine and cosine is rounded as the oracle rounds it."""
import dataclasses

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from microcosmos_b200 import COSSERAT_SCHEME, baseline_config, scenarios  # noqa: E402
from microcosmos_b200.engine import Actuation, DeviceState, Plan  # noqa: E402
from oracle import ref_numpy as O  # noqa: E402

TOL = 1e-5


def config(solver, cycles):
    over = dict(cycles_per_step=cycles, enable_fluid=False, enable_steric=False)
    if solver == "cosserat":
        return dataclasses.replace(COSSERAT_SCHEME, dt=0.01, stiffness_stretch=10000.0, stiffness_shear=10000.0, **over)
    return baseline_config(**over)


def check(sc, cfg, steps):
    st = DeviceState.from_scenario(sc)
    act = Actuation.from_scenario(sc)
    Plan.for_states([st], [cfg], [0.01]).rollout([st], steps, actuations=[act])
    out = st.host()
    ocfg = O.Config(**{f.name: getattr(cfg, f.name) for f in dataclasses.fields(O.Config)})
    a = (sc.act_c, sc.act_amp, sc.act_omega, sc.act_phase) if sc.act_amp is not None else None
    ref, _ = O.simulate(O.state_from_scenario(sc), ocfg, 0.01, steps, act=a)
    for k in ("position", "theta"):
        assert O.rel_l2(out[k], getattr(ref, k)) < TOL, k


@pytest.mark.parametrize("solver", ["pbd", "cosserat"])
@pytest.mark.parametrize("nodes", [2, 3, 31, 32, 33, 44, 45, 66, 67, 255, 256])
def test_rods_of_every_shape(nodes, solver):
    check(scenarios.make_scenario(320, 300, 3, nodes, seed=nodes, amp=0.3, period=20.0), config(solver, 20), 3)


@pytest.mark.parametrize("cycles", [1, 19, 20, 21, 45])
def test_iteration_counts_around_the_chunk(cycles):
    check(scenarios.make_scenario(96, 96, 4, 40, seed=cycles, amp=0.3, period=20.0), config("pbd", cycles), 3)


@pytest.mark.parametrize("nodes", [20, 70])
def test_operands_outside_the_fast_range(nodes):
    """Angles more than two turns apart, and an edge of zero length: the general path."""
    sc = scenarios.make_scenario(96, 96, 2, nodes, seed=1, amp=0.3, period=20.0)
    sc.theta[5] += np.float32(40.0)
    sc.position[9] = sc.position[8]
    check(sc, config("pbd", 20), 2)
