"""The touched cells' runs at the lengths where they are kept differently: up to 8 and up to 16
contributions sorted in registers, more through the pool, more than a bucket through the overflow
list; with 2- to 5-point kernels, against the float32 oracle.

Tolerance: the bars of test_gpu_parity.py (rel-L2 1e-5; u* 1e-4; velocities, difference quotients
of positions, 1e-3): sums are taken in the oracle's order."""
import dataclasses

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from microcosmos_b200 import baseline_config, scenarios  # noqa: E402
from microcosmos_b200.engine import DeviceState, Plan  # noqa: E402
from oracle import ref_numpy as O  # noqa: E402


@pytest.mark.parametrize("kernel", [2, 3, 4, 5])
@pytest.mark.parametrize("clump", [3, 8, 9, 16, 17, 33, 200])
def test_runs_of_every_length(clump, kernel):
    """500 separate nodes; `clump` of them share one spot, so that its cells' runs are about that
    long, and a rod's worth lie around it."""
    sc = scenarios.make_scenario(96, 112, 1, 500, seed=clump, spacing=0.0, actuate=False)
    rng = np.random.default_rng(clump)
    pos = rng.uniform(0, 1, (500, 2)) * np.array([112, 96])
    pos[50:50 + clump] = np.array([40.3, 17.6]) + rng.uniform(0, 0.3, (clump, 2))
    pos[300:330] = np.array([41.0, 18.0]) + rng.uniform(-3, 3, (30, 2))
    none = np.zeros((0, 2), np.int32)
    sc = dataclasses.replace(sc, position=pos.astype(np.float32), velocity=(rng.normal(0, 0.5, (500, 2))).astype(np.float32),
                             pairs=none, theta=np.zeros(0, np.float32), rest_lengths=np.zeros(0, np.float32),
                             bending_pairs=none, bending_rest_angles=np.zeros(0, np.float32),
                             bending_stiffness=np.zeros(0, np.float32))
    cfg = baseline_config(ibm_kernel_size=kernel, enable_steric=False)
    st = DeviceState.from_scenario(sc)
    plan = Plan.for_states([st], [cfg], [0.01], ib_cluster=0)
    plan.profile(True)
    plan.rollout([st], 2, use_graph=False)
    if kernel >= 4:
        assert plan.profile_read()["ib_bins"][1] == 2
    out = st.host()
    ocfg = O.Config(**{f.name: getattr(cfg, f.name) for f in dataclasses.fields(O.Config)})
    ref, _ = O.simulate(O.state_from_scenario(sc), ocfg, 0.01, 2)
    for k, tol in (("position", 1e-5), ("f_grid", 1e-5), ("velocity", 1e-3), ("fluid_velocity", 1e-4)):
        assert O.rel_l2(out[k], getattr(ref, k)) < tol, (k, O.rel_l2(out[k], getattr(ref, k)))
