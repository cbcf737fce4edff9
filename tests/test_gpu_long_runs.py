"""Touched cells with many contributions: sorted by a warp in chunks of 32 and merges (lengths around
the chunk and its doublings), several of them shared among a CTA's warps.

Against the float32 oracle with the bars of test_gpu_touched_cells.py; and the cost: a step whose
points all lie in one spot (a collapsed rollout, or one whose positions are no longer numbers) takes
time about in proportion to their number."""
import dataclasses

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from microcosmos_b200 import baseline_config, scenarios  # noqa: E402
from microcosmos_b200.engine import DeviceState, Plan  # noqa: E402
from oracle import ref_numpy as O  # noqa: E402


def loose_nodes(pos, seed, H=96, W=112):
    """Nodes without rods."""
    rng = np.random.default_rng(seed)
    sc = scenarios.make_scenario(H, W, 1, 3, seed=seed, actuate=False)
    none, empty = np.zeros((0, 2), np.int32), np.zeros(0, np.float32)
    return dataclasses.replace(sc, position=pos.astype(np.float32), velocity=rng.normal(0, 0.5, pos.shape).astype(np.float32),
                               pairs=none, theta=empty, rest_lengths=empty, bending_pairs=none,
                               bending_rest_angles=empty, bending_stiffness=empty)


def bins_ms(sc, cfg, steps=2):
    """Time per step of ordering the contributions by cell, and the plan's final state."""
    st = DeviceState.from_scenario(sc)
    plan = Plan.for_states([st], [cfg], [0.01])
    plan.profile(True)
    plan.rollout([st], steps, use_graph=False)
    ms, launches = plan.profile_read()["ib_bins"]
    assert launches == steps
    return ms / steps, st.host()


@pytest.mark.parametrize("spots", [1, 9])
@pytest.mark.parametrize("clump", [31, 32, 33, 64, 65, 128, 129, 1000])
def test_lengths_around_the_chunks(clump, spots):
    """`clump` nodes on each of some spots, among 600 scattered ones."""
    clump = clump if spots == 1 else min(clump, 129)
    rng = np.random.default_rng(clump)
    pos = rng.uniform(0, 1, (600, 2)) * (112, 96)
    at = [np.array([20.3 + 9 * (s % 3), 17.6 + 8 * (s // 3)]) + rng.uniform(0, 0.3, (clump, 2)) for s in range(spots)]
    pos = rng.permutation(np.concatenate([pos] + at))
    cfg = baseline_config(enable_steric=False)
    _, out = bins_ms(loose_nodes(pos, clump), cfg)
    ocfg = O.Config(**{f.name: getattr(cfg, f.name) for f in dataclasses.fields(O.Config)})
    ref, _ = O.simulate(O.state_from_scenario(loose_nodes(pos, clump)), ocfg, 0.01, 2)
    for k, tol in (("position", 1e-5), ("f_grid", 1e-5), ("velocity", 1e-3), ("fluid_velocity", 1e-4)):
        assert O.rel_l2(out[k], getattr(ref, k)) < tol, (k, O.rel_l2(out[k], getattr(ref, k)))


def test_cost_grows_with_the_number_of_points():
    """8 times the points in one spot: 8 x log ratio (13/10) is 10.4 times the time for a sort, 64 for
    comparing every pair; the line between them is 20."""
    ms = []
    for n in (1024, 8192):
        pos = np.array([40.3, 17.6]) + np.random.default_rng(n).uniform(0, 0.1, (n, 2))
        bins_ms(loose_nodes(pos, 1), baseline_config(enable_steric=False))
        ms.append(bins_ms(loose_nodes(pos, 1), baseline_config(enable_steric=False))[0])
    assert ms[1] < 20 * ms[0], ms
