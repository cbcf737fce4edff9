"""The node-step kernel (one launch for the node side of a step, taken by plans of small
rollouts) against the separate kernels, over the forms it accepts: kernel sizes, both rod
solvers, synthetic pairs, force clamp, no steric field, no fluid, a lattice other than the
domain, odd and non-square grids, uneven batches, recording, sizes around its limits.  Asking for
another layout of the IB kernels (one CTA per rollout cluster) keeps a plan on the separate
kernels.  Both sum in the same order, so every output is the same bits."""
import dataclasses

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from microcosmos_b200 import COSSERAT_SCHEME, baseline_config, scenarios  # noqa: E402
from microcosmos_b200.engine import Actuation, DeviceState, Plan, Record  # noqa: E402

COSSERAT = dataclasses.replace(COSSERAT_SCHEME, dt=0.01, stiffness_stretch=10000.0, stiffness_shear=10000.0,
                               viscosity=0.1, ibm_kernel_size=3, enable_steric=True)


def rollout(scs, cfgs, steps, separate, record=False, calls=1, use_graph=True):
    sts = [DeviceState.from_scenario(s) for s in scs]
    plan = Plan.for_states(sts, cfgs, [0.01] * len(scs), ib_cluster=1 if separate else 0)
    recs = [Record.allocate(s, steps, every=2) for s in sts] if record else None
    for k in range(calls):
        acts = [Actuation.from_scenario(s, t0=k * steps) for s in scs]
        plan.rollout(sts, steps, actuations=acts, records=recs, use_graph=use_graph)
    plan.profile(True)  # kernel names of one more step
    plan.profile_reset()
    plan.rollout(sts, 1, actuations=[Actuation.from_scenario(s) for s in scs], use_graph=False)
    fused = plan.profile_read()["node_step"][1] > 0
    out = [s.host() for s in sts]
    if record:
        out += [{k: getattr(r, k).cpu().numpy() for k in ("position", "velocity", "steric", "fluid_velocity")}
                for r in recs]
    return out, fused, plan.read_flags()


def assert_same(scs, cfgs, steps=4, fused=True, **kw):
    a, fa, flags_a = rollout(scs, cfgs, steps, False, **kw)
    b, fb, flags_b = rollout(scs, cfgs, steps, True, **kw)
    assert fa == fused and not fb
    assert flags_a == flags_b
    for x, y in zip(a, b):
        for k in x:
            np.testing.assert_array_equal(x[k], y[k], err_msg=k)


@pytest.mark.parametrize("over", [
    dict(), dict(ibm_kernel_size=1), dict(ibm_kernel_size=2), dict(ibm_kernel_size=3),
    dict(enable_steric=False), dict(enable_fluid=False), dict(enable_fluid=False, enable_steric=False),
    dict(synthetic_node_width=0.7), dict(enable_force_clamp=True, max_fluid_velocity=0.01),
    dict(steric_neighbor_skip=0), dict(steric_neighbor_skip=9), dict(ibm_iterations=0), dict(ibm_iterations=1),
    dict(node_mass=0.5, damping=0.9)])
def test_configurations(over):
    assert_same([scenarios.make_scenario(60, 77, 5, 23, seed=3, amp=0.3, period=20.0)], [baseline_config(**over)])


def test_cosserat_and_mixed_batch():
    scs = [scenarios.make_scenario(64, 48, 3, 40, seed=1), scenarios.make_scenario(33, 50, 1, 7, seed=2),
           scenarios.make_scenario(96, 96, 6, 16, seed=3)]
    assert_same(scs, [COSSERAT, baseline_config(ibm_kernel_size=2), baseline_config(enable_steric=False)])


@pytest.mark.parametrize("use_graph", [True, False])
def test_recording_and_continued_calls(use_graph):
    scs = [scenarios.make_scenario(40, 56, 3, 20, seed=5, amp=0.3, period=20.0)]
    assert_same(scs, [baseline_config()], steps=5, record=True, use_graph=use_graph)
    assert_same(scs, [baseline_config()], steps=3, calls=3, use_graph=use_graph)


def test_lattice_other_than_the_domain():
    sc = scenarios.make_scenario(48, 40, 3, 20, seed=6)
    lattice = scenarios.make_scenario(72, 30, 1, 4, seed=7)
    sc = dataclasses.replace(sc, f_grid=lattice.f_grid, fluid_velocity=lattice.fluid_velocity)
    assert_same([sc], [baseline_config()])


@pytest.mark.parametrize("filaments,nodes,fused", [(1, 1, True), (1, 2, True), (1, 256, True), (16, 25, True), (16, 26, False),
                                                   (12, 32, True), (15, 45, False), (40, 60, False)])
def test_sizes_around_the_limit(filaments, nodes, fused):
    sc = scenarios.make_scenario(128, 128, filaments, nodes, seed=nodes) if nodes > 1 else single_node()
    assert_same([sc], [baseline_config()], fused=fused)


def single_node():
    sc = scenarios.make_scenario(32, 32, 1, 2, seed=4)
    return dataclasses.replace(sc, position=sc.position[:1], velocity=sc.velocity[:1], pairs=sc.pairs[:0],
                               theta=sc.theta[:0], rest_lengths=sc.rest_lengths[:0])


def test_many_points_in_one_cell():
    """All rods on one spot: runs of hundreds of contributions."""
    sc = scenarios.make_scenario(64, 64, 12, 30, seed=8)
    sc.position[:] = np.float32(20.25) + np.float32(1e-3) * np.arange(sc.N, dtype=np.float32)[:, None] % np.float32(0.5)
    assert_same([sc], [baseline_config()], steps=2)
