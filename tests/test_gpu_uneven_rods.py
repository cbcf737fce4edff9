"""Rods of several lengths in one rollout, more of them than the node-step kernel has teams of warps
for: a team then runs rods of different numbers of warps one after another, and the exchange
buffers and named barriers of one must be free before the next begins.  Against the separate
kernels, which run one rod per CTA: the same bits; and the float32 oracle, with the bar of
test_gpu_chain.py (rel-L2 1e-5 of positions and angles)."""
import dataclasses

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from microcosmos_b200 import COSSERAT_SCHEME, baseline_config, scenarios  # noqa: E402
from oracle import ref_numpy as O  # noqa: E402
from test_gpu_node_step import assert_same, rollout  # noqa: E402


def world(sizes, seed, H=200, W=220):
    """Chains of the given numbers of nodes, each a gently turning walk of unit steps."""
    rng = np.random.default_rng(seed)
    pairs, bpairs = scenarios.line_topology(sizes)
    pos, theta = [], []
    for n in sizes:
        a = rng.uniform(0, 2 * np.pi) + np.cumsum(rng.normal(0, 0.1, n - 1))
        step = np.stack([np.cos(a), np.sin(a)], 1)
        pos.append(rng.uniform(0, 1, 2) * (W, H) + np.concatenate([np.zeros((1, 2)), np.cumsum(step, 0)]))
        theta.append(np.arctan2(step[:, 1], step[:, 0]))
    base = scenarios.make_scenario(H, W, 1, 3, seed=seed)
    B = len(bpairs)
    f32 = np.float32
    return dataclasses.replace(
        base, position=np.mod(np.concatenate(pos), (W, H)).astype(f32), velocity=rng.normal(0, 0.2, (sum(sizes), 2)).astype(f32),
        pairs=pairs, theta=np.concatenate(theta).astype(f32), rest_lengths=np.ones(len(pairs), f32), bending_pairs=bpairs,
        bending_rest_angles=np.zeros(B, f32), bending_stiffness=np.full(B, 0.1, f32), act_c=np.zeros(B, f32),
        act_amp=np.full(B, 0.2, f32), act_omega=np.full(B, 0.3, f32), act_phase=rng.uniform(0, 6, B).astype(f32))


def config(solver, kernel):
    if solver == "pbd":
        return baseline_config(ibm_kernel_size=kernel)
    return dataclasses.replace(COSSERAT_SCHEME, dt=0.01, stiffness_stretch=10000.0, stiffness_shear=10000.0, viscosity=0.1,
                               ibm_kernel_size=kernel, enable_steric=True)


# rods of 2 and 3 warps in teams of 4; of 2 to 5 warps in a team of 10; equal lengths, several per team
SIZES = [[70] + [40] * 6 + [60] * 3, [40, 200, 60], [200, 100, 40, 60, 80], [66] * 7, [30, 90, 50, 20, 70, 40, 33, 2, 88]]


@pytest.mark.parametrize("solver", ["cosserat", "pbd"])
@pytest.mark.parametrize("sizes", SIZES, ids=["70-40-60", "40-200-60", "200-to-40", "66x7", "2-to-90"])
def test_uneven_rods(sizes, solver):
    sc, cfg = world(sizes, len(sizes)), config(solver, 3)
    assert_same([sc], [cfg], steps=3)
    out, fused, _ = rollout([sc], [dataclasses.replace(cfg, enable_fluid=False, enable_steric=False)], 2, False)
    assert fused
    ocfg = O.Config(**{f.name: getattr(cfg, f.name) for f in dataclasses.fields(O.Config)})
    ocfg = dataclasses.replace(ocfg, enable_fluid=False, enable_steric=False)
    acts = (sc.act_c, sc.act_amp, sc.act_omega, sc.act_phase)
    ref, _ = O.simulate(O.state_from_scenario(sc), ocfg, 0.01, 2, act=acts)
    ref, _ = O.simulate(ref, ocfg, 0.01, 1, act=acts)  # the one more step of rollout()
    for k in ("position", "theta"):
        assert O.rel_l2(out[0][k], getattr(ref, k)) < 1e-5, k


@pytest.mark.parametrize("solver", ["cosserat", "pbd"])
def test_operands_outside_the_fast_range(solver):
    """Two coinciding nodes in every rod: each rod is done again on the general path."""
    sizes = SIZES[0]
    sc = world(sizes, 3)
    first = np.cumsum([0] + sizes[:-1])
    sc.position[first + 9] = sc.position[first + 8]
    sc.theta[5] += np.float32(40.0)
    assert_same([sc], [config(solver, 3)], steps=2)
