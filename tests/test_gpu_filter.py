"""The steric filter at the side lengths and values per thread where its kernels change shape: the
smallest transforms of each radix, every remainder of the last pass, sides of 3 * 2^a, sides of two
families in one plan and in one rollout, odd counts of rows and columns.  Against the float64
oracle's filter of the same deposit; the bar is the repository's for the steric field, rel-L2 1e-5
(float32 transforms are near 2e-7)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from microcosmos_b200 import baseline_config, scenarios  # noqa: E402
from microcosmos_b200.engine import DeviceState, Plan  # noqa: E402
from oracle import ref_numpy as O  # noqa: E402


def check(sizes, fft_values):
    scs = [scenarios.make_scenario(h, w, 2, 9, seed=h + w, actuate=False) for h, w in sizes]
    sts = [DeviceState.from_scenario(s) for s in scs]
    cfg = baseline_config(enable_fluid=False)
    Plan.for_states(sts, [cfg] * len(scs), [0.01] * len(scs), fft_values=fft_values).rollout(sts, 1)
    for sc, st in zip(scs, sts):
        pred = sc.position + sc.velocity * np.float32(0.01)
        dep = O.steric_deposit(sc.H, sc.W, pred, 1.0).astype(np.float64)
        want = O.gaussian_filter(dep, cfg.steric_sigma)
        assert O.rel_l2(st.host()["steric"], want) < 1e-5, (sc.H, sc.W)


@pytest.mark.parametrize("fft_values", [4, 8, 16])
@pytest.mark.parametrize("side", [16, 32, 64, 128, 256, 512, 1024, 2048, 4096])
def test_powers_of_two(side, fft_values):
    check([(side, 64), (64, side)], fft_values)


@pytest.mark.parametrize("side", [12, 24, 48, 96, 192, 384, 768, 1536])
def test_three_times_powers_of_two(side):
    check([(side, side), (side, 48)], 0)


def test_families_beside_each_other_and_mixed():
    check([(128, 64), (96, 48), (90, 60), (67, 71)], 0)
    check([(128, 96), (96, 64), (90, 64), (64, 50)], 0)
    check([(65, 128), (128, 63), (33, 96)], 16)
