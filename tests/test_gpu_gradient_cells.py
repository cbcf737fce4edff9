"""Gradients where the entries by cell and the rod kernels of the reverse step change shape: runs of
up to 8, up to 16 and more entries per cell (crowded nodes) with 2- to 5-point kernels, rods below
and above the 128 nodes kept one per thread, iteration counts around the lengths of the tables.

Against the float32 gradient oracle over 2 steps.  The bar is test_gpu_adjoint.py's, widened by
what rounding does to the oracle itself: GRAD_TOL + 4 x rel-L2(float32 oracle, float64 oracle)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from microcosmos_b200 import scenarios  # noqa: E402
from oracle import ref_numpy as O  # noqa: E402
from test_gpu_adjoint import GRAD_TOL, case, cotangent, gpu_grads, oracle_grads  # noqa: E402


def check(sc, oc, steps=2):
    cot = cotangent(sc, 1)
    fin, g = gpu_grads(sc, oc, steps, cot)
    s32, g32 = oracle_grads(sc, oc, steps, cot, np.float32)
    _, g64 = oracle_grads(sc, oc, steps, cot, np.float64)
    assert O.rel_l2(fin["position"], s32.position) < 1e-5
    for k in g32:
        bar = GRAD_TOL + 4 * O.rel_l2(g32[k], g64[k])
        assert O.rel_l2(g[k], g32[k]) < bar, (k, O.rel_l2(g[k], g32[k]), bar)


@pytest.mark.parametrize("kernel", [2, 4, 5])
@pytest.mark.parametrize("filaments", [1, 6])
def test_crowded_cells(filaments, kernel):
    sc = case(40, 32, filaments, 12, seed=filaments)
    mid = sc.position.mean(0)
    sc.position = ((sc.position - mid) * np.float32(0.12) + mid).astype(np.float32)
    check(sc, O.Config(ibm_kernel_size=kernel, enable_steric=False))


@pytest.mark.parametrize("nodes", [3, 127, 128, 129])
def test_rod_lengths(nodes):
    check(case(160, 144, 2, nodes, seed=nodes), O.Config(enable_fluid=False, enable_steric=False))


@pytest.mark.parametrize("cycles", [1, 10, 11, 21, 41])
def test_iteration_counts(cycles):
    check(case(32, 32, 2, 10, seed=cycles),
          O.Config(enable_fluid=False, enable_steric=False, cycles_per_step=cycles))


@pytest.mark.parametrize("every", [1, 2, 3, 6])
def test_segments_recomputed_beside_the_reverse(every):
    """The recomputed inputs of neighbouring segments are kept apart: the same bits as one segment."""
    sc, steps = case(40, 32, 3, 12, seed=every), 7
    cot = cotangent(sc, 2)
    want = gpu_grads(sc, O.Config(), steps, cot, ckpt=steps)[1]
    got = gpu_grads(sc, O.Config(), steps, cot, ckpt=every)[1]
    for k in want:
        assert got[k].tobytes() == want[k].tobytes(), k
