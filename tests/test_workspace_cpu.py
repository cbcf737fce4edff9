"""What a plan's workspace is made of, in bytes per lattice cell (host only): the populations twice
(72), the deposit and the filter's row pass (8), the cloud-in-cell bins (8), and for the IB
contributions of a cell a counter, a list head (8) and a bucket: of 16 entries, or of 8 in plans of
the node-step kernel, which fill none."""
import ctypes

import pytest

from microcosmos_b200 import PBD_SCHEME, _lib, baseline_config, scenarios
from test_abi_cpu import _create, lib  # noqa: F401


@pytest.mark.parametrize("nodes,filaments,cfg,bucket", [(16, 1, PBD_SCHEME, 8), (32, 4, baseline_config(), 8),
                                                        (64, 40, baseline_config(), 16)])
def test_bytes_per_cell(lib, nodes, filaments, cfg, bucket):  # noqa: F811
    side, n = 512, 3
    pairs, bends = scenarios.line_topology([nodes] * filaments)
    N = nodes * filaments
    st, h = _create([(side, side, N, pairs, bends, cfg, 0.01)] * n)
    assert st == _lib.MC_OK
    size = lib.mc_plan_workspace_bytes(h)
    lib.mc_plan_destroy(h)
    cells = n * side * side
    # per contribution at most 220 B (its weight, slot, run row and the touched cell's state), per node
    # and side a few arrays
    rest = n * (N * cfg.ibm_kernel_size ** 2 * 220 + N * 200 + side * 100 + 16384)
    per_cell = 72 + 8 + 8 + 8 + 4 * bucket
    assert per_cell * cells <= size <= per_cell * cells + rest, (size / cells, per_cell)
