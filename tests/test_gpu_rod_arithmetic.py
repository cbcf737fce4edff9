"""The chain rods' branch-free square root, reciprocal, quotients and one-period modulo against the
plain operations, and whole rods on the fast and on the general path: the same bits wherever the
fast path says that it holds.  No tolerance: each is stated to be correctly rounded over its range.
The root and the reciprocal over every significand; quotients, directions and the modulo over
half a billion random operands each, the ends of their ranges among them."""
import ctypes
import os
import subprocess

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from microcosmos_b200 import build  # noqa: E402

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("rod") / "rod_arithmetic.so")
    cmd = [build.nvcc(), *build.ARCH, *build.FLAGS, "-o", so, os.path.join(HERE, "rod_arithmetic.cu")]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    return ctypes.CDLL(so)


def ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def none_differ(call, *args):
    bad = torch.zeros(1, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    assert call(*args, ptr(bad)) == 0
    assert int(bad) == 0, int(bad)


def test_root_of_every_significand(lib):
    """From the bound 2^-50 to 2^38, beyond what components below 2^17 can give."""
    none_differ(lib.check_root, -50, 36)


def test_reciprocal_of_every_significand(lib):
    none_differ(lib.check_reciprocal, -30, 30)


@pytest.mark.parametrize("check", ["check_quotient", "check_unit", "check_modulo"])
def test_random_operands(lib, check):
    none_differ(getattr(lib, check), ctypes.c_uint64(2025))


@pytest.mark.parametrize("solver", [0, 1], ids=["pbd", "cosserat"])
@pytest.mark.parametrize("cycles", [1, 2, 20])
@pytest.mark.parametrize("kind", [0, 1, 2, 3], ids=["ordinary", "coinciding", "far-angle", "far-node"])
def test_rods_on_both_paths(lib, solver, cycles, kind):
    """The same bits where the fast path holds.  It holds for most ordinary rods, and notices operands
    outside its range (a Cosserat rod's angle is pulled to its segment, which has one even where
    two nodes coincide)."""
    rods = 4096
    bad = torch.zeros(1, dtype=torch.int64, device="cuda")
    left = torch.zeros(1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    assert lib.check_rods(rods, ctypes.c_uint64(7 + kind), solver, cycles, kind, ptr(bad), ptr(left)) == 0
    assert int(bad) == 0
    if kind == 0:
        assert int(left) < rods // 2, int(left)
    if kind == 3 or (solver == 0 and kind == 1):
        assert int(left) == rods, int(left)
