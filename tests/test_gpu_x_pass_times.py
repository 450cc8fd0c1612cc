"""The in-place advection kernel against the two-pass one at the sizes where no third of the
spectrum is empty (64, 128 and 256 points): it is the one that runs, so it must not be the
slower one.  Each time is the least of several averages; the margin is their spread."""

import ctypes
import math
import os

import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def BLD():
    import torch
    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for -m gpu tests")
    import BoundaryLayerDynamics as B
    return B


def _x_pass(BLD, n, precision, members, family):
    from BoundaryLayerDynamics import _capi
    saved = os.environ.get("BLD_X_KERNEL")
    os.environ["BLD_X_KERNEL"] = family
    try:
        dom = BLD.Domain((4 * math.pi, 2 * math.pi, 2.0), BLD.SmoothWall(), BLD.SmoothWall())
        m = BLD.Model((n, n, 16), dom, BLD.incompressible_flow(1 / 180, constant_forcing=1), precision=precision, members=members)
    finally:
        if saved is None:
            del os.environ["BLD_X_KERNEL"]
        else:
            os.environ["BLD_X_KERNEL"] = saved
    name = m.kernels()["advection"]["x"]
    assert name.startswith("k_adv_row<" if family == "inplace" else "k_adv_x2<"), name
    m.prepare()
    best = math.inf
    for _ in range(6):
        p = _capi.BldPhaseTimes()
        _capi.check(m._lib.bld_time_phases(m._h, 40, 3, ctypes.byref(p)))
        best = min(best, p.x_ms[0])
    return best


@pytest.mark.parametrize("n,precision,members", [(42, "fp64", 64), (84, "fp64", 16), (168, "mixed", 4)])
def test_in_place_is_not_slower(BLD, n, precision, members):
    row, two = (_x_pass(BLD, n, precision, members, f) for f in ("inplace", "twopass"))
    assert row < 1.03 * two, (n, precision, row, two)
