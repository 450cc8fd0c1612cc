"""The in-place x kernels and the line y passes are the ones that run by default.

Sizes at both ends and in the middle of those they are compiled for, in both precision
forms; and sizes above them, where the other families run.
"""

import math
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def BLD():
    import torch
    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for -m gpu tests")
    import BoundaryLayerDynamics as B
    return B


def _les(BLD, res, **kw):
    dom = BLD.Domain((2 * math.pi, math.pi, 1.0), BLD.RoughWall(1e-4), BLD.FreeSlipBoundary())
    return BLD.Model(res, dom, BLD.incompressible_flow(1e-5, constant_forcing=1, sgs_model=BLD.StaticSmagorinskyModel()), **kw)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n", [12, 16, 30, 64, 98, 100, 128, 192, 252])
def test_in_place_and_line_kernels(BLD, n, precision):
    m = _les(BLD, (n, n, 4), precision=precision)
    k = m.kernels()
    assert k["advection"]["x"].startswith("k_adv_row<"), k
    assert k["sgs"]["x"].startswith("k_sgs_x<") and k["sgs"]["x"].endswith(", in place>"), k
    for space in ("advection", "sgs"):
        assert k[space]["inv_y"].startswith("k_inv_yl<") and k[space]["fwd_y"].startswith("k_fwd_yl<"), k


def test_other_families_above(BLD):
    k = _les(BLD, (384, 384, 3)).kernels()          # double precision: in place up to 324 and 432 points
    assert not k["sgs"]["x"].endswith(", in place>") and not k["advection"]["x"].startswith("k_adv_row<"), k
    assert not any(k[s][d].startswith(("k_inv_yl<", "k_fwd_yl<")) for s, d in (("advection", "inv_y"), ("advection", "fwd_y"))), k


@pytest.mark.parametrize("switch,space,kernel", [
    ({"BLD_X_KERNEL": "inplace"}, "advection", "k_adv_row<"),
    ({"BLD_X_KERNEL": "block"}, "advection", "k_adv_x<"),
    ({"BLD_SGS_X_KERNEL": "twopass"}, "sgs", "k_sgs_x<"),
])
def test_switches(BLD, switch, space, kernel):
    saved = {k: os.environ.get(k) for k in switch}
    os.environ.update(switch)
    try:
        k = _les(BLD, (64, 12, 6)).kernels()
    finally:
        for v, old in saved.items():
            if old is None:
                del os.environ[v]
            else:
                os.environ[v] = old
    assert k[space]["x"].startswith(kernel), k
    if space == "sgs":      # the two-pass lines, on the layout of nine terms that the line passes do not write
        assert k[space]["x"].endswith(", 0, 64>") and not k[space]["inv_y"].startswith("k_inv_yl<"), k


@pytest.mark.parametrize("lines", ["lines", "block"])
def test_line_switch(BLD, lines):
    saved = os.environ.get("BLD_Y_KERNEL")
    os.environ["BLD_Y_KERNEL"] = lines
    try:
        k = _les(BLD, (64, 12, 6)).kernels()
    finally:
        if saved is None:
            del os.environ["BLD_Y_KERNEL"]
        else:
            os.environ["BLD_Y_KERNEL"] = saved
    assert k["sgs"]["fwd_y"].startswith("k_fwd_yl<") == (lines == "lines"), k
