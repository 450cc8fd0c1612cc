"""The in-place Smagorinsky kernel is as accurate as the one whose vertical stress derivatives
do not share their lines with the stresses that are differentiated along x.

Rates of a rough-wall boundary layer (log law with noise, where the vertical derivative of
the wall stress is largest) against the double-precision oracle, in the mixed form, whose
rounding is what is compared: the ratio of the two kernels' errors over 1e5 values and three
states scatters by less than half a percent."""

import math
import os

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def BLD():
    import torch
    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for -m gpu tests")
    import BoundaryLayerDynamics as B
    return B


def _les(api, res, eta, **kw):
    dom = api.Domain((2 * math.pi, math.pi, 1.0), api.RoughWall(1e-4), api.FreeSlipBoundary(),
                     *([api.SinusoidalMapping(eta)] if eta else []))
    return api.Model(res, dom, api.incompressible_flow(1e-5, constant_forcing=1, sgs_model=api.StaticSmagorinskyModel()), **kw)


@pytest.mark.parametrize("res,eta", [((64, 64, 32), None), ((64, 64, 48), 0.8), ((96, 64, 40), None), ((128, 64, 48), None)])
def test_error_of_the_rates(oracle, BLD, res, eta):
    om = _les(oracle, res, eta)
    models = {}
    for family in ("", "twopass"):
        saved = os.environ.get("BLD_SGS_X_KERNEL")
        os.environ["BLD_SGS_X_KERNEL"] = family
        try:
            models[family] = _les(BLD, res, eta, precision="mixed")
        finally:
            if saved is None:
                del os.environ["BLD_SGS_X_KERNEL"]
            else:
                os.environ["BLD_SGS_X_KERNEL"] = saved
    error = {family: np.zeros(3) for family in models}
    for seed in range(3):
        rng = np.random.default_rng(seed)
        m = models[""]
        for f in om.fields:
            shape = m.get_field(f).shape
            height = (np.arange(shape[0]) + (1.0 if f == "vel3" else 0.5)) / res[2]
            law = np.log(height[:, None, None] / 1e-4) / 0.4
            m.set_field(f, law * ((f == "vel1") + 0.1 * rng.uniform(-1, 1, shape)))
        st = m.get_state()
        ref = om.compute_rates(st)
        for family, gm in models.items():
            got = gm.compute_rates(st)
            error[family] += [rel_l2(got[f], ref[f]) for f in om.fields]
    assert (error[""] < 1.02 * error["twopass"]).all(), (error, [m.kernels()["sgs"]["x"] for m in models.values()])
