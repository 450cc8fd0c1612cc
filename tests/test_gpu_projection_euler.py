"""The tile projection that forms the Euler stage u + dt f(u) itself, against the oracle.

Layer counts are the edges of its segments: fewer layers than one segment, whole
segments, one layer more and less, and the longer segments above 128 layers; tiles
of 4, 8 and 16 columns, the last one partly past the modes.  One Euler step of a
channel flow, with prescribed forcing and with a prescribed mean flow (whose
correction follows the projection).
"""

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


def _build(api, res, **source):
    dom = api.Domain((4 * math.pi, 2 * math.pi, 2.0), api.SmoothWall(), api.SmoothWall(), api.SinusoidalMapping(0.7))
    return api.Model(res, dom, api.incompressible_flow(1 / 180, **source))


def _forced(BLD, res, tile, **source):
    env = {"BLD_PROJ_TILE": str(tile), "BLD_PROJ_EULER": "1", "BLD_PROJ_PIPE": "0"}
    saved = {k: os.environ.get(k) for k in env}
    os.environ.update(env)
    try:
        return _build(BLD, res, **source)
    finally:
        for k, v in saved.items():
            if v is None:
                del os.environ[k]
            else:
                os.environ[k] = v


@pytest.mark.parametrize("n3", [3, 7, 8, 9, 40, 96, 127, 136, 200])
@pytest.mark.parametrize("tile", [4, 8, 16])
@pytest.mark.parametrize("source", [dict(constant_forcing=1), dict(constant_flux=10.0)])
def test_euler_stage_in_the_tile(oracle, BLD, n3, tile, source):
    res = (12, 10, n3)
    om, gm = _build(oracle, res, **source), _forced(BLD, res, tile, **source)
    rng = np.random.default_rng(n3)
    st = {}
    for f in om.fields:
        shape = om.state[f].shape
        st[f] = rng.standard_normal(shape) + 1j * rng.standard_normal(shape)
        st[f][:, 0, 0] = st[f][:, 0, 0].real
    gm.set_state(st)
    om.state.update({f: v.copy() for f, v in st.items()})
    om.evolve(1e-4, 1e-4, method=oracle.Euler)
    gm.evolve(1e-4, 1e-4, method=BLD.Euler)
    for f in om.fields:
        e = rel_l2(gm.state[f], om.state[f])
        assert e < 1e-12, (n3, tile, f, e)
