"""The in-place x kernels (k_adv_row, and k_sgs_x on rows) against the oracle.

Sizes are the edges of their shapes: the smallest lines, odd second radices (no
padding between blocks), radices that leave lanes of a warp idle, one and two rows
per block, row counts that are not multiples of four, the fewest layers, one layer
per z chunk, and several members with one inactive.  Tolerances are those of the
other kernel families: 1e-12 in double precision and 1e-5 in the mixed form.
"""

import math

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


def _les(api, res, **kw):
    dom = api.Domain((2 * math.pi, math.pi, 1.0), api.RoughWall(1e-4), api.FreeSlipBoundary(),
                     api.SinusoidalMapping(0.5))
    procs = api.incompressible_flow(1e-5, constant_forcing=1, sgs_model=api.StaticSmagorinskyModel())
    return api.Model(res, dom, procs, **kw)


def _state(om, seed):
    rng = np.random.default_rng(seed)
    st = {}
    for f in om.fields:
        shape = om.state[f].shape
        k1 = np.arange(shape[2])[None, None, :]
        k2 = np.abs(om.grid.wavenumbers(2))[None, :, None]
        st[f] = (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)) / (1.0 + k1 ** 2 + k2 ** 2)
    om.apply_projections(st)
    return st


@pytest.mark.parametrize("res", [(12, 12, 3), (18, 16, 5), (23, 30, 4), (50, 42, 7), (70, 54, 6), (98, 16, 9),
                                 (100, 84, 17), (108, 10, 4), (150, 14, 5), (192, 12, 6), (252, 16, 4),
                                 (256, 18, 5), (320, 12, 4), (64, 35, 5)])
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("mixed", 1e-5)])
def test_les_rates(oracle, BLD, res, precision, tol):
    om, gm = _les(oracle, res), _les(BLD, res, precision=precision)
    names = gm.kernels()
    P = names["advection"]["P"][0]
    if P <= 432:
        assert names["advection"]["x"].startswith("k_adv_row<"), names
    assert names["sgs"]["x"].startswith("k_sgs_x<"), names
    st = _state(om, seed=sum(res))
    ref, got = om.compute_rates(st), gm.compute_rates(st)
    for f in om.fields:
        e = rel_l2(got[f], ref[f])
        assert e < tol, (res, precision, f, e, names)


@pytest.mark.parametrize("res", [(512, 8, 4), (384, 6, 5)])
def test_les_rates_long_rows_mixed(oracle, BLD, res):
    """The radix-32 and radix-24 lines (768 and 576 points for advection)."""
    om, gm = _les(oracle, res), _les(BLD, res, precision="mixed")
    assert gm.kernels()["advection"]["x"].startswith("k_adv_row<"), gm.kernels()
    st = _state(om, seed=9)
    ref, got = om.compute_rates(st), gm.compute_rates(st)
    for f in om.fields:
        e = rel_l2(got[f], ref[f])
        assert e < 1e-5, (res, f, e)


def test_members_and_mask(oracle, BLD):
    """Three members of one handle with one switched off: the others advance as alone."""
    res = (30, 28, 6)
    om = _les(oracle, res)
    gm = _les(BLD, res, members=3)
    states = [_state(om, seed=20 + m) for m in range(3)]
    for m, st in enumerate(states):
        gm.set_state(st, member=m)
    gm.prepare()
    before = gm.get_state(1)
    gm.set_active([1, 0, 1])
    gm.step(3, 1e-4)
    for m in (0, 2):
        alone = _les(BLD, res)
        alone.set_state(states[m])
        alone.prepare()
        alone.step(3, 1e-4)
        got, ref = gm.get_state(m), alone.get_state(0)
        for f in om.fields:
            assert rel_l2(got[f], ref[f]) < 1e-13, (m, f)
    for f in om.fields:
        assert np.array_equal(gm.get_state(1)[f], before[f]), f


@pytest.mark.parametrize("res,les", [((16, 16, 8), True), ((64, 64, 32), True), ((96, 96, 48), True), ((64, 48, 33), False),
                                     ((192, 192, 24), False)])
@pytest.mark.parametrize("method", ["SSPRK33", "SSPRK22", "Euler", "AB2"])
def test_overlapped_launches_change_nothing(oracle, BLD, res, les, method):
    """Step graphs whose kernels are set up while the one before them ends give the bits of
    graphs without (the kernels and their order are the same)."""
    import os
    if les:
        om = _les(oracle, res)
        build = lambda: _les(BLD, res)
    else:
        dom = lambda api: api.Domain((4 * math.pi, 2 * math.pi, 2.0), api.SmoothWall(), api.SmoothWall())
        procs = lambda api: api.incompressible_flow(1 / 180, constant_forcing=1)
        om = oracle.Model(res, dom(oracle), procs(oracle))
        build = lambda: BLD.Model(res, dom(BLD), procs(BLD))
    st = _state(om, seed=31)
    out = []
    for off in ("0", "1"):
        saved = os.environ.get("BLD_NO_OVERLAP")
        os.environ["BLD_NO_OVERLAP"] = off
        try:
            gm = build()
            gm.set_state(st)
            gm.prepare()
            gm.step(7, 1e-4, method)
            out.append(gm.get_state())
        finally:
            if saved is None:
                del os.environ["BLD_NO_OVERLAP"]
            else:
                os.environ["BLD_NO_OVERLAP"] = saved
    for f in om.fields:
        assert np.array_equal(out[0][f], out[1][f]), (res, method, f)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_bounded_wait_timeout_exit(oracle, BLD, precision):
    """With the device's wait limit at 0 the kernels take their timeout exit and the call
    reports BLD_ERR_TIMEOUT; with the limit restored the handle is exact again."""
    from BoundaryLayerDynamics import _capi
    res = (64, 12, 6)
    om, gm = _les(oracle, res), _les(BLD, res, precision=precision)
    st = _state(om, seed=17)
    lib = _capi.load()
    _capi.check(lib.bld_set_wait_limit(0, 0))
    try:
        with pytest.raises(_capi.BldError) as err:
            gm.compute_rates(st)
        assert err.value.status == _capi.BLD_ERR_TIMEOUT, err.value
    finally:
        _capi.check(lib.bld_set_wait_limit(0, -1))
    ref, got = om.compute_rates(st), gm.compute_rates(st)
    for f in om.fields:
        assert rel_l2(got[f], ref[f]) < (1e-12 if precision == "fp64" else 1e-5), f
