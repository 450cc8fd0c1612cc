"""Pinned host arrays may change as soon as an upload has returned: the copy into them is
only enqueued, and the call waits for it."""

import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("res", [(24, 24, 24), (96, 96, 135)])    # 0.1 and 9.8 MB a field
def test_pinned_upload_may_be_overwritten(res):
    import torch
    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for -m gpu tests")
    import BoundaryLayerDynamics as B
    from BoundaryLayerDynamics import _capi
    dom = B.Domain((2 * math.pi, math.pi, 1.0), B.SmoothWall(), B.FreeSlipBoundary())
    m = B.Model(res, dom, B.incompressible_flow(1e-3))
    fields = ("vel1", "vel2", "vel3")
    rng = np.random.default_rng(1)
    for _ in range(5):
        want = {f: rng.standard_normal(m.zeros(f).shape) + 1j * rng.standard_normal(m.zeros(f).shape) for f in fields}
        pinned = [torch.from_numpy(want[f].copy()).pin_memory() for f in fields]
        _capi.check(m._lib.bld_set_state(m._h, 0, *[p.data_ptr() for p in pinned]))
        for p in pinned:
            p.zero_()
        got = m.get_state()
        for f in fields:
            assert np.array_equal(got[f], want[f]), (res, f)
