"""Host arrays that cross the C ABI through the staged copies, and around them.

Arrays below and above the size from which the copies are staged, whose parts are
not whole chunks, from several threads at once (one uses the staging buffers, the
others the driver's path), into pageable and pinned memory: the values come back
bit by bit.
"""

import math
import threading

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


def _model(BLD, res):
    dom = BLD.Domain((2 * math.pi, math.pi, 1.0), BLD.SmoothWall(), BLD.FreeSlipBoundary())
    return BLD.Model(res, dom, BLD.incompressible_flow(1e-3))


def _state(m, seed):
    rng = np.random.default_rng(seed)
    return {f: rng.standard_normal(m.zeros(f).shape) + 1j * rng.standard_normal(m.zeros(f).shape)
            for f in ("vel1", "vel2", "vel3")}


# bytes per field: 0.1, 1.96 (below 2 MiB), 2.07, 9.8 MB
@pytest.mark.parametrize("res", [(24, 24, 24), (64, 64, 62), (64, 64, 66), (96, 96, 135)])
def test_round_trip(BLD, res):
    m = _model(BLD, res)
    for seed in range(3):
        st = _state(m, seed)
        m.set_state(st)
        got = m.get_state()
        for f in st:
            assert np.array_equal(got[f], st[f]), (res, f)


def test_threads(BLD):
    models = [_model(BLD, (96, 96, 40)) for _ in range(3)]
    bad = []

    def work(m, seed):
        for r in range(5):
            st = _state(m, 10 * seed + r)
            m.set_state(st)
            got = m.get_state()
            if not all(np.array_equal(got[f], st[f]) for f in st):
                bad.append((seed, r))

    threads = [threading.Thread(target=work, args=(m, k)) for k, m in enumerate(models)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad


def test_pinned_memory(BLD):
    import torch
    m = _model(BLD, (64, 64, 80))
    st = _state(m, 4)
    m.set_state(st)
    out = [torch.empty(m.zeros(f).shape, dtype=torch.complex128).pin_memory() for f in ("vel1", "vel2", "vel3")]
    assert m._lib.bld_get_state(m._h, 0, *[o.data_ptr() for o in out]) == 0
    for f, o in zip(("vel1", "vel2", "vel3"), out):
        assert np.array_equal(o.numpy(), st[f]), f
