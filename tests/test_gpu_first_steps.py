"""The first steps of a model, or of a new time step, before graphs are made for them.

A few steps are enqueued kernel by kernel, so that a short run and a time step that
changes from call to call pay for no graph; the same kernels in the same order give the
same bits as the graphs that follow.  A call makes the graphs that it launches, and an
ensemble only its parents' executable form.
"""

import math

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


def _model(BLD, res=(16, 12, 8), les=True, **kw):
    if les:
        dom = BLD.Domain((2 * math.pi, math.pi, 1.0), BLD.RoughWall(1e-4), BLD.FreeSlipBoundary())
        procs = BLD.incompressible_flow(1e-5, constant_forcing=1, sgs_model=BLD.StaticSmagorinskyModel())
    else:
        dom = BLD.Domain((4 * math.pi, 2 * math.pi, 2.0), BLD.SmoothWall(), BLD.SmoothWall())
        procs = BLD.incompressible_flow(1 / 180, constant_flux=1.0)
    return BLD.Model(res, dom, procs, **kw)


def _state(m, seed=3):
    rng = np.random.default_rng(seed)
    st = {}
    for f in ("vel1", "vel2", "vel3"):
        shape = m.zeros(f).shape
        st[f] = 0.1 * (rng.standard_normal(shape) + 1j * rng.standard_normal(shape))
        st[f][:, 0, 0] = 5.0
    return st


def _start(m):
    m.set_state(_state(m))
    m.prepare()


def _graphs(m):
    return m.kernels()["step_graphs"]


def test_graphs_are_made_once_they_pay(BLD):
    m = _model(BLD)
    _start(m)
    for _ in range(4):
        m.step(1, 1e-4)
    assert _graphs(m) == 0
    m.step(1, 1e-4)
    assert _graphs(m) == 1
    for k in range(300):      # a time step of its own in every call
        m.step(1, 1e-5 * (2 + k % 290) / 300)
    assert _graphs(m) == 1


def test_a_call_makes_the_graphs_it_launches(BLD):
    m = _model(BLD)
    _start(m)
    m.step(2, 1e-4)
    m.step(2, 1e-4)
    assert _graphs(m) == 0
    m.step(2, 1e-4)          # a first and a last step, none between
    assert _graphs(m) == 2
    m.step(3, 1e-4)
    assert _graphs(m) == 3
    n = _model(BLD)
    _start(n)
    n.step(9, 1e-4)
    assert _graphs(n) == 3


@pytest.mark.parametrize("les", [True, False])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("method", ["SSPRK33", "SSPRK22", "Euler", "AB2"])
@pytest.mark.parametrize("steps", [[1, 1, 1], [3], [2, 1]])
def test_enqueued_steps_give_the_bits_of_graph_steps(BLD, les, precision, method, steps):
    m = _model(BLD, les=les, precision=precision)
    out = []
    for _ in range(2):
        m.set_state(_state(m))
        m.prepare()
        m.profiles_start()
        for n in steps:
            m.step(n, 1e-4, method)
        out.append([m.get_state()[f] for f in ("vel1", "vel2", "vel3")] + [np.asarray(m.profiles_read())])
        m.step(7, 1e-4, method)      # enough for the graphs of the second pass ...
        m.step(1, 1e-4, method)
        m.step(2, 1e-4, method)
    assert _graphs(m) > 0
    for a, b in zip(*out):
        assert np.array_equal(a, b), (les, precision, method, steps)


def test_ensemble_makes_parents_only(BLD):
    from BoundaryLayerDynamics.ensemble import Ensemble
    models = [_model(BLD, (12, 12, 6)), _model(BLD, (16, 16, 8), members=2)]
    for m in models:
        for k in range(m.members):
            m.set_state(_state(m, k), member=k)
    ens = Ensemble(models)
    ens.prepare()
    ens.step(1, 1e-4)
    assert sorted(map(_graphs, models)) == [0, 1]
    ens.step(2, 1e-4)
    assert sorted(map(_graphs, models)) == [0, 3]
    ens.step(4, 1e-4)
    assert sorted(map(_graphs, models)) == [0, 4]
