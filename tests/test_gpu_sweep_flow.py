"""The sweeps without barriers (the automatic form of hard-contact steps beyond a few contacts)
against the cooperative grid form (nbgs_sweeps = 2): the updates of every body come in the same
order, so the states are equal bit for bit."""
import numpy as np
import pytest

from pe_b200 import _abi, scenes

pytestmark = pytest.mark.gpu


def _run(s, precision, model, sweeps, steps, mode, residual=False):
    from pe_b200.engine import Engine
    e = Engine(solver=_abi.HCSITS, precision=precision, relaxation_model=model,
               max_iterations=sweeps).load_scene(s)
    e.set_tuning(nbgs_sweeps=mode)
    e.set_residual(residual)
    for k in steps:
        e.step(s.dt, k)
    out = e.download() + (e.download_boxes() if s.nmbox else ())
    st = e.stats()
    e.close()
    return out, st


def _equal(a, b):
    for x, y in zip(a[0], b[0]):
        assert np.array_equal(x, y)
    assert a[1]["contacts"] == b[1]["contacts"] and a[1]["colors"] == b[1]["colors"]
    assert a[1]["contacts"] > 768     # beyond the compact single-block form


@pytest.mark.parametrize("precision", [_abi.FP64, _abi.MIXED])
@pytest.mark.parametrize("model", [0, 1, 2, 3, 4, 5])
def test_models(precision, model):
    s = scenes.nbgs_box(1, n=4111, dims=(16.0, 16.0, 40.0), dense=True)
    s.materials[:, 2:4] = 0.2
    if model >= 2:
        s.materials[:, 0] = 1000.0    # as in the relaxation models' own dense test
    _equal(_run(s, precision, model, 20, (2,), 0), _run(s, precision, model, 20, (2,), 2))


@pytest.mark.parametrize("precision", [_abi.FP64, _abi.MIXED])
@pytest.mark.parametrize("n,width,sweeps", [(1100, 9.0, 1), (1500, 10.0, 100), (131071, 51.0, 7)])
def test_sizes_and_graphs(precision, n, width, sweeps):
    """From a few hundred contacts in small colours to more contacts than the launch has lanes;
    the 17 steps of the smaller ones include a replayed graph."""
    s = scenes.nbgs_box(2, n=n, mu=0.3, dims=(width, width, 60.0), dense=True)
    steps = (1, 2) if n > 100000 else (1, 17)
    _equal(_run(s, precision, 1, sweeps, steps, 0), _run(s, precision, 1, sweeps, steps, 2))


@pytest.mark.parametrize("layers,per_side,model", [(5, 4, 0), (6, 6, 1)])
def test_moving_boxes(layers, per_side, model):
    s = scenes.box_stack(layers, per_side, overlap=0.0)
    _equal(_run(s, _abi.FP64, model, 40, (2,), 0), _run(s, _abi.FP64, model, 40, (2,), 2))


def test_residual_and_last_change():
    s = scenes.nbgs_box(3, n=3001, mu=0.4, dims=(14.0, 14.0, 60.0), dense=True)
    a = _run(s, _abi.FP64, 1, 30, (1, 1), 0, True)
    b = _run(s, _abi.FP64, 1, 30, (1, 1), 2, True)
    _equal(a, b)
    assert a[1]["delta_max"] == b[1]["delta_max"] and a[1]["residual"] == b[1]["residual"]
