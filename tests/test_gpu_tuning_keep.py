"""The library's own choice of the list step's form (dem_split -1) is a tuning like the others: reading and
setting the tuning, or changing another field of it, keeps it, and the autotuner times it."""
import numpy as np
import pytest

from pe_b200 import _abi, scenes

pytestmark = pytest.mark.gpu


def _launches(e, s):
    e.set_state(s.x, s.v, s.w)
    for _ in range(3):    # buffers, capture, the choice by the list entries read back
        e.step(s.dt, 33)
        e.download()
    n0 = e.kernel_launches()
    e.step(s.dt, 64)
    n1 = e.kernel_launches()
    return n1 - n0, e.download()


@pytest.mark.parametrize("change", [{}, {"dem_grid": 1}, {"nbgs_sweeps": 2}, {"dem_variant": 2}])
def test_other_fields_leave_the_choice(change):
    from pe_b200.engine import Engine
    s = scenes.dem_lattice(1, side=12)
    e = Engine(gravity=s.gravity).load_scene(s)
    assert e.tuning()["dem_split"] == -1
    own, ref = _launches(e, s)
    e.set_tuning(**dict(e.tuning(), **change))
    assert e.tuning()["dem_split"] == -1
    again, out = _launches(e, s)
    e.set_tuning(**dict(e.tuning(), dem_split=0))
    plain, out0 = _launches(e, s)
    e.close()
    assert again == own and own < 64 < plain     # one kernel per graph, two per step
    for a, b, c in zip(ref, out, out0):
        assert np.array_equal(a, b) and np.array_equal(a, c)


def test_other_skin_keeps_the_choice():
    from pe_b200.engine import Engine
    s = scenes.dem_lattice(1, side=12)
    e = Engine(gravity=s.gravity).load_scene(s)
    own, _ = _launches(e, s)
    t = e.tuning()
    e.set_tuning(**dict(t, skin=1.5 * t["skin"]))
    assert _launches(e, s)[0] == own
    e.close()


def test_no_cooperative_launches_no_steps_kernel():
    """rebuild_per_sm -1 turns cooperative launches off, the steps kernel's too."""
    from pe_b200.engine import Engine
    s = scenes.dem_lattice(1, side=12)
    e = Engine(gravity=s.gravity).load_scene(s)
    _, ref = _launches(e, s)
    e.set_tuning(**dict(e.tuning(), rebuild_per_sm=-1))
    n, out = _launches(e, s)
    e.close()
    assert n > 64
    for a, b in zip(ref, out):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("precision", [_abi.FP64, _abi.MIXED])
def test_autotune_can_keep_the_choice(precision):
    """A scene whose steps take half the time in one kernel: the tuner leaves the choice in place."""
    from pe_b200.engine import Engine
    s = scenes.dem_lattice(1, side=12)
    e = Engine(gravity=s.gravity, precision=precision).load_scene(s)
    own, _ = _launches(e, s)
    e.set_state(s.x, s.v, s.w)
    t = e.autotune(s.dt, 100)
    assert t["dem_split"] == e.tuning()["dem_split"] == -1
    assert _launches(e, s)[0] == own
    e.close()


@pytest.mark.parametrize("form", [-2, 3])
def test_unknown_forms_are_refused(form):
    from pe_b200.engine import Engine, PeB200Error
    s = scenes.dem_lattice(1, side=4)
    e = Engine(gravity=s.gravity).load_scene(s)
    with pytest.raises(PeB200Error) as ei:
        e.set_tuning(dem_split=form)
    assert ei.value.code == _abi.ERR_ARG
    assert e.tuning()["dem_split"] == -1
    e.close()
