"""The list step's form picked by the library (and, for scenes in contact, changed between calls)
against the plain form set by the caller: the same states bit for bit."""
import numpy as np
import pytest

from pe_b200 import _abi, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [_abi.FP64, _abi.MIXED])
@pytest.mark.parametrize("kind,n", [("dense", 13), ("dense", 30), ("dense", 86), ("large", 120000),
                                    ("large", 650001), ("two_materials", 31)])
def test_picked_form_agrees(kind, n, precision):
    from pe_b200.engine import Engine
    if kind == "large":
        side = 200.0 * (n / 1048576.0) ** (1.0 / 3.0)
        s = scenes.dem_large(3, n=n, dims=(side, side, 2.0 * side + 20.0))
    else:
        s = scenes.dem_dense(3, nx=n, ny=n, nz=n)
        if kind == "two_materials":
            s.materials = np.concatenate([s.materials, [scenes.material(2.0, 5e4, 20.0, 30.0, 0.2)]])
            s.mat[::3] = 1
            s.plane_mat[::2] = 1
    out = []
    for pick in (True, False):
        e = Engine(solver=_abi.DEM, precision=precision).load_scene(s)
        if not pick:
            e.set_tuning()
        for steps in (1, 33, 40, 17):
            e.step(s.dt, steps)
        out.append(e.download())
        assert e.validate() == 0
        e.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("precision", [_abi.FP64, _abi.MIXED])
@pytest.mark.parametrize("case", ["one", "lattice", "rebuilds", "overflow", "batch", "75776", "75777",
                                  "113664", "113665"])
def test_steps_kernel_agrees(case, precision):
    """Small scenes run many steps in one kernel; a caller that sets the tuning gets a launch per
    step.  From one sphere to the largest scene of either precision and one more, through rebuilds,
    a list buffer that overflows, and calls of odd and even step counts."""
    from pe_b200.engine import Engine
    kw, dt_scale = {}, 1.0
    if case == "one":
        ss = [scenes.dem_lattice(1, side=1)]
    elif case == "batch":
        ss = scenes.batched_ensemble(2, scenes=9, nmin=20, nmax=900)
    elif case in ("lattice", "rebuilds"):
        ss = [scenes.dem_lattice(1, side=11)]
        if case == "rebuilds":
            ss[0].v *= 40.0
    elif case == "overflow":
        ss = [scenes.dem_dense(4, nx=9, ny=9, nz=9)]
        kw["max_contacts"] = 64
    else:
        n = int(case)
        side = 200.0 * (n / 1048576.0) ** (1.0 / 3.0)
        ss = [scenes.dem_large(3, n=n, dims=(side, side, 2.0 * side + 20.0))]
    out = []
    for pick in (True, False):
        e = Engine(solver=_abi.DEM, precision=precision, gravity=ss[0].gravity, **kw)
        e.load_scene(ss[0]) if len(ss) == 1 else e.load_scenes(ss)
        if not pick:
            e.set_tuning()
        for steps in (1, 2, 7, 33, 16, 40):
            e.step(ss[0].dt, steps)
            mid = e.download()
        e.set_state(*[np.concatenate([getattr(s, f) for s in ss]) for f in "xvw"])
        e.step(ss[0].dt, 19)
        st = e.neighbor_list_stats()
        if case == "rebuilds":
            assert st["rebuilds"] > 4
        out.append(tuple(mid) + tuple(e.download()))
        e.close()
    for a, b in zip(*out):
        if case == "overflow":   # the buffer grows a few steps earlier or later: another sum order
            assert np.abs(a - b).max() <= 1e-9 * max(1.0, np.abs(b).max()) * (
                1.0 if precision == _abi.FP64 else 1e5)
        else:
            assert np.array_equal(a, b)
