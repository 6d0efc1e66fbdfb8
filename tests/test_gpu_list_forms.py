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
