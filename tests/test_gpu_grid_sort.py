"""The grid sort in one kernel against the separate kernels (rebuild_per_sm = -1), and the recorded
candidates against the search through FP64 records (dem_grid = 1): the states are equal bit for
bit, from a body per grid to cells of dozens of bodies."""
import numpy as np
import pytest

from pe_b200 import _abi, scenes

pytestmark = pytest.mark.gpu


def _crowd(n, small, seed=0):
    """n spheres of radius `small` at random in a box whose cells are sized by one sphere of radius
    1: dozens share a cell and many touch more partners than a sphere records."""
    rng = np.random.default_rng(seed)
    r = np.concatenate([np.full(n, small), [1.0]])
    x = np.concatenate([rng.uniform(0.1, 3.9, (n, 3)), [[2.0, 2.0, 5.0]]])
    return scenes._scene(x, rng.normal(0.0, 0.1, x.shape), r, np.zeros(n + 1),
                         scenes.box_planes([0, 0, 0], [4, 4, 7]), np.zeros(6), np.zeros((0, 15)), [],
                         [scenes.material(1.0, 1e2, 1.0, 1.0, 0.3)], (0.0, 0.0, -9.81), 1e-5, 4, "crowd")


def _scene(name):
    if name.startswith("crowd"):
        return _crowd(int(name[5:]), 0.25)
    n = int(name)
    side = max(4.0, 200.0 * (n / 1048576.0) ** (1.0 / 3.0))
    return scenes.dem_large(n, n=n, dims=(side, side, 2.0 * side + 20.0))


@pytest.mark.parametrize("precision", [_abi.FP64, _abi.MIXED])
@pytest.mark.parametrize("lists", [False, True])
@pytest.mark.parametrize("name", ["1", "2", "255", "2049", "40001", "300007", "crowd700"])
def test_forms_agree(name, lists, precision):
    from pe_b200.engine import Engine
    s = _scene(name)
    out = []
    for kw in ({}, {"rebuild_per_sm": -1}, {"dem_grid": 1}):
        e = Engine(solver=_abi.DEM, precision=precision, neighbor_lists=lists).load_scene(s)
        e.set_tuning(**kw)
        e.step(s.dt, 3)
        e.set_state(s.x, s.v, s.w)   # a second search, from another body order
        e.step(s.dt, 2)
        out.append(e.download())
        e.close()
    for o in out[1:]:
        for a, b in zip(o, out[0]):
            assert np.array_equal(a, b)
