"""Scenes with moving boxes step on one stream while the stage timers run, and with the boxes beside the
spheres otherwise: the same states bit for bit, so no kernel of the overlapped step reads what another
one is still to write; and every stage is timed in every step."""
import numpy as np
import pytest

from pe_b200 import _abi, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["tumbling", "spheres_and_boxes", "boxes_only", "one_box"])
@pytest.mark.parametrize("grid", [0, 1])
def test_one_stream_agrees(name, grid):
    from pe_b200.engine import Engine
    if name == "tumbling":
        s = scenes.tumbling_boxes(3, side=4)
    elif name == "boxes_only":
        s = scenes.tumbling_boxes(4, side=3, spheres=False)
    else:
        s = scenes.spheres_and_boxes(5, sphere_side=20, box_side=4 if name == "spheres_and_boxes" else 1)
        s.mbox_x[:, 2] -= 2.0   # into the spheres
    out = []
    for timed in (False, True):
        e = Engine(solver=_abi.DEM, precision=_abi.FP64).load_scene(s)
        e.set_tuning(dem_grid=grid)
        e.set_profiling(timed)
        for steps in (1, 30):
            e.step(s.dt, steps)
        out.append(tuple(e.download()) + tuple(e.download_boxes()))
        if timed and s.n > 0:
            p = e.profile()
            assert p["dem_step"][1] == 31 and p["sort"][1] == 31, p
        e.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
