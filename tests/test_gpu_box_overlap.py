"""Scenes with moving boxes: the boxes' geometry and step run beside the spheres' kernels on a second
stream.  Steps queued together and steps each waited for give the same states bit for bit, with the
recorded candidates and with the search through FP64 records, also after a new upload of the boxes."""
import numpy as np
import pytest

from pe_b200 import _abi, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["tumbling", "spheres_and_boxes", "boxes_only", "one_box"])
def test_overlapped_steps_agree(name):
    from pe_b200.engine import Engine
    if name == "tumbling":
        s = scenes.tumbling_boxes(3, side=4)
    elif name == "boxes_only":
        s = scenes.tumbling_boxes(4, side=3, spheres=False)
    else:
        s = scenes.spheres_and_boxes(5, sphere_side=20, box_side=4 if name == "spheres_and_boxes" else 1)
        s.mbox_x[:, 2] -= 2.0   # into the spheres
    out = []
    for queued in (True, False):
        for grid in (0, 1):
            e = Engine(solver=_abi.DEM, precision=_abi.FP64).load_scene(s)
            e.set_tuning(dem_grid=grid)
            for again in range(2):
                if again:
                    e.set_state(s.x, s.v, s.w)
                    e.upload_boxes(s.mbox_x, s.mbox_q, s.mbox_v, s.mbox_w, s.mbox_len, s.mbox_mat)
                if queued:
                    e.step(s.dt, 25)
                else:
                    for _ in range(25):
                        e.step(s.dt)
                        e.download_boxes()
            out.append(tuple(e.download()) + tuple(e.download_boxes()))
            e.close()
    for o in out[1:]:
        for a, b in zip(o, out[0]):
            assert np.array_equal(a, b)
