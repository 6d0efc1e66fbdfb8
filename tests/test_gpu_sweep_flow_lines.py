"""Stacks of boxes on both sides of the contact count from which their sweeps run without barriers (1,100
without friction, 96 with it; fewer stay in one block): bit for bit the cooperative grid form's."""
import numpy as np
import pytest

from pe_b200 import _abi, scenes

pytestmark = pytest.mark.gpu


def _run(s, model, mode):
    from pe_b200.engine import Engine
    e = Engine(solver=_abi.HCSITS, precision=_abi.FP64, relaxation_model=model,
               max_iterations=40).load_scene(s)
    e.set_tuning(nbgs_sweeps=mode)
    e.step(s.dt, 2)
    out = e.download_boxes()
    n = e.stats()["contacts"]
    e.close()
    return n, out


@pytest.mark.parametrize("model,line,stacks", [(0, 1100, [(2, 2), (3, 4), (4, 4), (5, 5), (6, 6)]),
                                               (1, 96, [(1, 2), (2, 2), (2, 3), (3, 3), (6, 6)])])
def test_both_sides_of_the_line(model, line, stacks):
    counts = []
    for layers, per_side in stacks:
        s = scenes.box_stack(layers, per_side, overlap=0.0)
        n, out = _run(s, model, 0)
        m, ref = _run(s, model, 2)
        assert n == m
        for a, b in zip(out, ref):
            assert np.array_equal(a, b)
        counts.append(n)
    assert min(counts) <= line < max(counts), counts
