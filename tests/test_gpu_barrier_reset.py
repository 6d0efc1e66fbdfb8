"""A wait that ran out leaves arrivals in the grid barriers' words.  The self-test leaves them as a block
that gave up does; once the timeout is reported the words are as new, and the steps that follow give
the states of a context without it, bit for bit, in every form whose kernels meet at such barriers."""
import numpy as np
import pytest

from pe_b200 import _abi, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [_abi.FP64, _abi.MIXED])
@pytest.mark.parametrize("case", ["steps", "form0", "form1", "form2", "grid", "packed"])
def test_steps_after_a_timeout(case, precision):
    from pe_b200.engine import Engine
    kw = {}
    if case == "packed":
        s = scenes.nbgs_box(2, n=1500, mu=0.3, dims=(10.0, 10.0, 60.0), dense=True)
        kw = dict(solver=_abi.HCSITS, relaxation_model=1, max_iterations=20)
    else:
        s = scenes.dem_lattice(1, side=12)
        s.v *= 40.0   # the lists are rebuilt within the steps
        kw = dict(neighbor_lists=case != "grid")
    out = []
    for timeout in (False, True):
        e = Engine(precision=precision, gravity=s.gravity, **kw).load_scene(s)
        if case.startswith("form"):
            e.set_tuning(dem_split=int(case[4]))
        for steps in (20, 1, 38):
            e.step(s.dt, steps)
            if timeout:
                assert e.selftest_timeout(polls=2000) == _abi.ERR_TIMEOUT
        out.append(e.download())
        e.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
