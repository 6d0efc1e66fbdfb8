"""Hard-contact steps planned without contacts, for a few and for any number: a call whose contacts
outgrow its plan repeats the rest under the full one.  One step per call and all steps in one call
give the same states bit for bit."""
import numpy as np
import pytest

from pe_b200 import _abi, scenes

pytestmark = pytest.mark.gpu


def _falling(n_floor, n_cloud):
    """n_floor spheres resting on the floor well apart, and a lattice of n_cloud that lands on the
    floor within a few steps: few contacts, then many."""
    s = scenes.nbgs_box(3, n=n_floor + n_cloud, mu=0.3, dims=(100.0, 100.0, 40.0))
    k = np.arange(n_floor + n_cloud)
    s.r[:] = 0.5
    s.x[:, 0] = (k % 60) * 1.5 + 1.0
    s.x[:, 1] = (k // 60) * 1.5 + 1.0
    s.x[:, 2] = 0.5 - 1e-4
    s.x[n_floor:, 2] = 0.52
    s.v[:] = 0.0
    s.v[n_floor:, 2] = -1.0
    return s


@pytest.mark.parametrize("precision", [_abi.FP64, _abi.MIXED])
@pytest.mark.parametrize("n_floor,n_cloud", [(0, 3), (5, 20), (90, 60), (130, 10), (90, 1500)])
def test_plans_agree(n_floor, n_cloud, precision):
    from pe_b200.engine import Engine
    s = _falling(n_floor, n_cloud)
    out = []
    for calls in ((1,) * 44, (3, 41), (20, 24)):
        e = Engine(solver=_abi.HCSITS, precision=precision, relaxation_model=1,
                   max_iterations=20).load_scene(s)
        for again in range(2):
            if again:   # the plans of the first run's end meet its beginning
                e.set_state(s.x, s.v, s.w)
            for k in calls:
                e.step(s.dt, k)
        out.append(e.download())
        assert e.stats()["contacts"] >= n_floor
        e.close()
    for o in out[1:]:
        for a, b in zip(o, out[0]):
            assert np.array_equal(a, b)
