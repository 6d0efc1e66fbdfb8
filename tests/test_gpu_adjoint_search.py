"""The adjoint's partner search: the recorded candidates, a sphere with more of them than are
recorded, and segments whose searches are not kept."""
import numpy as np
import pytest

from pe_b200 import _abi, scenes
from pe_b200.adjoint import LossSpec, make_single_material, set_params

pytestmark = pytest.mark.gpu


def _engine(s, **kw):
    from pe_b200.engine import Engine
    return Engine(solver=_abi.DEM, precision=_abi.FP64, **kw).load_scene(s)


def _shell(count):
    """`count` spheres of radius 0.1 pressed 0.002 into one of radius 0.3, none touching another."""
    k = np.arange(count) + 0.5
    z = 1.0 - 2.0 * k / count
    a = np.pi * (1.0 + 5.0 ** 0.5) * k
    d = np.stack([np.sqrt(1.0 - z * z) * np.cos(a), np.sqrt(1.0 - z * z) * np.sin(a), z], -1)
    x = np.concatenate([[[1.0, 1.0, 1.0]], 1.0 + 0.398 * d])
    rng = np.random.default_rng(5)
    s = scenes.small_random(0, n=count + 1)
    s.x, s.r = x, np.concatenate([[0.3], np.full(count, 0.1)])
    s.v, s.w = rng.normal(0.0, 0.2, x.shape), rng.normal(0.0, 0.5, x.shape)
    s.planes = scenes.box_planes([0, 0, 0], [2, 2, 2])
    return make_single_material(s, k_n=1e4, c_n=50.0, c_t=40.0, mu=0.3, density=200.0)


@pytest.mark.parametrize("count", [16, 17, 24])
def test_more_candidates_than_recorded(count):
    s, steps = _shell(count), 6
    spec = LossSpec.for_scene(s, z_open=1.0, width=0.3)

    def loss(t):
        e = _engine(t, neighbor_lists=False)
        e.step(t.dt, steps)
        x = e.download()[0]
        e.close()
        return spec.value(x)

    e = _engine(s)
    e.adjoint_forward(steps, s.dt, 3)
    x = e.download()[0]
    gx = spec.grad(x)
    _, gv, _, gp = e.adjoint_backward(gx, np.zeros_like(gx), np.zeros_like(gx))
    e.close()
    fd, ad = [], []
    for i, a in ((0, 2), (1, 2), (count // 2, 0)):
        p, m = s.copy(), s.copy()
        p.v[i, a] += 1e-6
        m.v[i, a] -= 1e-6
        fd.append((loss(p) - loss(m)) / 2e-6)
        ad.append(gv[i, a])
    assert np.abs(np.array(ad) - fd).max() < 1e-4 * np.abs(fd).max() + 1e-10

    def kn(d):
        return set_params(s, 1e4 + d, 50.0, 40.0, 0.3)

    f = (loss(kn(0.1)) - loss(kn(-0.1))) / 0.2
    assert abs(gp[0] - f) < 1e-4 * abs(f) + 1e-9


def test_searches_kept_or_repeated():
    """A segment of 700 states of 21,952 spheres keeps no searches (they would pass the limit), one
    of 35 does: the gradients are equal bit for bit, and so is the state left behind."""
    s = scenes.dem_dense(1, nx=28, ny=28, nz=28)
    rng = np.random.default_rng(2)
    g = [rng.normal(size=s.x.shape) for _ in range(3)]
    out = []
    for every in (700, 35):
        e = _engine(s)
        e.adjoint_forward(700, s.dt, every)
        before = e.download()
        out.append(tuple(before) + tuple(e.adjoint_backward(*g)) + tuple(e.download()))
        e.step(s.dt, 2)
        out[-1] += tuple(e.download())
        e.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
    for a, b in zip(out[0][:3], out[0][7:10]):
        assert np.array_equal(a, b)
