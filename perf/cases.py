"""Performance cases of the rigid-body step: what a program that uses this library has it do.

A pass hands a scene's state to its context, advances it by the case's steps and reads the new
state back into host arrays, all through ``pe_b200.Engine``: a program that steps many scenes, or
one scene from many initial states, pays for exactly this.  The scenes are the generators of
``pe_b200.scenes`` at the sizes of the reference configurations and at generic ones.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from pe_b200 import _abi, scenes
from pe_b200.engine import Engine

_MODELS = {"frictionless": _abi.INELASTIC_FRICTIONLESS,
           "coulomb": _abi.APPROX_INELASTIC_COULOMB_DECOUPLING}


def listed():
    return [
        # a program that owns its bodies and calls the library once per time step (the way the
        # collision system inside pe does): a small scene, so launches and copies are all there is
        dict(name="one_step_512", kind="lattice", side=8, precision="fp64", lists=True, steps=1),
        # the plain CPU-runnable configuration, whole: 4096 spheres, 1000 FP64 steps
        dict(name="lattice_4096", kind="lattice", side=16, precision="fp64", lists=True,
             steps=1000),
        # the large configuration, whole: 1M spheres poured at 30% volume, mixed precision
        dict(name="large_1m_mixed", kind="large", n=1048576, precision="mixed", lists=True,
             steps=1000),
        # the plain FP64 form that searches the cell grid every step, an odd body count
        dict(name="grid_600011_fp64", kind="large", n=600011, precision="fp64", lists=False,
             steps=30),
        # a packing where every sphere is in contact every step
        dict(name="dense_1m_mixed", kind="dense", nx=128, ny=128, nz=64, precision="mixed",
             lists=True, steps=200),
        # the batched ensemble: independent scenes of uneven size in one context
        dict(name="ensemble_64_mixed", kind="ensemble", scenes=64, nmin=1024, nmax=65536,
             precision="mixed", lists=True, steps=200),
        # the hard-contact configuration, whole: 32,768 spheres released in a box, 200 steps
        dict(name="settle_32k_mixed", kind="nbgs", n=32768, dense=False, width=40.0,
             precision="mixed", model="frictionless", sweeps=100, steps=200),
        # hard contacts of a settled packing with friction (the default relaxation model)
        dict(name="packed_32k_coulomb", kind="nbgs", n=32768, dense=True, width=32.0,
             precision="mixed", model="coulomb", sweeps=100, steps=16),
        # the same in FP64 without friction, an odd body count
        dict(name="packed_20011_fp64", kind="nbgs", n=20011, dense=True, width=27.0,
             precision="fp64", model="frictionless", sweeps=100, steps=16),
        # moving boxes under the hard-contact solver: a 6 x 6 x 6 stack of cubes
        dict(name="box_stack_216", kind="stack", layers=6, per_side=6, model="coulomb",
             sweeps=100, steps=4),
        # boxes falling onto spheres under the DEM law
        dict(name="boxes_on_spheres", kind="boxes", sphere_side=48, box_side=10, steps=40),
        # gradients: forward run with checkpoints and the adjoint of it
        dict(name="adjoint_16224", kind="adjoint", nx=26, ny=26, nz=24, steps=100, every=25),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["lattice", "large", "grid", "dense", "ensemble", "nbgs", "nbgs", "stack",
                       "boxes", "adjoint"])
    precision = rng.choice(["fp64", "mixed"])
    if kind == "lattice":
        side = _log(rng, 5, 40)
        return dict(kind="lattice", side=side, precision=precision, lists=rng.random() < 0.75,
                    steps=_log(rng, 1, 400))
    if kind in ("large", "grid"):
        return dict(kind="large", n=_log(rng, 2000, 1000000), precision=precision,
                    lists=kind == "large", steps=_log(rng, 4, 400 if kind == "large" else 60))
    if kind == "dense":
        return dict(kind="dense", nx=_log(rng, 12, 120), ny=_log(rng, 12, 120),
                    nz=_log(rng, 6, 60), precision=precision, lists=True, steps=_log(rng, 4, 120))
    if kind == "ensemble":
        k = _log(rng, 4, 64)
        return dict(kind="ensemble", scenes=k, nmin=512, nmax=_log(rng, 2048, 49152),
                    precision=precision, lists=True, steps=_log(rng, 8, 150))
    if kind == "nbgs":
        dense = rng.random() < 0.7
        n = _log(rng, 400, 32000)
        return dict(kind="nbgs", n=n, dense=dense,
                    width=float(math.ceil((n if dense else 4 * n) ** (1.0 / 3.0))),
                    precision=precision, model=rng.choice(["frictionless", "coulomb"]),
                    sweeps=rng.choice([30, 50, 100]), steps=_log(rng, 2, 14 if dense else 100))
    if kind == "stack":
        return dict(kind="stack", layers=rng.randint(2, 6), per_side=rng.randint(2, 6),
                    model=rng.choice(["frictionless", "coulomb"]), sweeps=rng.choice([50, 100]),
                    steps=rng.randint(1, 4))
    if kind == "boxes":
        return dict(kind="boxes", sphere_side=_log(rng, 12, 46), box_side=rng.randint(2, 9),
                    steps=_log(rng, 4, 40))
    return dict(kind="adjoint", nx=rng.randint(8, 25), ny=rng.randint(8, 25),
                nz=rng.randint(6, 22), steps=_log(rng, 10, 90), every=rng.choice([7, 10, 25, 50]))


def _scenes(case, seed):
    kind = case["kind"]
    if kind == "lattice":
        return [scenes.dem_lattice(seed, side=case["side"])]
    if kind == "large":
        # the slab of the large configuration, its cross-section scaled with the body count
        side = max(10.0, 200.0 * (case["n"] / 1048576.0) ** (1.0 / 3.0))
        return [scenes.dem_large(seed, n=case["n"], dims=(side, side, 2.0 * side + 20.0))]
    if kind in ("dense", "adjoint"):
        return [scenes.dem_dense(seed, nx=case["nx"], ny=case["ny"], nz=case["nz"])]
    if kind == "ensemble":
        # the same scene sizes for every seed; positions mirrored or not, velocities drawn anew
        ss = scenes.batched_ensemble(0, scenes=case["scenes"], nmin=case["nmin"],
                                     nmax=case["nmax"])
        rng = np.random.default_rng(seed)
        for s in ss:
            for a in range(2):
                if rng.random() < 0.5:
                    s.x[:, a] = -s.planes[2 * a + 1, 3] - s.x[:, a]
            s.v = rng.normal(0.0, 0.1, size=s.v.shape)
        return ss
    if kind == "nbgs":
        w = case["width"]
        mu = 0.5 if case["model"] == "coulomb" else 0.0
        return [scenes.nbgs_box(seed, n=case["n"], mu=mu, dims=(w, w, 3.0 * w + 10.0),
                                dense=case["dense"])]
    if kind == "stack":
        s = scenes.box_stack(case["layers"], case["per_side"], overlap=0.0)
        rng = np.random.default_rng(seed)
        s.mbox_v = rng.normal(0.0, 0.01, size=s.mbox_v.shape)
        s.mbox_w = rng.normal(0.0, 0.01, size=s.mbox_w.shape)
        return [s]
    if kind == "boxes":
        return [scenes.spheres_and_boxes(seed, sphere_side=case["sphere_side"],
                                         box_side=case["box_side"])]
    raise ValueError(kind)


def _host(a):
    """A copy of `a` in page-locked host memory, as numpy."""
    t = torch.from_numpy(np.ascontiguousarray(a, np.float64))
    return (t.pin_memory() if torch.cuda.is_available() else t.clone()).numpy()


def prepare(case, seed):
    ss = _scenes(case, seed)
    hard = case["kind"] in ("nbgs", "stack")
    kw = {}
    if hard:
        kw = dict(relaxation_model=_MODELS[case["model"]], max_iterations=case["sweeps"])
    e = Engine(solver=_abi.HCSITS if hard else _abi.DEM,
               precision=_abi.MIXED if case.get("precision") == "mixed" else _abi.FP64,
               gravity=ss[0].gravity, neighbor_lists=case.get("lists", True), **kw)
    if len(ss) == 1:
        e.load_scene(ss[0])
    else:
        e.load_scenes(ss)
    x, v, w = (_host(np.concatenate([getattr(s, f) for s in ss])) for f in "xvw")
    state = {"case": case, "e": e, "dt": ss[0].dt, "in": (x, v, w),
             "out": tuple(_host(np.zeros_like(x)) for _ in range(3))}
    if ss[0].nmbox:
        s = ss[0]
        state["boxes"] = (s.mbox_x, s.mbox_q, s.mbox_v, s.mbox_w, s.mbox_len, s.mbox_mat)
    if case["kind"] == "adjoint":
        rng = np.random.default_rng(seed + 7)
        state["grad"] = tuple(_host(rng.normal(0.0, 1.0, size=x.shape)) for _ in range(3))
    return state


def run(state):
    e, case = state["e"], state["case"]
    e.set_state(*state["in"])
    if case["kind"] == "adjoint":
        e.adjoint_forward(case["steps"], state["dt"], case["every"])
        out = e.download(out=state["out"])
        return tuple(out) + tuple(e.adjoint_backward(*state["grad"]))
    if "boxes" in state:
        e.upload_boxes(*state["boxes"])
    e.step(state["dt"], case["steps"])
    out = e.download(out=state["out"])
    if "boxes" in state:
        return tuple(out) + tuple(e.download_boxes())
    return out


def _spheres(case):
    k = case["kind"]
    if k == "lattice":
        return case["side"] ** 3
    if k in ("large", "nbgs"):
        return case["n"]
    if k in ("dense", "adjoint"):
        return case["nx"] * case["ny"] * case["nz"]
    if k == "ensemble":   # the mean of log-uniform counts
        return int(case["scenes"] * (case["nmax"] - case["nmin"])
                   / math.log(case["nmax"] / case["nmin"]))
    if k == "stack":
        return 1
    return case["sphere_side"] ** 3


def work(case):
    """The state in (72 bytes a sphere) and out again; every step reads and writes the state it
    advances (positions and radius in FP64, velocities in the case's precision); every sweep
    reads a contact's frame and masses and reads and writes the corrections of its bodies."""
    k, n, steps = case["kind"], _spheres(case), case["steps"]
    io = 144.0 * n
    real = 4 if case.get("precision") == "mixed" else 8
    state = 2.0 * (32 + 6 * real)
    if k in ("nbgs", "stack"):
        contacts = 0.0
        if k == "stack":
            boxes = case["layers"] * case["per_side"] ** 2
            contacts, n, io = 16.0 * boxes, boxes, 208.0 * boxes
        elif case["dense"]:
            contacts = 0.6 * n
        friction = case["model"] == "coulomb"
        per = (28 if friction else 12) * real + 4 * 6 * real
        return {"bytes": io + steps * (n * state + case["sweeps"] * contacts * per),
                "flops": steps * case["sweeps"] * contacts * (250.0 if friction else 120.0)
                + steps * n * 60.0}
    pairs = {"dense": 3.0, "adjoint": 3.0}.get(k, 0.05) * n
    flops = steps * (40.0 * n + 150.0 * pairs)
    if k == "adjoint":   # forward, recomputation, and the reverse step of about twice the work
        return {"bytes": 2 * io + 4.0 * steps * n * state, "flops": 4 * flops}
    if k == "boxes":
        m = case["box_side"] ** 3
        return {"bytes": io + 208.0 * m + steps * (n * state + m * 208.0),
                "flops": flops + steps * m * 500.0}
    return {"bytes": io + steps * n * state, "flops": flops}


# ---- 64-bit values ------------------------------------------------------------------------------

def _candidates(x, r, scene, skin):
    """Pairs (i < j) of one scene closer than r_i + r_j + skin."""
    n = x.shape[0]
    h = 2.0 * float(r.max()) + skin
    c = torch.floor((x - x.amin(0)) / h).long()
    dim = (c.amax(0) + 1).tolist()

    def key(b, cx, cy, cz):
        return ((scene[b] * dim[2] + cz) * dim[1] + cy) * dim[0] + cx

    own = key(slice(None), c[:, 0], c[:, 1], c[:, 2])
    keys, order = torch.sort(own, stable=True)
    slot = torch.empty_like(order)
    slot[order] = torch.arange(n, device=x.device)
    ii, jj = [], []
    for dz in (0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                if (dz, dy, dx) < (0, 0, 0):
                    continue
                cx, cy, cz = c[:, 0] + dx, c[:, 1] + dy, c[:, 2] + dz
                ok = (cx >= 0) & (cx < dim[0]) & (cy >= 0) & (cy < dim[1]) & (cz < dim[2])
                i = torch.nonzero(ok).squeeze(1)
                t = key(i, cx[i], cy[i], cz[i])
                lo, hi = torch.searchsorted(keys, t), torch.searchsorted(keys, t, right=True)
                if (dx, dy, dz) == (0, 0, 0):
                    lo = slot[i] + 1
                for k in range(int((hi - lo).max()) if i.numel() else 0):
                    m = lo + k < hi
                    a, b = i[m], order[(lo + k)[m]]
                    d2 = ((x[a] - x[b]) ** 2).sum(1)
                    m = d2 < (r[a] + r[b] + skin) ** 2
                    ii.append(a[m])
                    jj.append(b[m])
    i, j = torch.cat(ii), torch.cat(jj)
    return torch.minimum(i, j), torch.maximum(i, j)


class _Dem:
    """The linear spring-dashpot step of spheres between axis-aligned walls, in 64 bits."""

    def __init__(self, ss):
        dev = "cuda" if torch.cuda.is_available() else "cpu"

        def t(a):
            return torch.from_numpy(np.ascontiguousarray(a, np.float64)).to(dev)

        self.r = t(np.concatenate([s.r for s in ss]))
        self.x, self.v, self.w = (t(np.concatenate([getattr(s, f) for s in ss])) for f in "xvw")
        scene = np.repeat(np.arange(len(ss)), [s.n for s in ss])
        self.scene = torch.from_numpy(scene).to(dev)
        mat = np.array([s.materials[0] for s in ss])[scene]   # one material per scene
        m = 4.0 / 3.0 * math.pi * self.r ** 3 * t(mat[:, 0])
        self.im, self.ii = (1.0 / m)[:, None], (1.0 / (0.4 * m * self.r ** 2))[:, None]
        self.kn, self.cn, self.ct, self.mu = (t(f)[:, None] for f in (
            mat[:, 6] / 2, mat[:, 7] / 2, mat[:, 8] / 2, mat[:, 2] * 2))
        self.lo = t(np.array([s.planes[[0, 2, 4], 3] for s in ss])[scene])
        self.hi = t(np.array([-s.planes[[1, 3, 5], 3] for s in ss])[scene])
        self.g, self.dt = t(ss[0].gravity), ss[0].dt
        self.skin = 0.1 * float(self.r.min())
        self.at = None

    def _law(self, n, dist, rvel, q):
        """The force on body 1 of each contact; q: its four coefficients."""
        nvel = (n * rvel).sum(1, keepdim=True)
        fn = torch.clamp(-q[0] * dist - q[1] * nvel, min=0.0)
        vt = n * nvel - rvel
        l2 = (vt * vt).sum(1, keepdim=True)
        some = l2 > 0
        length = torch.sqrt(torch.where(some, l2, torch.ones_like(l2)))
        ft = torch.minimum(q[2] * length, q[3] * fn)
        return fn * n + torch.where(some, ft / length, torch.zeros_like(ft)) * vt

    def step(self, x, v, w, q=None):
        r = self.r[:, None]
        if self.at is None or float((x.detach() - self.at).norm(dim=1).max()) > 0.49 * self.skin:
            self.at = x.detach().clone()
            self.pairs = _candidates(self.at, self.r, self.scene, self.skin)
        i, j = self.pairs
        with torch.no_grad():
            near = (x[i] - x[j]).norm(dim=1) - self.r[i] - self.r[j] < -1e-8
        i, j = i[near], j[near]

        def coef(b):
            return q if q is not None else [c[b] for c in (self.kn, self.cn, self.ct, self.mu)]

        F, T = torch.zeros_like(x), torch.zeros_like(x)
        d = x[i] - x[j]
        length = d.norm(dim=1, keepdim=True)
        dist, n = length - r[i] - r[j], d / length
        r2 = n * (r[j] + 0.5 * dist)
        r1 = r2 - d
        rvel = v[i] + torch.linalg.cross(w[i], r1) - v[j] - torch.linalg.cross(w[j], r2)
        f = self._law(n, dist, rvel, coef(i))
        F = F.index_add(0, i, f).index_add(0, j, -f)
        T = T.index_add(0, i, torch.linalg.cross(r1, f)).index_add(0, j, torch.linalg.cross(r2, -f))
        for a in range(3):
            for sign, at in ((1.0, self.lo), (-1.0, self.hi)):
                with torch.no_grad():
                    gap = sign * (x[:, a] - at[:, a]) - self.r
                    b = torch.nonzero(gap < -1e-8).squeeze(1)
                if b.numel() == 0:
                    continue
                n = torch.zeros(b.numel(), 3, dtype=x.dtype, device=x.device)
                n[:, a] = sign
                dist = (sign * (x[b, a] - at[b, a]) - self.r[b])[:, None]
                r1 = -(r[b] + dist) * n
                f = self._law(n, dist, v[b] + torch.linalg.cross(w[b], r1), coef(b))
                F = F.index_add(0, b, f)
                T = T.index_add(0, b, torch.linalg.cross(r1, f))
        v = v + (F * self.im + self.g) * self.dt
        w = w + T * self.ii * self.dt
        return x + v * self.dt, v, w


def exact(case, seed):
    # the hard-contact sweeps stop before they converge, so their result depends on the order of
    # the contacts; contacts of moving boxes have no short 64-bit restatement
    if case["kind"] in ("nbgs", "stack", "boxes"):
        return None
    d = _Dem(_scenes(case, seed))
    s = (d.x, d.v, d.w)
    if case["kind"] != "adjoint":
        for _ in range(case["steps"]):
            s = d.step(*s)
        return s
    q = [c[0, 0].clone().requires_grad_() for c in (d.kn, d.cn, d.ct, d.mu)]
    start = [a.clone().requires_grad_() for a in s]
    s = start
    for _ in range(case["steps"]):
        s = d.step(*s, q)
    rng = np.random.default_rng(seed + 7)
    g = [torch.from_numpy(rng.normal(0.0, 1.0, size=tuple(d.x.shape))).to(d.x.device) for _ in s]
    grads = torch.autograd.grad(list(s), start + q, g)
    return tuple(a.detach() for a in s) + grads[:3] + (torch.stack(grads[3:]),)
