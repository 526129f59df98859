"""The energy kernel's queue of owned row entries at its edges -- rows of 0, 1, 31, 32, 33, 64 and 65
entries J > I -- and the learned term's weight gradients of more replicas than one launch takes (16).
Against the FP64 oracle at the reweighting tests' 1e-10 (1e-9 with the learned term)."""

import numpy as np
import pytest

from oracle import orc
from revsim import Engine, SwEngine, constants as C, diamond as D, mlp

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    import build
    build.build()


def _cluster(n, box=3.0, seed=0):
    """n waters on a grid of 0.22 nm: every pair of molecules is within the cutoff, so that molecule I
    owns n - 1 - I entries."""
    rng = np.random.default_rng(seed)
    g = np.stack(np.meshgrid(*[np.arange(5)] * 3, indexing="ij"), -1).reshape(-1, 3)
    g = g[np.argsort(((g - 2) ** 2).sum(1), kind="stable")][:n]
    o = 1.0 + 0.22 * g + rng.uniform(-0.01, 0.01, (n, 3))
    q = rng.normal(size=(n, 2, 3))
    q /= np.linalg.norm(q, axis=2, keepdims=True)
    x = np.stack([o, o + 0.0957 * q[:, 0], o + 0.0957 * q[:, 1]], 1)
    return x.reshape(-1, 3)


@pytest.mark.parametrize("n", [1, 2, 32, 33, 34, 65, 66])
@pytest.mark.parametrize("inter", ["lj", "buff"])
def test_owned_entries(n, inter):
    x, box = _cluster(n), 3.0
    s, p = orc.make_system(n, box, inter), np.array(C.default_params(inter))
    Eo, go = orc.energy_grads(s, p, x, orc.neighbor_pairs(s, x))
    e = Engine(n, box, inter_type=inter)
    e.set_params(p)
    e.set_state(x, np.zeros_like(x))
    E, g = e.energy_grad()
    e.close()
    assert abs(E[0] - Eo) <= 1e-10 * abs(Eo)
    assert np.abs(g[0] - go).max() <= 1e-10 * np.abs(go).max()


def _groups(n_cl, nt):
    a = mlp.H * mlp.NRBF + mlp.H
    b = a + mlp.H * mlp.H + mlp.H
    per = b + mlp.H + 1
    return [np.arange(n_cl)] + [n_cl + t * per + np.arange(*r) for t in range(nt) for r in ((0, a), (a, b), (b, per))]


def _close(g, ref, groups, tol):
    return all(np.abs(g[i] - ref[i]).max() <= tol * np.abs(ref[i]).max() for i in groups)


@pytest.mark.parametrize("reps", [17, 33])
def test_water_replicas_with_the_learned_term(reps):
    ns = [3 + r % 5 for r in range(reps)]
    box = 3.0
    xs = [_cluster(n, seed=r) for r, n in enumerate(ns)]
    th = mlp.init_params(3) + np.random.default_rng(4).normal(scale=0.05, size=mlp.N_PARAMS)
    p = np.concatenate([C.default_params("lj"), th])
    e = Engine(ns, [box] * reps, precision="fp64", mlp=True)
    e.set_params(p)
    x = np.concatenate(xs)
    e.set_state(x, np.zeros_like(x))
    E, g = e.energy_grad()
    e.close()
    groups = _groups(7, 3)
    for r in range(reps):
        s = orc.make_system(ns[r], box, "lj", mlp=True)
        Eo, go = orc.energy_grads(s, p, xs[r], orc.neighbor_pairs(s, xs[r]))
        assert abs(E[r] - Eo) <= 1e-9 * abs(Eo)
        assert _close(g[r], go, groups, 1e-9), r


@pytest.mark.parametrize("reps", [17, 33])
def test_diamond_replicas_with_the_learned_term(reps):
    th = D.init_mlp_params(3) + np.random.default_rng(8).normal(scale=0.1, size=D.MLP_NPARAMS)
    p = np.concatenate([D.default_params(), th])
    xs = []
    for r in range(reps):
        x, box = D.diamond_coords(3, noise=0.01, seed=60 + r)
        xs.append(x)
    n = len(xs[0])
    rng = np.random.default_rng(9)
    w, ac = rng.normal(size=(reps * n, 3)), rng.normal(size=(reps * n, 3))
    with SwEngine([n] * reps, [box] * reps, precision="fp64", mlp=True) as e:
        e.set_params(p)
        e.set_state(np.concatenate(xs), np.zeros((reps * n, 3)))
        _, _, dth = e.force_vjp(w, ac)
    groups = _groups(7, 1)
    for r in range(reps):
        ref = orc.sw_contract(orc.make_sw_system(n, box, mlp=True), p, xs[r], ac[r * n:(r + 1) * n])
        assert _close(dth[r], ref, groups, 1e-9), r
