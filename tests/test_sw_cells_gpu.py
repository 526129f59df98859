"""The diamond engine's cell scan and terms where their split changes: replicas of unequal size, one
of them with more cells than a pass of its scan takes (2,048), atoms across the box's faces; and the
derivatives away from the default parameters, where no tangent vanishes by chance."""

import numpy as np
import pytest

from oracle import orc
from revsim import SwEngine, diamond as D

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    import build
    build.build()


def _nrel(a, b):
    return np.linalg.norm(np.asarray(a) - np.asarray(b)) / np.linalg.norm(np.asarray(b))


def test_cells_of_unequal_replicas():
    """13 unit cells a side: 16 list cells a side, two passes.  FP64 sums of at most a few hundred
    terms in another order: 1e-10 relative."""
    boxes, xs = [], []
    for k, cells in enumerate((3, 13, 4)):
        x, box = D.diamond_coords(cells, noise=0.01, seed=20 + k)
        xs.append((x + 0.37 * box) % box)
        boxes.append(box)
    e = SwEngine([len(x) for x in xs], boxes, precision="fp64")
    e.set_params(D.default_params())
    e.set_state(np.concatenate(xs), np.zeros((sum(map(len, xs)), 3)))
    F = e.forces()
    e.close()
    o = 0
    for x, box in zip(xs, boxes):
        s = orc.make_sw_system(len(x), box)
        assert _nrel(F[o:o + len(x)], orc.sw_forces(s, D.default_params(), x)) < 1e-10
        o += len(x)


@pytest.mark.parametrize("prec,tol", [("fp64", 1e-9), ("mixed", 1e-4)])
def test_parameter_tangents(prec, tol):
    """The VJP and the dtheta contraction with every parameter moved by a few per cent."""
    x, box = D.diamond_coords(3, noise=0.012, seed=9)
    p = np.array(D.default_params()) * np.array([1.03, 0.96, 1.02, 0.95, 1.04, 0.99, 1.05])
    rng = np.random.default_rng(10)
    w, ac = rng.normal(size=x.shape), rng.normal(size=x.shape)
    s = orc.make_sw_system(len(x), box)
    Fo, Go, J = orc.sw_forces_grads(s, p, x, w)
    dpo = (ac.reshape(-1)[:, None] * J).sum(axis=0)
    e = SwEngine(len(x), box, precision=prec)
    e.set_params(p)
    e.set_state(x, np.zeros_like(x))
    F, G, dp = e.force_vjp(w, ac)
    e.close()
    assert _nrel(F, Fo) < tol and _nrel(G, Go) < tol
    # each derivative against the largest contribution to it that the mixed sums round
    assert np.all(np.abs((dp[0] - dpo) * p) <= tol * np.abs(dpo * p).max()), (dp, dpo)
