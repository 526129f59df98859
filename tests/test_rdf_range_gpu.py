"""The RDF loss away from positions inside the box and grid points above 0: atoms far from the origin
(the kernels' FP32 distance test must not decide what it cannot resolve), non-finite positions, and a
grid point at x = 0 that carries no weight.  Against the oracle at the RDF tests' 1e-11."""

import numpy as np
import pytest

from oracle import orc
from revsim import Engine, RdfTerm, constants as C, systems

pytestmark = pytest.mark.gpu

N_MOL, BOX = 150, 2.6


@pytest.fixture(scope="module", autouse=True)
def _built():
    import build
    build.build()


def _loss_grad(x, args):
    e = Engine(N_MOL, BOX)
    e.set_params(C.default_params())
    e.set_state(x, np.zeros_like(x))
    e.set_loss([RdfTerm(*args)])
    l, g = e.loss_grad()
    e.close()
    return l[0], g


@pytest.mark.parametrize("shift", [-1.3, 41.0, 42.0, 1e4, 1e6])
@pytest.mark.parametrize("sel", [(0, 0), (0, 1)])
def test_far_from_the_origin(shift, sel):
    x = systems.water_coords(N_MOL, BOX, seed=3) + shift
    args = (*sel, 0.005, 0.005, 0.0005, 0.04, 200, 0, 1, np.random.default_rng(4).uniform(0.2, 1.5, 200), 2, 0.7)
    lo, go = orc.loss_grad(orc.make_system(N_MOL, BOX), orc.Loss([orc.RdfTerm(*args)]), x)
    l, g = _loss_grad(x, args)
    assert abs(l - lo) <= 1e-11 * abs(lo)
    assert np.linalg.norm(g - go) <= 1e-11 * np.linalg.norm(go)


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_non_finite_positions_have_no_pairs(bad):
    x = systems.water_coords(N_MOL, BOX, seed=3)
    args = (0, 0, 0.005, 0.005, 0.0005, 0.04, 200, 0, 1, np.ones(200), 2, 0.7)
    x[3 * 17] = bad
    l, g = _loss_grad(x, args)
    assert np.isfinite(l) and np.isfinite(g).all() and not g[3 * 17].any()


def test_no_weight_at_zero():
    """Intramolecular O-H pairs reach the point x = 0, where h is infinite; a term of weight 0 has no
    gradient all the same."""
    x = systems.water_coords(N_MOL, BOX, seed=3)
    args = (0, 1, 0.0, 0.005, 0.002, 0.15, 100, 0, 1, np.ones(100), 1, 0.0)
    _, g = _loss_grad(x, args)
    assert not g.any()


@pytest.mark.parametrize("n_mol", [31, 33, 257, 300])
@pytest.mark.parametrize("sel", [(0, 0), (0, 1), (1, 1)])
def test_long_windows(n_mol, sel):
    """Windows of 100 points (a lane per pair, CTAs of less than a tile)."""
    x = systems.water_coords(n_mol, BOX, seed=n_mol)
    args = (*sel, 0.005, 0.005, 0.002, 0.25, 200, 0, 1, np.random.default_rng(n_mol).uniform(0.2, 1.5, 200), 2, 0.7)
    lo, go = orc.loss_grad(orc.make_system(n_mol, BOX), orc.Loss([orc.RdfTerm(*args)]), x)
    e = Engine(n_mol, BOX)
    e.set_params(C.default_params())
    e.set_state(x, np.zeros_like(x))
    e.set_loss([RdfTerm(*args)])
    l, g = e.loss_grad()
    e.close()
    assert abs(l[0] - lo) <= 1e-11 * abs(lo)
    assert np.linalg.norm(g - go) <= 1e-11 * np.linalg.norm(go)
