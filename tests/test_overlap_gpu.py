"""Overlapping atoms of two molecules: the energy is infinite, with the sign of the term that diverges,
not NaN (r = 0 is a plain value of every form but those that divide by r)."""

import numpy as np
import pytest

from revsim import Engine, RevsimError, constants as C, mlp

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    import build
    build.build()


def _pair(a, b):
    """Two waters, the second the first reflected so that its atom b lies on the first's atom a."""
    m = np.array([[1.0, 1.0, 1.0], [1.0957, 1.0, 1.0], [0.976, 1.0927, 1.0]])
    n = -m
    n += m[a] - n[b]
    n[b] = m[a]
    return np.concatenate([m, n])


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("a,b,sign,inter", [(1, 1, 1, "lj"), (2, 1, 1, "buck"), (0, 1, -1, "lj"), (1, 0, -1, "buff"),
                                            (0, 0, 1, "dexp")])
def test_energy_of_overlapping_atoms(prec, a, b, sign, inter):
    e = Engine(2, 2.6, inter_type=inter, precision=prec)
    e.set_params(C.default_params(inter))
    e.set_state(_pair(a, b), np.zeros((6, 3)))
    E, _ = e.energy_grad()
    e.close()
    assert E[0] == sign * np.inf


def test_energy_of_overlapping_atoms_with_the_learned_term():
    """The learned term's share is finite at r = 0: its weights' derivatives too."""
    e = Engine(2, 2.6, precision="fp64", mlp=True)
    e.set_params(np.concatenate([C.default_params(), mlp.init_params(3)]))
    e.set_state(_pair(1, 1), np.zeros((6, 3)))
    E, g = e.energy_grad()
    e.close()
    assert E[0] == np.inf
    assert np.isfinite(g[0, len(C.default_params()):]).all()


@pytest.mark.parametrize("a,b", [(0, 0), (0, 1), (1, 1)])
@pytest.mark.parametrize("with_mlp", [False, True])
def test_forces_of_overlapping_atoms_are_an_error(a, b, with_mlp):
    """An error of the call, also where the NaN distance would be the learned term's table index."""
    e = Engine(2, 2.6, precision="fp64", mlp=with_mlp)
    p = C.default_params()
    e.set_params(np.concatenate([p, mlp.init_params(3)]) if with_mlp else p)
    x = _pair(a, b)
    e.set_state(x, np.zeros((6, 3)))
    with pytest.raises(RevsimError):
        e.forces()
    with pytest.raises(RevsimError):
        e.force_vjp(np.ones_like(x), np.ones_like(x))
    e.set_state(x + np.arange(6)[:, None] // 3 * 0.5, np.zeros((6, 3)))
    assert np.isfinite(e.forces()).all()
    e.close()
