"""Loss terms set again on one engine: buffers and uploads that a term keeps from the one before it must
not outlive a change of any of its values.  After each change the loss and its gradient, and a forward
and reverse pass (as plain launches and through CUDA graphs), are those of a fresh engine.  The sums use
FP64 atomics, whose order varies in the last bits: 1e-12 relative, as in the graph tests."""

from dataclasses import replace

import numpy as np
import pytest

from conftest import relaxed_gas
from revsim import Engine, RdfTerm, RevsimError, constants as C, systems
from revsim.gas import GasEngine

pytestmark = pytest.mark.gpu

N_STEPS = 12


@pytest.fixture(scope="module", autouse=True)
def _built():
    import build
    build.build()


def _terms():
    rng = np.random.default_rng(51)
    a = RdfTerm(0, 0, 0.005, 0.005, 0.0005, 0.04, 200, 0, 1, rng.uniform(0.2, 1.5, 200), 2, 1.0)
    b = RdfTerm(0, 1, 0.1, 0.0005, 0.0005, 0.04, 4801, 124, 6, rng.uniform(0.2, 1.5, 200), 1, 0.3)
    return a, b


def _changes():
    a, b = _terms()
    other = replace(a, target=a.target[::-1].copy())
    return [("first", [a, b]), ("same", [a, b]), ("targets", [other, b]), ("weight", [other, replace(b, weight=0.6)]),
            ("selection", [replace(other, sel2=1), b]), ("slice", [a, replace(b, slice_start=130)]), ("norm", [replace(a, norm=1), b]),
            ("width", [replace(a, width=0.0006), b]), ("swapped", [b, a]), ("back", [a, b]), ("fewer", [b]), ("more", [b, a, other]),
            ("none", []), ("again", [a, b])]


def _close(a, b):
    a, b = np.asarray(a), np.asarray(b)
    return np.all(np.abs(a - b) <= 1e-12 * max(np.abs(b).max(), 1e-300))


def _passes(e, x, v, seeds):
    e.set_state(x, v)
    l, g = e.loss_grad()
    lf = e.forward(seeds, 1.0, N_STEPS, N_STEPS, 0.001)
    lr, gp = e.reverse(seeds, 1.0, N_STEPS, N_STEPS, N_STEPS, 0.001)
    return l, g, lf, lr, gp


@pytest.mark.parametrize("graphs", [False, True])
def test_terms_set_again(small_water, graphs):
    n, box, x, v = small_water
    seeds = systems.noise_seeds(N_STEPS, seed=6)
    e = Engine(n, box)
    e.set_params(C.default_params())
    e.set_graph_mode(graphs)
    for name, terms in _changes():
        e.set_loss(terms)
        if not terms:
            continue
        got = _passes(e, x, v, seeds)
        e.rdf(0)   # (its histogram lies where the slice sums do)
        again = _passes(e, x, v, seeds)
        fresh = Engine(n, box)
        fresh.set_params(C.default_params())
        fresh.set_loss(terms)
        ref = _passes(fresh, x, v, seeds)
        fresh.close()
        assert all(_close(a, b) for a, b in zip(got, ref)), name
        assert all(_close(a, b) for a, b in zip(again, ref)), name
    e.close()


@pytest.mark.parametrize("graphs", [False, True])
def test_after_a_refused_term(small_water, graphs):
    n, box, x, v = small_water
    seeds = systems.noise_seeds(N_STEPS, seed=7)
    a, b = _terms()
    e = Engine(n, box)
    e.set_params(C.default_params())
    e.set_graph_mode(graphs)
    e.set_loss([a, b])
    ref = _passes(e, x, v, seeds)
    for bad in ([a, replace(b, norm=3)], [replace(b, width=-1.0), a], [replace(a, target=2 * a.target), replace(b, x_min=0.1002)]):
        with pytest.raises(RevsimError):
            e.set_loss(bad)
        e.set_loss([a, b])
        assert all(_close(p, q) for p, q in zip(_passes(e, x, v, seeds), ref))
    e.close()


def test_box_changes_the_normaliser(small_water):
    """The normaliser follows the box, also when the terms are the same as before."""
    n, box, x, v = small_water
    terms = list(_terms())
    e = Engine(n, box)
    e.set_params(C.default_params())
    for L in (box, 1.02 * box, box):
        e.set_box(L)
        e.set_loss(terms)
        e.set_state(x * (L / box), v)
        got = e.loss_grad()
        fresh = Engine(n, L)
        fresh.set_params(C.default_params())
        fresh.set_loss(terms)
        fresh.set_state(x * (L / box), v)
        ref = fresh.loss_grad()
        fresh.close()
        assert all(_close(a, b) for a, b in zip(got, ref))
    e.close()


def test_gas_terms_set_again():
    nw, ng, box = 130, 4, 2.6
    _, p, x, v = relaxed_gas(nw, ng, box, steps=20)
    seeds = systems.noise_seeds(N_STEPS, seed=8)

    def passes(e):
        e.set_state(x, v)
        f = e.forward(seeds, 1.0, N_STEPS, 4, 0.001, "diff_rdf")
        r = e.reverse(seeds, 1.0, N_STEPS, 4, 4, 0.001, "diff_rdf")
        return [np.asarray(q) for q in (*f, *r) if q is not None]

    e = GasEngine(nw, ng, box)
    e.set_params(p)
    for name, terms in _changes():
        if not terms:
            continue
        e.set_rdf(terms)
        got = passes(e)
        fresh = GasEngine(nw, ng, box)
        fresh.set_params(p)
        fresh.set_rdf(terms)
        ref = passes(fresh)
        fresh.close()
        assert len(got) == len(ref) and all(_close(a, b) for a, b in zip(got, ref)), name
    a, b = _terms()
    with pytest.raises(RevsimError):
        e.set_rdf([a, replace(b, norm=3)])
    e.set_rdf([a, b])
    fresh = GasEngine(nw, ng, box)
    fresh.set_params(p)
    fresh.set_rdf([a, b])
    assert all(_close(q, r) for q, r in zip(passes(e), passes(fresh)))
    fresh.close()
    e.close()
