"""The fused step kernels where their decomposition into pair and update warps can go wrong:
CTAs of one molecule, at and just past an update warp's ten, partial last CTAs, every lane
count and loop form in both directions; and replicas on both sides of the box side above which
one periodic image serves a molecule pair, in one launch.  Forces, VJP and the dtheta
contraction against the FP64 oracle at the tolerances of the other parity tests (1e-10 FP64,
1e-5 / 1e-4 mixed); the loop forms of one lane count give the same bits."""

import numpy as np
import pytest

from conftest import relaxed_water
from oracle import orc
from revsim import Engine, constants as C

pytestmark = pytest.mark.gpu

N_MOL, BOX = 151, 2.6


@pytest.fixture(scope="module", autouse=True)
def _built():
    import build
    build.build()


def _relaxed(n_mol, box):
    out = relaxed_water(n_mol, box)
    return np.asarray(out[0] if isinstance(out, tuple) else out)


def _reference(x, n_mol, box, inter, w, ac):
    s = orc.make_system(n_mol, box, inter)
    p = np.array(C.default_params(inter))
    pairs = orc.neighbor_pairs(s, x)
    F, G, _ = orc.forces_grads(s, p, x, pairs, w, jac=False)
    return F, G, orc.contract(s, p, x, pairs, ac)


def _close(a, b, tol):
    return np.linalg.norm(a - b) <= tol * np.linalg.norm(b)


@pytest.mark.parametrize("prec,tol", [("fp64", (1e-10, 1e-10)), ("mixed", (1e-5, 1e-4))])
@pytest.mark.parametrize("inter", ["lj", "buff"])
def test_cta_edges(prec, tol, inter):
    x = _relaxed(N_MOL, BOX)
    rng = np.random.default_rng(3)
    w, ac = rng.normal(size=x.shape), rng.normal(size=x.shape)
    Fo, Go, to = _reference(x, N_MOL, BOX, inter, w, ac)
    e = Engine(N_MOL, BOX, inter_type=inter, precision=prec)
    e.set_params(C.default_params(inter))
    e.set_state(x, np.zeros_like(x))
    for G, mols in ((32, (1, 10, 11)), (16, (2, 10, 12)), (8, (4, 12, 20))):
        bits = set()
        for m in mols:
            for U in (1, 2, 3):
                if U == 3 and G * m > 256:
                    continue
                if prec == "mixed" and U == 2 and G * m > 256:
                    continue
                e.set_launch_shape(G, m, U)
                F, Gv, th = e.force_vjp(w, ac)
                Ff = e.forces()
                assert _close(F, Fo, tol[0]) and _close(Gv, Go, tol[1]) and _close(th[0], to, tol[1])
                assert np.array_equal(F, Ff)
                bits.add((F.tobytes(), Gv.tobytes(), th.tobytes()))
        assert len(bits) == 1
    e.close()


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_boxes_on_both_sides_of_the_one_image_rule(prec):
    """Small (per-slot images) and large (one image per molecule pair) boxes in one launch give
    the bits each gives alone."""
    sizes = [(150, 2.5), (151, 2.64), (140, 2.45)]
    xs = [_relaxed(n, b) for n, b in sizes]
    e = Engine([n for n, _ in sizes], [b for _, b in sizes], precision=prec)
    e.set_params(C.default_params())
    x = np.concatenate(xs)
    e.set_state(x, np.zeros_like(x))
    e.set_launch_shape(16, 8, 1)
    F = e.forces()
    e.close()
    o = 0
    for (n, b), xr in zip(sizes, xs):
        s = orc.make_system(n, b)
        Fo = orc.forces(s, np.array(C.default_params()), xr, orc.neighbor_pairs(s, xr))
        e = Engine(n, b, precision=prec)
        e.set_params(C.default_params())
        e.set_state(xr, np.zeros_like(xr))
        e.set_launch_shape(16, 8, 1)
        Fa = e.forces()
        e.close()
        assert np.array_equal(F[o:o + 3 * n], Fa)
        assert _close(Fa, Fo, 1e-10 if prec == "fp64" else 1e-5)
        o += 3 * n
