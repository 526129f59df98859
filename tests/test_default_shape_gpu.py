"""The shape the step kernels run with when none is set: on both sides of the molecule counts where it
changes its lanes and loop form (forces, VJP and dtheta of every replica against the FP64 oracle, at the
tolerances of the other parity tests), and that reading, setting back, setting one kernel alone or
visiting the half-shell mode leaves it as it was."""

import numpy as np
import pytest

from conftest import relaxed_water
from oracle import orc
from revsim import Engine, RevsimError, constants as C, systems

pytestmark = pytest.mark.gpu

N_MOL, BOX = 150, 2.6


@pytest.fixture(scope="module", autouse=True)
def _built():
    import build
    build.build()


@pytest.fixture(scope="module")
def box():
    x, _ = relaxed_water(N_MOL, BOX)
    rng = np.random.default_rng(41)
    w, ac = rng.normal(size=x.shape), rng.normal(size=x.shape)
    s = orc.make_system(N_MOL, BOX)
    p = np.array(C.default_params())
    pairs = orc.neighbor_pairs(s, x)
    F, G, _ = orc.forces_grads(s, p, x, pairs, w, jac=False)
    return x, w, ac, F, G, orc.contract(s, p, x, pairs, ac)


def _engine(n, b, prec):
    e = Engine(n, b, precision=prec)
    e.set_params(C.default_params())
    return e


def _close(a, b, tol):
    return np.linalg.norm(a - b) <= tol * np.linalg.norm(b)


@pytest.mark.parametrize("prec,reps,lanes", [("mixed", 1, 32), ("mixed", 8, 32), ("mixed", 9, 32), ("mixed", 16, 32),
                                             ("mixed", 19, 16), ("mixed", 40, 16), ("fp64", 1, 32), ("fp64", 26, 32),
                                             ("fp64", 27, 16)])
def test_default_shapes_against_the_oracle(box, prec, reps, lanes):
    x, w, ac, Fo, Go, to = box
    tol = (1e-10, 1e-10) if prec == "fp64" else (1e-5, 1e-4)
    e = _engine([N_MOL] * reps, [BOX] * reps, prec)
    e.set_state(np.tile(x, (reps, 1)), np.zeros((reps * len(x), 3)))
    shapes = e.launch_shape(0), e.launch_shape(1)
    F, G, th = e.force_vjp(np.tile(w, (reps, 1)), np.tile(ac, (reps, 1)))
    Ff = e.forces()
    for which in (0, 1):
        e.set_launch_shape(*shapes[which], which=which)
    assert (e.launch_shape(0), e.launch_shape(1)) == shapes
    assert np.array_equal(e.forces(), Ff) and np.array_equal(F, Ff)
    e.close()
    assert shapes[0][0] == shapes[1][0] == lanes
    for r in range(reps):
        o = slice(r * len(x), (r + 1) * len(x))
        assert _close(F[o], Fo, tol[0]) and _close(G[o], Go, tol[1]) and _close(th[r], to, tol[1])


# molecules per CTA of the reverse kernel: those of one wave over 148 SMs, else its fill
@pytest.mark.parametrize("prec,n,b,mols", [("mixed", 400, 2.48, 3), ("mixed", 2600, 4.3, 18), ("mixed", 3000, 4.5, 22),
                                           ("fp64", 400, 2.48, 3), ("fp64", 3000, 4.5, 7), ("fp64", 4500, 5.2, 10)])
def test_setting_back_changes_nothing(prec, n, b, mols):
    e = _engine(n, b, prec)
    rev, fwd = e.launch_shape(0), e.launch_shape(1)
    assert rev[1] == mols
    e.set_launch_shape(*rev, which=0)
    e.set_launch_shape(*fwd, which=1)
    assert (e.launch_shape(0), e.launch_shape(1)) == (rev, fwd)
    e.close()
    # one kernel's loop form alone: the other kernel's shape stays
    e = _engine(n, b, prec)
    e.set_launch_shape(0, 0, 3, which=0)
    assert e.launch_shape(0)[0] == rev[0] and e.launch_shape(0)[2] == 3 and e.launch_shape(1) == fwd
    e.close()
    # lanes alone, back and forth
    e = _engine(n, b, prec)
    for lanes in (8, 16, 32, rev[0]):
        e.set_launch_shape(lanes, 0, 0)
        assert e.launch_shape(0)[0] == e.launch_shape(1)[0] == lanes
    assert (e.launch_shape(0), e.launch_shape(1)) == (rev, fwd)
    with pytest.raises(RevsimError):
        e.set_launch_shape(32, 33, 1)
    e.close()


@pytest.mark.parametrize("ns,rev,fwd", [([394] * 3, (32, 2, 2), (32, 2, 1)), ([181] * 16, (16, 4, 1), (16, 4, 1)),
                                        ([150] * 17, (32, 9, 1), (32, 9, 1)), ([700, 1100], (32, 13, 1), (32, 13, 1))])
def test_one_wave_counts_the_replicas(ns, rev, fwd):
    """No CTA straddles two replicas: 3 boxes of 394 are 150 CTAs of eight molecules, one too many an SM."""
    e = Engine(ns, [2.6 if n < 500 else 3.3 for n in ns], precision="mixed")
    assert (e.launch_shape(0), e.launch_shape(1)) == (rev, fwd)
    e.close()


@pytest.mark.parametrize("n,b", [(400, 2.48), (2600, 4.3), (3000, 4.5)])
def test_half_shell_and_back(n, b):
    e = _engine(n, b, "mixed")
    shapes = e.launch_shape(0), e.launch_shape(1)
    x = systems.water_coords(n, b, seed=1)
    e.set_state(x, np.zeros_like(x))
    F = e.forces()
    e.set_pair_mode("half_shell")
    assert e.launch_shape(0) == e.launch_shape(1) == (32, 8, 1)
    assert _close(e.forces(), F, 1e-5)
    e.set_pair_mode("both_sides")
    assert (e.launch_shape(0), e.launch_shape(1)) == shapes
    assert np.array_equal(e.forces(), F)
    # a shape that was set is kept
    e.set_launch_shape(16, 12, 1)
    e.set_pair_mode("half_shell")
    e.set_pair_mode("both_sides")
    assert e.launch_shape(0) == e.launch_shape(1) == (16, 12, 1)
    e.close()
