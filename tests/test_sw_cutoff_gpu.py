"""The diamond engine's terms for pairs just inside the cutoff r = a sigma, where 1/t, t = r / sigma - a,
grows without bound and only e^{1/t} = 0 keeps the terms finite: forces, VJP, the seven parameters'
contraction and the stress loss's gradients against the FP64 oracle, at the tolerances of the other
parity tests (1e-10 / 1e-9 FP64, 1e-5 / 1e-4 mixed)."""

import numpy as np
import pytest

from oracle import orc
from revsim import SwEngine, diamond as D

pytestmark = pytest.mark.gpu

T = (-1e-3, -1e-6, -1e-9, -4e-10, -1e-10, -1e-11, -1e-12, -1e-13)


@pytest.fixture(scope="module", autouse=True)
def _built():
    import build
    build.build()


def _nrel(a, b):
    return np.linalg.norm(np.asarray(a) - np.asarray(b)) / np.linalg.norm(np.asarray(b))


def _crystal():
    """A crystal with one pair of second neighbours at each t of T."""
    x, box = D.diamond_coords(4, noise=0.004, seed=31)
    p = np.array(D.default_params())
    a, sig = p[2], p[5]
    used = set()
    for t in T:
        for i in range(len(x)):
            d = x - x[i]
            r = np.linalg.norm(d, axis=1)
            j = int(np.argmin(np.abs(r - a * sig)))
            new = x[i] + d[j] * (sig * (a + t) / r[j])
            near = set(np.flatnonzero(r < 2.5 * a * sig))   # no other pair's atoms about
            if near & used or new.min() < 0.0 or new.max() > box:
                continue
            rn = np.linalg.norm(new - x[i]) / sig
            if not (rn < a and abs(rn - a - t) < 0.1 * abs(t)):
                continue
            x[j] = new
            used |= {i, j}
            break
        else:
            raise AssertionError("no pair for t = %g" % t)
    return x, box, p


@pytest.mark.parametrize("prec,ftol,gtol", [("fp64", 1e-10, 1e-9), ("mixed", 1e-5, 1e-4)])
def test_pairs_just_inside_the_cutoff(prec, ftol, gtol):
    x, box, p = _crystal()
    rng = np.random.default_rng(32)
    w, ac, v = (rng.normal(size=x.shape) for _ in range(3))
    target = rng.normal(scale=50.0, size=9)
    s = orc.make_sw_system(len(x), box)
    Fo, Go, J = orc.sw_forces_grads(s, p, x, w)
    dpo = (ac.reshape(-1)[:, None] * J).sum(axis=0)
    lo, gxo, gvo, gpo = orc.sw_loss_grad(s, p, orc.make_sw_loss(D.STRESS_WEIGHT, target), x, v)
    with SwEngine(len(x), box, precision=prec) as e:
        e.set_params(p)
        e.set_state(x, v)
        F, G, dp = e.force_vjp(w, ac)
        e.set_loss(D.STRESS_WEIGHT, target)
        l, gx, gv, gp = e.loss_grad()
    assert _nrel(F, Fo) <= ftol and _nrel(G, Go) <= gtol
    assert np.abs(dp[0] - dpo).max() <= gtol * np.abs(dpo).max()
    assert abs(l[0] - lo) <= gtol * abs(lo)
    assert _nrel(gx, gxo) <= gtol and _nrel(gv, gvo) <= gtol
    assert np.abs(gp[0] - gpo).max() <= gtol * np.abs(gpo).max()
