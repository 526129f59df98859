"""The gas engine's rows and step kernels at the sizes where their split changes: a CTA's worth of
atoms and one more, several waves, no water or no gas, the smallest box; and positions outside the
box, whose FP32 distance tests decide nothing."""

import numpy as np
import pytest

from oracle import orc
from revsim import constants as C, systems
from revsim.gas import GasEngine

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    import build
    build.build()


# n_water, n_gas, box: one atom kind only; 1 to 41 atoms; a row longer than one pass of a warp's
# 128 tests; 2,832 atoms (more than one wave of FP64 pair warps); the smallest box, 2 x 1.2 nm
CASES = [(1, 0, 2.6), (0, 1, 2.6), (0, 40, 2.5), (1, 1, 2.4), (13, 1, 2.4), (120, 7, 2.4), (940, 6, 3.1)]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n_water,n_gas,box", CASES)
@pytest.mark.parametrize("outside", [False, True])
def test_forces_and_vjp_match_the_oracle(n_water, n_gas, box, precision, outside):
    s = orc.make_gas_system(n_water, n_gas, box, "lj")
    x = systems.gas_water_coords(n_water, n_gas, box, seed=n_water)
    p = np.array(C.gas_default_params("lj"))
    rng = np.random.default_rng(5)
    if outside:
        # shift the origin and leave the atoms there: up to 0.4 nm below zero
        x = x - np.array([0.4, 0.01, 0.2])
    w, ac = rng.normal(size=x.shape), rng.normal(size=x.shape)
    Fo, Go, dpo = orc.gas_forces_grads(s, p, x, w, ac, orc.gas_neighbor_pairs(s, x))
    e = GasEngine(n_water, n_gas, box, "lj", precision=precision)
    e.set_params(p)
    e.set_state(x, np.zeros_like(x))
    F = e.forces()
    F2, G, dp = e.force_vjp(w, ac)
    E = e.energy()
    e.close()
    # FP64: sums of at most 10^3 terms in another order.  Mixed: a displacement of two FP32
    # coordinates below 3.5 nm is off by at most 4e-7 nm, 3e-6 of the shortest distance, and the
    # steepest term grows with the 14th power of it (its Jacobian with the 15th).
    tol, tol_g = (1e-11, 1e-10) if precision == "fp64" else (1e-4, 2e-4)
    # forces and VJP come from kernels that form the pair terms alike
    assert np.abs(F - F2).max() <= tol * np.abs(Fo).max()
    assert np.abs(F - Fo).max() <= tol * np.abs(Fo).max()
    assert np.abs(G - Go).max() <= tol_g * np.abs(Go).max()
    assert np.abs(dp - dpo).max() <= tol_g * max(np.abs(dpo).max(), 1e-300)
    Eo = orc.gas_energy(s, p, x, orc.gas_neighbor_pairs(s, x))
    assert abs(E - Eo) <= 1e-10 * max(abs(Eo), 1.0)


def test_forward_and_reverse_over_several_waves():
    """2,832 atoms from unwrapped positions: the reverse pass returns to the start."""
    n_water, n_gas, box, n = 940, 6, 3.1, 24
    x = systems.gas_water_coords(n_water, n_gas, box, seed=1)
    v = systems.gas_water_velocities(n_water, n_gas, seed=2)
    seeds = systems.noise_seeds(n, seed=3)
    e = GasEngine(n_water, n_gas, box, "lj")
    e.set_params(np.array(C.gas_default_params("lj")))
    e.set_state(x - 0.3, v)
    e.forward(seeds, 1.0, n, 12, 0.0002, "diff")
    e.reverse(seeds, 1.0, n, 12, 12, 0.0002, "diff")
    xr, _ = e.get_state()
    e.close()
    d = xr - (x - 0.3)
    d -= box * np.round(d / box)
    assert np.abs(d).max() < 1e-9
