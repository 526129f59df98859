"""The one-CTA cell pass at the edges of its range: 8,192 molecules (its members fill their shared
memory) against the four-kernel pass at 8,193, and one molecule alone.  The same rows, so the same
forces up to the order of a row's sum (10^3 FP64 terms)."""

import numpy as np
import pytest

from revsim import Engine, constants as C, systems

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    import build
    build.build()


def _forces(ns, boxes, xs):
    e = Engine(ns, boxes, precision="fp64")
    e.set_params(C.default_params())
    e.set_state(np.concatenate(xs), np.zeros((3 * sum(ns), 3)))
    F = e.forces()
    e.close()
    return F


def test_one_cta_cells_match_four_kernels():
    n, box = 4096, 5.0
    x = systems.water_coords(n, box, seed=1)
    y = systems.water_coords(n, box, seed=2)
    z = systems.water_coords(1, 2.5, seed=3)
    one = _forces([n, n], [box, box], [x, y])
    four = _forces([n, 1, n], [box, 2.5, box], [x, z, y])
    alone = _forces([n], [box], [x])
    scale = np.abs(alone).max()
    assert np.abs(one[:3 * n] - alone).max() <= 1e-11 * scale
    assert np.abs(one[:3 * n] - four[:3 * n]).max() <= 1e-11 * scale
    assert np.abs(one[3 * n:] - four[3 * n + 3:]).max() <= 1e-11 * np.abs(one[3 * n:]).max()
    assert np.abs(_forces([1], [2.5], [z]) - four[3 * n:3 * n + 3]).max() <= 1e-11 * np.abs(four[3 * n:3 * n + 3]).max() + 1e-9
