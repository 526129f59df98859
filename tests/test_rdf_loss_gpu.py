"""The RDF loss kernels at the sizes where their decomposition can go wrong: one atom, the
edges of the warps' first-atom groups (8) and of the staged tiles (256), odd and even rings of
equal sets, every pair of selections, slices of every stride, grids with and without the
normaliser polynomial, windows clipped at both ends of the grid.  Tolerance: the sums hold
positive terms whose Gaussians and normalisers are good to ~1e-14 relative, so 1e-11 of the
loss and of the gradient's norm leaves three digits of margin."""

import numpy as np
import pytest

from oracle import orc
from revsim import Engine, RdfTerm, constants as C, systems

pytestmark = pytest.mark.gpu

# x_min, step, width, exp_cutoff, n_grid, slice_start, slice_stride, n_target
GRIDS = {
    "fine": (0.1, 0.0005, 0.0005, 0.04, 4801, 124, 6, 281),
    "whole_fine": (0.2, 0.002, 0.0005, 0.0413, 700, 0, 1, 700),
    "coarse": (0.005, 0.005, 0.0005, 0.04, 200, 0, 1, 200),
    "no_polynomial": (0.02, 0.02, 0.0009, 0.06, 60, 1, 2, 29),
    "short_grid": (0.28, 0.001, 0.0004, 0.03, 40, 3, 5, 7),
    "one_point": (0.25, 0.0025, 0.0005, 0.04, 60, 30, 1, 1),
}


@pytest.fixture(scope="module", autouse=True)
def _built():
    import build
    build.build()


def _check(n_mol, box, sel, grid, norm):
    x = systems.water_coords(n_mol, box, seed=n_mol)
    g = GRIDS[grid]
    rng = np.random.default_rng(n_mol + norm)
    args = (*sel, *g[:7], rng.uniform(0.2, 1.5, g[7]), norm, 0.7)
    lo, go = orc.loss_grad(orc.make_system(n_mol, box), orc.Loss([orc.RdfTerm(*args)]), x)
    e = Engine(n_mol, box)
    e.set_params(C.default_params())
    e.set_state(x, np.zeros_like(x))
    e.set_loss([RdfTerm(*args)])
    l, gx = e.loss_grad()
    e.close()
    assert abs(l[0] - lo) <= 1e-11 * abs(lo)
    assert np.linalg.norm(gx - go) <= 1e-11 * np.linalg.norm(go) + 1e-300


@pytest.mark.parametrize("n_mol", [1, 2, 3, 7, 8, 9, 16, 17, 128, 129, 255, 256, 257, 264, 300])
@pytest.mark.parametrize("sel", [(0, 0), (0, 1), (1, 0), (1, 1)])
def test_ring_and_tile_edges(n_mol, sel):
    _check(n_mol, 2.5, sel, "fine", 2)


@pytest.mark.parametrize("grid", sorted(GRIDS))
@pytest.mark.parametrize("norm", [1, 2])
@pytest.mark.parametrize("sel", [(0, 0), (0, 1)])
def test_grids(grid, norm, sel):
    _check(150, 2.6, sel, grid, norm)


def test_ragged_replicas():
    """Replicas of unequal size in one launch: each one's loss and gradient as alone."""
    ns, boxes = [5, 300, 1, 131], [2.5, 2.6, 2.45, 2.55]
    xs = [systems.water_coords(n, b, seed=n) for n, b in zip(ns, boxes)]
    g = GRIDS["fine"]
    target = np.random.default_rng(0).uniform(0.5, 1.5, g[7])
    e = Engine(ns, boxes)
    e.set_params(C.default_params())
    e.set_state(np.concatenate(xs), np.zeros((3 * sum(ns), 3)))
    e.set_loss([RdfTerm(0, 0, *g[:7], target), RdfTerm(0, 1, *g[:7], target, 1, 0.3)])
    l, gx = e.loss_grad()
    e.close()
    o = 0
    for r, (n, b) in enumerate(zip(ns, boxes)):
        lo, go = orc.loss_grad(orc.make_system(n, b), orc.Loss(
            [orc.RdfTerm(0, 0, *g[:7], target), orc.RdfTerm(0, 1, *g[:7], target, 1, 0.3)]), xs[r])
        assert abs(l[r] - lo) <= 1e-11 * abs(lo)
        assert np.linalg.norm(gx[o:o + 3 * n] - go) <= 1e-11 * np.linalg.norm(go) + 1e-300
        o += 3 * n


# the value kernel's forms: 16 or 32 lanes a pair, or a lane a pair -- too many points a window (41),
# sums too many for 16 lanes' copies (300) and for 32 lanes' (600), factors too far apart
FORMS = {
    "16_of_300": (0.005, 0.005, 0.0005, 0.04, 300, 0, 1, 300),
    "32_of_600": (0.003, 0.003, 0.0005, 0.04, 600, 0, 1, 600),
    "steep": (0.005, 0.005, 0.00002, 0.04, 200, 0, 1, 200),
}


@pytest.mark.parametrize("form", sorted(FORMS))
def test_value_forms(form):
    GRIDS[form] = FORMS[form]
    _check(150, 2.6, (0, 0), form, 2)
    _check(150, 2.6, (0, 1), form, 1)


@pytest.mark.parametrize("step", [0.0625, 0.03125])
def test_window_with_both_ends_on_points(step):
    """A pair at a distance that is a grid point, with a cutoff of a whole number of steps (all exact
    in binary): 17 (33) points in the window of 16 (32) steps."""
    x = np.zeros((6, 3)) + 1.0
    x[3:, 0] += 1.0
    x[[1, 4], 1] += 0.0957
    x[[2, 5], 2] += 0.0957
    n = int(2.0 / step)
    args = (0, 0, step, step, 0.05, 0.5, n, 0, 1, np.linspace(0.0, 1.0, n), 2, 1.0)
    lo, go = orc.loss_grad(orc.make_system(2, 4.0), orc.Loss([orc.RdfTerm(*args)]), x)
    e = Engine(2, 4.0)
    e.set_params(C.default_params())
    e.set_state(x, np.zeros_like(x))
    e.set_loss([RdfTerm(*args)])
    l, gx = e.loss_grad()
    e.close()
    assert abs(l[0] - lo) <= 1e-11 * abs(lo)
    assert np.linalg.norm(gx - go) <= 1e-11 * np.linalg.norm(go) + 1e-300
