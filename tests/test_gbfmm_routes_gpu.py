"""The two forms of the GBFMM moments and potential (products over the boxes of
one shape, one box at a time) give the same numbers on every grid, lmax and
kernel, alone and mixed in a batch, and a grid whose boxes all differ does not
pay for a product that it cannot share."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

QUAD = (2, 2)


def _axis(dage, cells, uneven, seed):
    h = np.full(cells, 0.21) if not uneven else np.random.default_rng(seed).uniform(0.15, 0.3, cells)
    return dage.Grid1D(-3 * float(h.sum()), cells, 7, 1, h)


def _grid(dage, cells, uneven=(False,) * 3):
    return dage.Grid3D(tuple(_axis(dage, c, u, i) for i, (c, u) in enumerate(zip(cells, uneven))))


def _op(dage, g, lmax, energy, level=2):
    k = dict(lmax=lmax, maxlevel=level, quad=dage.GaussQuad(*QUAD))
    return dage.GBFMMHelmholtz3D(g, energy, **k) if energy else dage.GBFMMCoulomb3D(g, **k)


def _both(dage, g, lmax, energy, level=2):
    """(moments, potential of fixed expansions) of a plan."""
    op = _op(dage, g, lmax, energy, level)
    rng = np.random.default_rng(3)
    rho = np.asfortranarray(rng.uniform(-0.5, 1.0, g.shape))
    q = op.multipole_moments(rho)
    L = rng.normal(size=q.shape)
    return q, op.evaluate_local_expansions(L, np.asfortranarray(rng.normal(size=g.shape)))


@pytest.mark.parametrize("energy", [0.0, -0.5])
@pytest.mark.parametrize("cells,uneven,level,lmax", [
    ((4, 4, 4), (0, 0, 0), 2, 0),       # one cell a box
    ((5, 7, 6), (0, 0, 0), 2, 3),       # eight shapes; 16 harmonics: two row tiles
    ((9, 8, 4), (0, 0, 0), 2, 14),      # 225 harmonics, 16 points a step
    ((8, 8, 8), (0, 0, 0), 2, 15),      # 64 alike
    ((8, 5, 4), (1, 0, 1), 2, 5),       # 36 harmonics: a row tile of four
    ((20, 21, 22), (0, 0, 0), 2, 12),   # tiles of 24, 8: both forms by the rule
    ((20, 20, 20), (0, 0, 1), 2, 8),    # four shapes of 16
    ((16, 16, 17), (0, 0, 0), 3, 6),    # 512 boxes: more than a tile of 64
])
def test_forms_agree(dage, monkeypatch, cells, uneven, level, lmax, energy):
    """A sum of n terms in another order is off by at most n eps of the sum of
    magnitudes; the harmonics' recurrences add lmax eps (16 times that here)."""
    g = _grid(dage, cells, uneven)
    out = {}
    for form in ("box", "product", None):
        if form:
            monkeypatch.setenv("DAGE_GBFMM_FORM", form)
        else:
            monkeypatch.delenv("DAGE_GBFMM_FORM", raising=False)
        out[form] = _both(dage, g, lmax, energy, level)
    for form in ("product", None):
        for a, b in zip(out["box"], out[form]):
            assert np.abs(a - b).max() <= 1e-12 * np.abs(a).max()


def test_forms_mixed_in_a_batch(dage):
    """Densities whose boxes share much, little and nothing, Coulomb and
    Helmholtz, against single operators."""
    grids = [_grid(dage, (20, 20, 20)), _grid(dage, (9, 8, 10), (True,) * 3), _grid(dage, (21, 18, 19)),
             _grid(dage, (20, 20, 20)), _grid(dage, (9, 8, 10), (True,) * 3), _grid(dage, (5, 6, 7))]
    energies = [0.0, -0.4, -0.7, -0.5, 0.0, 0.0]
    lmax = 10
    rng = np.random.default_rng(5)
    rhos = [np.asfortranarray(rng.uniform(0.0, 1.0, g.shape)) for g in grids]
    batch = dage.GBFMMBatch(grids, lmax=lmax, quad=dage.GaussQuad(*QUAD))
    for es in (np.zeros(6), energies, np.full(6, -0.6)):
        batch.set_energies(es)
        outs = [np.zeros(g.shape, order="F") for g in grids]
        E = batch.apply(rhos, outs, energy=True)
        for g, rho, V, e, en in zip(grids, rhos, outs, E, es):
            V1, e1 = _op(dage, g, lmax, en).apply(rho, energy=True)
            assert np.abs(V - V1).max() <= 1e-12 * np.abs(V1).max()
            assert abs(e - e1) <= 1e-12 * abs(e1)


def test_boxes_that_differ_go_one_at_a_time(dage):
    """Moments at 121^3, lmax 12: 64 boxes alike take 0.16 ms, all different
    0.42 ms one at a time (4.1 ms as 64 products of one)."""
    import torch

    times = []
    for uneven in (False, True):
        g = _grid(dage, (20, 20, 20), (uneven,) * 3)
        op = _op(dage, g, 12, 0.0)
        n = g.shape
        rho = torch.rand(n[2], n[1], n[0], dtype=torch.float64, device="cuda")
        best = 1e9
        for _ in range(10):
            t = time.perf_counter()
            op.multipole_moments(rho)
            best = min(best, time.perf_counter() - t)
        times.append(best)
    assert times[1] <= 8 * times[0]
