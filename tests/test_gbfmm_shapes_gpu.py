"""Moments and local-expansion evaluation where the boxes' shapes differ: even
splits (one shape), uneven splits (up to eight), cells of different sizes
(every box its own), over the lmax range and its tile remainders."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _grids(dage, oracle, cells, uneven_cells):
    rng = np.random.default_rng(sum(cells))
    axes, oaxes = [], []
    for c in cells:
        h = np.full(c, 0.21) if not uneven_cells else rng.uniform(0.15, 0.3, c)
        qmin = -3 * float(h.sum())
        axes.append(dage.Grid1D(qmin, c, 7, 1, h))
        oaxes.append(oracle.Grid1D(qmin, c, 7, 1, h))
    return dage.Grid3D(tuple(axes)), oracle.Grid3D(tuple(oaxes))


@pytest.mark.parametrize("cells,uneven_cells,lmax", [
    ((4, 4, 4), False, 0), ((8, 8, 8), False, 15), ((8, 4, 12), False, 7),
    ((5, 7, 6), False, 13), ((9, 8, 4), False, 14), ((8, 5, 4), True, 12)])
def test_moments_and_evaluation(dage, oracle, cells, uneven_cells, lmax):
    """Against the oracle's point sums; both sum the same terms in 64 bits, in
    another order, with harmonics of coordinates equal to their rounding."""
    g, go = _grids(dage, oracle, cells, uneven_cells)
    rng = np.random.default_rng(7)
    rho = np.asfortranarray(rng.uniform(-0.5, 1.0, g.shape))
    op = dage.GBFMMCoulomb3D(g, lmax=lmax, quad=dage.GaussQuad(2, 2))
    plan = oracle.GBFMMPlan(go, 2)
    Q = op.multipole_moments(rho)
    N = (lmax + 1) ** 2
    L = rng.normal(size=(N, plan.nbox))
    V0 = np.asfortranarray(rng.normal(size=g.shape))
    V = op.evaluate_local_expansions(L, V0.copy(order="F"))
    want = V0.copy(order="F")
    for b in range(1, plan.nbox + 1):
        (x0, x1), (y0, y1), (z0, z1) = plan.points(b)
        subs = [oracle.subgrid(a, c0, c1) for a, (c0, c1) in zip(go.axes, plan.cells(b))]
        q = oracle.box_multipoles(lmax, subs[0].points, subs[0].weights(), subs[1].points,
                                  subs[1].weights(), subs[2].points, subs[2].weights(),
                                  rho[x0:x1, y0:y1, z0:z1], plan.center(b))
        assert np.abs(Q[:, b - 1] - q).max() <= 1e-12 * np.abs(q).max()
        own = plan.owned(b)
        pts = [go.axes[d].points[own[d][0]:own[d][1]] for d in range(3)]
        part = np.zeros(tuple(len(p) for p in pts), order="F")
        oracle.l2p(lmax, L[:, b - 1], plan.center(b), *pts, part)
        want[tuple(slice(o0, o1) for o0, o1 in own)] += part
    assert np.abs(V - want).max() <= 1e-12 * np.abs(want).max()
