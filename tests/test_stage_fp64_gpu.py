"""The FP64 stages at the sizes where their tiling can go wrong: fewer points
than a tile, remainders of the 128-row, 32-column and 4-K steps, axes of
different lengths, output grids of their own, groups of t-points that do not
divide the t-points, and accumulation over groups."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


def _axes(dage, cells, step, shift=0.0):
    return dage.Grid3D(tuple(dage.Grid1D.equidistant(-3 * c * step + shift, c, step) for c in cells))


@pytest.mark.parametrize("cells,out_cells,nlin,nlog", [
    ((1, 1, 1), None, 1, 0),        # 7 points: one partial tile, one t-point
    ((5, 1, 9), None, 10, 8),       # 31, 7, 55: less and more than 32 columns
    ((2, 11, 4), None, 33, 32),     # 13, 67, 25; 65 t-points: more than one group
    ((21, 3, 6), None, 7, 6),       # 127 rows and columns: one short of a tile
    ((8, 8, 8), (3, 5, 2), 9, 9),   # 49 -> 19, 31, 13 points
    ((3, 4, 5), (22, 6, 7), 9, 9),  # 19, 25, 31 -> 133, 37, 43
    ((30, 24, 20), None, 6, 13),    # 181, 145, 121: several tiles, groups and bands
])
@pytest.mark.parametrize("accumulate", [False, True])
def test_stages_against_matrices(dage, cells, out_cells, nlin, nlog, accumulate):
    """V against the plain contraction with the operator's own matrices.
    Every sum has at most n_in terms per axis and P over the t-points, and
    skipped entries are below 2^-64 of their row, so an element is off by at
    most (sum of the terms' counts) eps times the same sum of magnitudes."""
    step = 0.2
    g = _axes(dage, cells, step)
    go = g if out_cells is None else _axes(dage, out_cells, 0.17, 0.05)
    op = dage.Coulomb3D(g, go, quad=dage.GaussQuad(nlin, nlog))
    rng = np.random.default_rng(sum(cells))
    rho = np.asfortranarray(rng.normal(size=g.shape))
    V0 = np.asfortranarray(rng.normal(size=go.shape))
    V = V0.copy(order="F")
    op.apply(rho, out=V, coda=False, accumulate=accumulate)
    w = op.weights
    T = [op.matrix(d) for d in range(3)]
    want = np.zeros(go.shape)
    mag = np.zeros(go.shape)
    for p in range(len(w)):
        A = [t[:, :, p] for t in T]
        want += w[p] * np.einsum("ia,jb,kc,abc->ijk", *A, rho, optimize=True)
        mag += abs(w[p]) * np.einsum("ia,jb,kc,abc->ijk", *(abs(a) for a in A), abs(rho), optimize=True)
    if accumulate:
        want += V0
        mag += abs(V0)
    bound = 2 * (sum(g.shape) + len(w) + 8) * EPS * mag
    assert np.all(abs(V - want) <= bound)


def test_tile_width_changes_no_bit(dage, tmp_path):
    """A cached tile choice (any of the three widths per stage) gives the same
    bits: a warp sums its 32 columns over the same K in the same order."""
    import re

    g = _axes(dage, (9, 12, 8), 0.2)
    quad = dage.GaussQuad(8, 7)
    rng = np.random.default_rng(3)
    rho = np.asfortranarray(rng.normal(size=g.shape))
    cache = tmp_path / "tiles"
    dage.set_tune_cache(str(cache))
    try:
        V = dage.Coulomb3D(g, quad=quad).apply(rho)
        key = re.sub(r"( \d+){3}$", "", cache.read_text().strip().splitlines()[-1])
        for tiles in ((32, 64, 128), (128, 32, 64), (64, 128, 32)):
            dage.set_tune_cache(None)
            cache.write_text(f"{key} {tiles[0]} {tiles[1]} {tiles[2]}\n")
            dage.set_tune_cache(str(cache))
            op = dage.Coulomb3D(g, quad=quad)
            assert op.tiles == tiles
            np.testing.assert_array_equal(op.apply(rho), V)
    finally:
        dage.set_tune_cache(None)
