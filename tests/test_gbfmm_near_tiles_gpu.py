"""The fp16x3 near field at the sizes where its tiles and run tables can go
wrong: boxes of one cell (7 points), uneven splits, axes of different
lengths, both tile widths, own points just above a tile, odd row counts."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile", ["64", "128"])
@pytest.mark.parametrize("cells", [(4, 4, 4), (5, 9, 7), (8, 4, 11), (43, 6, 5), (5, 5, 44)])
def test_near_field_against_fp64(dage, monkeypatch, cells, tile):
    """Two FP16 parts hold 22 bits; three stages with FP32 partial sums stay
    within a few units of that, the far field being the same in both."""
    monkeypatch.setenv("DAGE_NEAR16_TILE", tile)
    step = 0.25
    g = dage.Grid3D(tuple(dage.Grid1D.equidistant(-3 * c * step, c, step) for c in cells))
    quad = dage.GaussQuad(6, 7)
    rng = np.random.default_rng(sum(cells))
    rho = np.asfortranarray(rng.uniform(0.0, 1.0, g.shape))
    V = dage.GBFMMCoulomb3D(g, lmax=3, quad=quad, precision="fp16x3").apply(rho)
    V64 = dage.GBFMMCoulomb3D(g, lmax=3, quad=quad).apply(rho)
    assert np.abs(V - V64).max() <= 1e-6 * np.abs(V64).max()


def test_batch_of_equal_and_uneven_grids(dage):
    """Several densities of one plan share a launch: each equals its own apply."""
    step = 0.25
    grids = [dage.Grid3D.cube(-3 * c * step, c, step) for c in (5, 8, 5, 5, 8)]
    quad = dage.GaussQuad(6, 7)
    rng = np.random.default_rng(5)
    rhos = [np.asfortranarray(rng.uniform(0.0, 10.0 ** k, g.shape)) for k, g in enumerate(grids)]
    outs = [np.zeros(g.shape, order="F") for g in grids]
    dage.GBFMMBatch(grids, lmax=3, quad=quad, precision="fp16x3").apply(rhos, outs)
    for g, r, v in zip(grids, rhos, outs):
        want = dage.GBFMMCoulomb3D(g, lmax=3, quad=quad, precision="fp16x3").apply(r)
        # the same kernels; only the far field's slab sums may differ
        assert np.abs(v - want).max() <= 1e-13 * np.abs(want).max()
