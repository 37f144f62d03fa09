"""The split-precision stages at the sizes where their tiles, K blocks, column
windows and run lists can go wrong: fewer rows, columns or K than one block,
remainders of the 8-row atoms, 32-K blocks, 32-column groups and 128-tiles,
axes of different lengths, output grids of their own, more than 32 K blocks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _axes(dage, cells, step, shift=0.0):
    return dage.Grid3D(tuple(dage.Grid1D.equidistant(-3 * c * step + shift, c, step) for c in cells))


# two FP16 parts hold 22 bits, two BF16 parts 16, three 24; a result sums
# three stages of products with FP32 partial sums, so a few units of that
BARS = {"fp16x3": 1e-6, "bf16x6": 1e-6, "bf16x3": 1e-5}


@pytest.mark.parametrize("precision", sorted(BARS))
@pytest.mark.parametrize("cells,out_cells", [
    ((1, 1, 1), None),           # 7: one partial tile in every direction
    ((5, 1, 11), None),          # 31, 7, 67
    ((21, 22, 3), None),         # 127, 133, 19: around one tile
    ((10, 16, 21), (3, 22, 5)),  # 61, 97, 127 -> 19, 133, 31
    ((2, 3, 172), (4, 2, 171)),  # 1033 points: more than 32 K blocks, 9 n-tiles
])
def test_against_fp64_operator(dage, precision, cells, out_cells):
    step = 0.25
    g = _axes(dage, cells, step)
    go = g if out_cells is None else _axes(dage, out_cells, 0.22, 0.07)
    quad = dage.GaussQuad(7, 6)
    rng = np.random.default_rng(sum(cells))
    rho = np.asfortranarray(rng.uniform(0.0, 1.0, g.shape))
    V = dage.Operator3D(g, go, quad, precision=precision).apply(rho, coda=False)
    V64 = dage.Operator3D(g, go, quad).apply(rho, coda=False)
    assert np.abs(V - V64).max() <= BARS[precision] * np.abs(V64).max()


@pytest.mark.parametrize("precision,ncell,nlin,nlog", [
    ("fp16x3", 30, 7, 6),   # 181^3: two t-points per intermediate launch, 13 in all: 2 2 2 2 | 2 2 1
    ("bf16x3", 27, 7, 6),   # 163^3: three: 3 3 2 | 3 2
    ("bf16x6", 24, 8, 3),   # 145^3, three parts: three: 3 3 2 | 3
])
def test_groups_of_several_intermediate_launches(dage, precision, ncell, nlin, nlog):
    """More than one launch of the first two stages per group of the last one:
    slots of the second intermediate written at their offset in the group, slots
    of the first one reused, a last launch of fewer t-points.  (One t-point per
    launch, 481^3, and the whole group in one, the cubes above, have none of
    these.)  A t-point in the wrong slot is an error of the t-point's share."""
    import torch

    g = dage.Grid3D.cube(-0.6 * ncell, ncell, 0.2)
    quad = dage.GaussQuad(nlin, nlog)
    n = g.shape[0]
    gen = torch.Generator(device="cuda").manual_seed(ncell)
    rho = torch.rand(n, n, n, dtype=torch.float64, device="cuda", generator=gen)
    V, V64 = torch.empty_like(rho), torch.empty_like(rho)
    op = dage.Coulomb3D(g, quad=quad, precision=precision)
    op.apply(rho, V)
    dage.Coulomb3D(g, quad=quad).apply(rho, V64)
    assert float((V - V64).abs().max()) <= BARS[precision] * float(V64.abs().max())
    again = torch.empty_like(V)
    op.apply(rho, again)
    assert torch.equal(V, again)
