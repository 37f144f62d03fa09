"""Device memory of the operators' intermediates: what is taken, when, and
what happens where a group of t-points does not fit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MIB = 1 << 20


def _free():
    import torch

    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


class _Leave:
    """Holds the device's free memory but `nbytes`."""

    def __init__(self, nbytes):
        import torch

        torch.cuda.empty_cache()
        self.t = torch.empty(_free() - nbytes, dtype=torch.uint8, device="cuda")

    def __enter__(self):
        return self

    def __exit__(self, *exc):
        import torch

        del self.t
        torch.cuda.empty_cache()


def _density(shape, seed=1):
    import torch

    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.rand(shape[2], shape[1], shape[0], dtype=torch.float64, device="cuda", generator=g)


def _apply(op, rho, V):
    """V's values; the cubes are the caller's, so only the operator allocates."""
    op.apply(rho, V)
    return V.cpu().numpy()


def test_fp64_group_is_chosen_once(dage):
    """121^3: six t-points take 162 MiB of intermediates, one takes 27.  An
    operator that met 100 MiB of free memory stays with one t-point: the same
    bits and no allocation later, when there is room."""
    g = dage.Grid3D.cube(-12.0, 20, 0.2)
    quad = dage.GaussQuad(7, 6)
    rho, V = _density(g.shape), _density(g.shape)
    full = _apply(dage.Coulomb3D(g, quad=quad), rho, V)  # tunes; room for the group
    op = dage.Coulomb3D(g, quad=quad)  # the tuner's choice is known: nothing allocated yet
    with _Leave(100 * MIB):
        V1 = _apply(op, rho, V)
        free = _free()
        V2 = _apply(op, rho, V)
        assert _free() == free
    free = _free()
    V3 = _apply(op, rho, V)
    assert _free() == free
    np.testing.assert_array_equal(V2, V1)
    np.testing.assert_array_equal(V3, V1)
    assert np.abs(V1 - full).max() <= 1e-13 * np.abs(full).max()


def test_fp64_first_apply_after_tuning_allocates_nothing(dage):
    g = dage.Grid3D.cube(-7.8, 13, 0.2)
    rho, V = _density(g.shape), _density(g.shape)
    _apply(dage.Coulomb3D(g, quad=dage.GaussQuad(5, 5)), rho, V)  # kernels loaded
    op = dage.Coulomb3D(g, quad=dage.GaussQuad(11, 8))
    free = _free()
    V1 = _apply(op, rho, V)
    assert _free() == free
    np.testing.assert_array_equal(_apply(op, rho, V), V1)


def _near_bytes(cells):
    """(U, one slot of W) in bytes of the FP64 near field of one density on
    4 x 4 x 4 boxes: near and own points of the widest box of each axis."""
    def axis(n):
        nc = [n // 4 + (v < n % 4) for v in range(4)]
        near = [sum(nc[max(v - 1, 0):v + 2]) * 6 + 1 for v in range(4)]
        own = [6 * c + (v == 3) for v, c in enumerate(nc)]
        return list(zip(near, own))
    boxes = [(x, y, z) for x in axis(cells[0]) for y in axis(cells[1]) for z in axis(cells[2])]
    u = max(y[0] * z[0] * x[1] for x, y, z in boxes)
    w = max(z[0] * x[1] * y[1] for x, y, z in boxes)
    return 8 * 64 * u, 8 * 64 * w


@pytest.mark.parametrize("slots", [1, 3])
def test_batch_intermediates_stay_in_the_budget(dage, slots):
    """One density of 121^3 (W of 45 MB, up to five slots without a budget)
    under a budget of U and `slots` slots of W: the batch takes that and no more
    (beside the matrices: 3 axes, 4 positions, P t-points, and a few MB of
    tables), and its plan keeps no intermediates of its own."""
    cells, P = (20, 20, 20), 8
    u, w = _near_bytes(cells)
    g = dage.Grid3D.cube(-12.0, 20, 0.2)
    quad = dage.GaussQuad(4, 4)
    rho, V, V1 = _density(g.shape), _density(g.shape), _density(g.shape)
    single = dage.GBFMMCoulomb3D(g, lmax=2, quad=quad)
    single.apply(rho, V1)
    del single
    matrices = 8 * 3 * 4 * P * 31 * 91
    free = _free()
    batch = dage.GBFMMBatch([g], lmax=2, quad=quad, near_budget_bytes=u + slots * w)
    batch.apply([rho], [V])
    assert free - _free() <= u + slots * w + matrices + 24 * MIB
    assert float((V - V1).abs().max()) <= 1e-13 * float(V1.abs().max())
