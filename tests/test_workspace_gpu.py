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


def _u16_slot(ncell, nbox_axis=4):
    """Bytes of one U slot of the fp16x3 near field (two FP16 planes of
    [x own of every box][z near, padded to 32][y near, padded to 8])."""
    nc = [ncell // nbox_axis + (v < ncell % nbox_axis) for v in range(nbox_axis)]
    near = max(sum(nc[max(v - 1, 0):v + 2]) for v in range(nbox_axis)) * 6 + 1
    return 4 * (ncell * 6 + 1) * nbox_axis**2 * (-(-near // 32) * 32) * (-(-near // 8) * 8)


def _near16_bytes(ncell, P):
    """The set's other intermediates (split input, W) and the plan's matrices."""
    n = ncell * 6 + 1
    nc = [ncell // 4 + (v < ncell % 4) for v in range(4)]
    own = max(6 * c + (v == 3) for v, c in enumerate(nc))
    near = max(sum(nc[max(v - 1, 0):v + 2]) for v in range(4)) * 6 + 1
    x = 4 * n * n * (-(-n // 8) * 8)
    w = 4 * min(P, 4) * n * 16 * (-(-own // 32) * 32) * (-(-near // 8) * 8)
    return x + w + 3 * (8 + 4 + 2) * P * n * (near + 8)


def test_near_field_takes_one_u_slot_where_t_points_do_not_share_tiles(dage):
    """217^3 owns 54 or 55 points a box: one t-point per stage-x tile, one slot
    of U (a second one would be 448 MB)."""
    ncell, quad = 36, dage.GaussQuad(2, 2)
    g = dage.Grid3D.cube(-21.6, ncell, 0.2)
    rho, V = _density(g.shape), _density(g.shape)
    dage.GBFMMCoulomb3D(g, lmax=2, quad=quad, precision="fp16x3").apply(rho, V)  # tunes
    free = _free()
    op = dage.GBFMMCoulomb3D(g, lmax=2, quad=quad, precision="fp16x3")
    op.apply(rho, V)
    used = free - _free()
    slot = _u16_slot(ncell)
    assert slot > 400 * MIB
    assert used <= slot + _near16_bytes(ncell, 4) + 64 * MIB


def test_near_field_with_room_for_one_u_slot(dage, monkeypatch):
    """181^3 owns 45 or 46 points a box: two t-points share a stage-x tile
    where there is room for two slots of U; where there is not, one is taken,
    with the same bits.  Single operator and batch."""
    monkeypatch.setenv("DAGE_NEAR16_TILE", "64")
    ncell, quad = 30, dage.GaussQuad(3, 2)
    g = dage.Grid3D.cube(-18.0, ncell, 0.2)
    rho, V = _density(g.shape), _density(g.shape)
    slot = _u16_slot(ncell)

    def single():
        op = dage.GBFMMCoulomb3D(g, lmax=2, quad=quad, precision="fp16x3")
        op.apply(rho, V)
        return op

    def batch():
        b = dage.GBFMMBatch([g], lmax=2, quad=quad, precision="fp16x3")
        b.apply([rho], [V])
        return b

    for make in (single, batch):
        make()  # kernels loaded
        free = _free()
        keep = make()
        need = free - _free()
        want = V.cpu().numpy()
        del keep
        V.zero_()
        with _Leave(need - slot // 2):
            keep = make()
            del keep
        np.testing.assert_array_equal(V.cpu().numpy(), want)


def test_split_precision_group_leaves_the_rest_its_room(dage):
    """121^3, fp16x3: six slots of the first intermediate take 35 MB more than
    one; an operator with 20 MB less than that form needs takes one slot, with
    the same bits."""
    g = dage.Grid3D.cube(-12.0, 20, 0.2)
    quad = dage.GaussQuad(7, 6)
    rho, V = _density(g.shape), _density(g.shape)

    def make():
        op = dage.Coulomb3D(g, quad=quad, precision="fp16x3")
        op.apply(rho, V)
        return op

    make()  # tunes
    free = _free()
    keep = make()
    need = free - _free()
    want = V.cpu().numpy()
    del keep
    V.zero_()
    with _Leave(need - 20 * MIB):
        keep = make()
        del keep
    np.testing.assert_array_equal(V.cpu().numpy(), want)


def test_fp64_near_field_group_leaves_host_cubes_their_room(dage):
    """GBFMM 121^3: five W slots (180 MB more than one) must not take the
    memory of the two 14 MB cubes that a host-array apply stages."""
    g = dage.Grid3D.cube(-12.0, 20, 0.2)
    quad = dage.GaussQuad(4, 4)
    rho, V = _density(g.shape), _density(g.shape)
    host = np.asfortranarray(rho.cpu().numpy().transpose(2, 1, 0))
    make = lambda: dage.GBFMMCoulomb3D(g, lmax=2, quad=quad)  # noqa: E731
    make().apply(rho, V)  # tunes
    free = _free()
    keep = make()
    need = free - _free()
    want = keep.apply(host)
    del keep
    with _Leave(need + 10 * MIB):
        got = make().apply(host)
    assert np.abs(got - want).max() <= 1e-13 * np.abs(want).max()


def test_refused_allocation_leaves_no_error_behind(dage):
    """A creation refused for memory fails with DAGE_E_NOMEM; the next one, of
    an operator that fits, is not affected."""
    g = dage.Grid3D.cube(-7.8, 13, 0.2)
    quad = dage.GaussQuad(3, 3)
    rho, V = _density(g.shape), _density(g.shape)
    dage.Coulomb3D(g, quad=quad).apply(rho, V)
    want = V.cpu().numpy()
    with _Leave(64 * MIB):
        with pytest.raises(dage.DageError) as e:
            dage.Coulomb3D(dage.Grid3D.cube(-24.0, 40, 0.2), quad=quad, precision="bf16x6")
        assert e.value.code == -3
        del e
        got = _apply(dage.Coulomb3D(g, quad=quad), rho, V)
    assert np.abs(got - want).max() <= 1e-13 * np.abs(want).max()  # another group of t-points


@pytest.mark.parametrize("precision", ["fp64", "fp16x3"])
def test_group_gives_way_to_host_cubes(dage, precision):
    """121^3: an operator whose group of t-points took the memory that a
    host-array apply stages its two 14 MB cubes in gives the group back."""
    g = dage.Grid3D.cube(-12.0, 20, 0.2)
    op = dage.Coulomb3D(g, quad=dage.GaussQuad(9, 8), precision=precision)
    rho, V = _density(g.shape), _density(g.shape)
    want = _apply(op, rho, V).transpose(2, 1, 0)
    host = np.asfortranarray(rho.cpu().numpy().transpose(2, 1, 0))
    with _Leave(10 * MIB):
        got = op.apply(host)
    assert np.abs(got - want).max() <= (1e-13 if precision == "fp64" else 0) * np.abs(want).max()
    with _Leave(10 * MIB):  # and stays as it is then
        np.testing.assert_array_equal(op.apply(host), got)
        out = [np.empty(g.shape, order="F")]
        with pytest.raises(dage.DageError) as e:  # the pipeline's second pair of cubes: no room left
            dage.apply_batched([op], [host], out)
        assert e.value.code == -3
        del e
    dage.apply_batched([op], [host], out)
    np.testing.assert_array_equal(out[0], got)
