"""Entries of a persistent tune cache that were timed with earlier kernels do
not decide the launches of the present ones."""
import pytest

pytestmark = pytest.mark.gpu


def test_entries_without_a_revision_are_timed_anew(dage, tmp_path):
    import torch

    prop = torch.cuda.get_device_properties(0)
    device = prop.name.replace(" ", "_") + f"/sm{prop.multi_processor_count}"
    old = {
        "op3d_fp64/37x37,37x37,37x37,P13": "128 32 128",
        "op3d_mixed3/37x37,37x37,37x37,P13": "4 3",
        "gbfmm_near_fp64/37x37x37,P13,boxes64": "128 32 128",
        "gbfmm_near_fp16x3/37x37x37,P13,boxes64": "128",
    }
    path = tmp_path / "tune.txt"
    path.write_text("".join(f"{device}/{k} {v}\n" for k, v in old.items()))
    dage.set_tune_cache(str(path))
    try:
        g = dage.Grid3D.cube(-3.6, 6, 0.2)
        quad = dage.GaussQuad(7, 6)
        dage.Coulomb3D(g, quad=quad)
        assert dage.Coulomb3D(g, quad=quad, precision="fp16x3").schedule[1] == 8  # not the entry's 3
        dage.GBFMMCoulomb3D(g, lmax=2, quad=quad)
        dage.GBFMMCoulomb3D(g, lmax=2, quad=quad, precision="fp16x3")
        lines = path.read_text().splitlines()[len(old):]
        for k in old:  # each was timed and stored under its own key
            assert sum(("/" + k + " ") in line for line in lines) == 1, (k, lines)
    finally:
        dage.set_tune_cache(None)
