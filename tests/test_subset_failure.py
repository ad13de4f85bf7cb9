"""A subset split that fails in the library is not taken for a finished one: the Python object
keeps no claim to it, the same split can be asked for again, and on the GPU the plan refuses
projections (listmode) or keeps the split before (SPECT) instead of running on freed lists."""
import types

import numpy as np
import pytest
import torch

from conftest import golden, rel_l2


class StubLib:
    """Stands for the library: every set_subsets entry point fails while `fail` is set."""

    def __init__(self):
        self.fail, self.calls = False, []

    def _set(self, plan, n, *lists):
        self.calls.append(n)
        return -3 if self.fail else 0

    gb_pet_set_subsets = gb_spect_set_subsets = gb_pet_sino_set_subsets = _set
    gb_spect_set_subset_lists = _set


def _objects():
    from pytomography_gb300.projectors.PET import PETLMSystemMatrix, PETSinogramSystemMatrix
    from pytomography_gb300.projectors.SPECT import SPECTSystemMatrix, StarGuideSystemMatrix
    lm = PETLMSystemMatrix.__new__(PETLMSystemMatrix)
    lm.proj_meta = types.SimpleNamespace(detector_ids=torch.zeros((12, 2)))
    sino = PETSinogramSystemMatrix.__new__(PETSinogramSystemMatrix)
    sino.proj_meta = types.SimpleNamespace(N_angles=12)
    sino.output_device = torch.device("cpu")
    spect = SPECTSystemMatrix.__new__(SPECTSystemMatrix)
    spect.proj_meta = types.SimpleNamespace(shape=(12, 4, 4), num_projections=12)
    spect._lists_epoch, spect.autotune_enabled = 0, False
    star = StarGuideSystemMatrix.__new__(StarGuideSystemMatrix)
    star.proj_meta = types.SimpleNamespace(angles=torch.arange(12.0), num_projections=12)
    star._H = types.SimpleNamespace(_plan=None)
    for sm in (lm, sino, spect, star):
        sm.device, sm._plan, sm._lib = torch.device("cpu"), None, StubLib()
        sm.subset_indices_array, sm.n_subsets = None, 1
    return {"lm": lm, "sino": sino, "spect": spect, "star": star}


@pytest.mark.parametrize("kind", ["lm", "sino", "spect", "star"])
def test_failed_split_is_asked_for_again(kind):
    sm = _objects()[kind]
    lib = sm._lib
    lib.fail = True
    with pytest.raises(RuntimeError, match="gbtomo error -3"):
        sm.set_n_subsets(4)
    assert sm.subset_indices_array is None
    lib.fail = False
    sm.set_n_subsets(4)
    assert lib.calls == [4, 4] and len(sm.subset_indices_array) == 4
    # a later split that fails leaves no claim to it either
    lib.fail = True
    with pytest.raises(RuntimeError):
        sm.set_n_subsets(3)
    assert sm.subset_indices_array is None or len(sm.subset_indices_array) == 4
    lib.fail = False
    sm.set_n_subsets(3)
    assert len(sm.subset_indices_array) == 3 and lib.calls[-1] == 3


@pytest.mark.gpu
@pytest.mark.parametrize("nth", [1, 2, 6])  # the tiles themselves, and the sort's buffers
def test_listmode_plan_without_tiles_refuses_and_recovers(nth, cuda):
    from pytomography_gb300.metadata import ObjectMeta
    from pytomography_gb300.metadata.PET import PETLMProjMeta
    from pytomography_gb300.projectors.PET import PETLMSystemMatrix
    info = dict(crystalTransNr=1, crystalTransSpacing=4.0, submoduleTransNr=1,
                submoduleTransSpacing=0.0, moduleTransNr=1, moduleTransSpacing=0.0,
                rsectorTransNr=32, crystalAxialNr=4, crystalAxialSpacing=4.0,
                submoduleAxialNr=1, submoduleAxialSpacing=0.0, moduleAxialNr=1,
                moduleAxialSpacing=0.0, rsectorAxialNr=1, radius=90.0, firstCrystalAxis=1,
                NrCrystalsPerRing=32, NrRings=4)
    rng = np.random.default_rng(3)
    i = rng.integers(0, 128, 900)
    ev = torch.as_tensor(np.stack([i, (i + rng.integers(1, 128, 900)) % 128], 1))
    sm = PETLMSystemMatrix(ObjectMeta([6.0] * 3, (20, 20, 5)),
                           PETLMProjMeta(ev, info=info, detector_ids_sensitivity=ev))
    img = torch.rand((20, 20, 5), device=cuda)
    whole = sm.forward(img)
    # a first failure takes the memory of the plan's patch layouts, the next one has none to take
    assert sm._lib.gb_inject_fault(b"alloc", 1) == 0
    sm.set_n_subsets(3)
    assert sm._lib.gb_inject_fault(b"alloc", nth) == 0
    with pytest.raises(RuntimeError):
        sm.set_n_subsets(7)
    sm._lib.gb_inject_fault(b"alloc", 0)
    with pytest.raises(RuntimeError, match="no event tiles"):
        sm.forward(img)
    with pytest.raises(RuntimeError, match="no event tiles"):
        sm.backward(whole)
    sm.set_n_subsets(7)
    assert torch.equal(sm.forward(img, 6), whole[6::7])
    assert torch.equal(sm.forward(img), whole)


@pytest.mark.gpu
@pytest.mark.parametrize("nth", [1, 2, 3])
def test_spect_plan_keeps_its_split_after_a_failure(nth, cuda):
    from test_faults_gpu import _sm
    d, H, f = _sm(cuda)
    H.set_n_subsets(2)
    want = H.forward(f, 1)
    assert H._lib.gb_inject_fault(b"alloc", nth) == 0
    with pytest.raises(RuntimeError):
        H.set_n_subsets(3)
    H._lib.gb_inject_fault(b"alloc", 0)
    assert H.n_subsets == 2 and torch.equal(H.forward(f, 1), want)
    H.set_n_subsets(3)
    ref = golden("spect_even")["fwd_att+psf_f32"]
    assert rel_l2(H.forward(f, 2).cpu().numpy(), ref[2::3]) < 1e-5
