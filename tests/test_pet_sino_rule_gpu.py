"""The choice between the line kernels of the sinogram projectors and tracing each LOR, on both
sides of its rule, with and without TOF: which kernels a call runs, and its result against the
float64 oracle (1e-5 relative L2, as in the other sinogram tests).  Few ring pairs and many slices
are traced; more slices than fit shared memory always; a TOF forward may stage its columns in two
rounds."""
import numpy as np
import pytest
import torch

import oracle
from conftest import rel_l2

pytestmark = pytest.mark.gpu
TOL = 1e-5

# image shape, voxel (mm), crystals, rings, radius (mm), TOF bins, line forward, line back
CASES = [
    ((40, 40, 1), (4.0, 4.0, 4.0), 24, 1, 120.0, 0, False, True),    # one ring
    ((40, 40, 1), (4.0, 4.0, 4.0), 24, 1, 120.0, 9, False, True),
    ((40, 41, 30), (4.0, 4.0, 2.0), 24, 2, 120.0, 0, False, True),   # two rings, many slices
    ((40, 41, 30), (4.0, 4.0, 2.0), 24, 2, 120.0, 9, False, True),
    ((40, 41, 12), (4.0, 4.0, 4.0), 24, 6, 120.0, 0, True, True),
    ((40, 41, 12), (4.0, 4.0, 4.0), 24, 6, 120.0, 9, True, True),
    ((130, 130, 250), (1.0, 1.0, 0.5), 16, 5, 90.0, 0, False, False),
    ((130, 130, 250), (1.0, 1.0, 0.5), 12, 18, 90.0, 9, True, False),  # two rounds of columns
    ((12, 12, 447), (8.0, 8.0, 0.5), 12, 22, 90.0, 0, False, False),  # profiles do not fit
    ((12, 12, 420), (8.0, 8.0, 0.5), 12, 8, 90.0, 13, False, False),
]


def _kernels(fn):
    from torch.profiler import ProfilerActivity, profile
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        out = fn()
        torch.cuda.synchronize()
    return out, " ".join(e.key for e in prof.key_averages())


@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(map(str, c[0])) +
                         f"-{c[3]}rings-tof{c[5]}")
def test_rule_and_result(case, cuda):
    from pytomography_gb300.metadata import ObjectMeta
    from pytomography_gb300.metadata.PET import PETSinogramPolygonProjMeta, PETTOFMeta
    from pytomography_gb300.projectors.PET import PETSinogramSystemMatrix
    shape, vox, nt, nr, radius, bins, line_fwd, line_bwd = case
    info = dict(crystalTransNr=1, crystalTransSpacing=4.0, submoduleTransNr=1,
                submoduleTransSpacing=0.0, moduleTransNr=1, moduleTransSpacing=0.0,
                rsectorTransNr=nt, crystalAxialNr=nr, crystalAxialSpacing=4.0,
                submoduleAxialNr=1, submoduleAxialSpacing=0.0, moduleAxialNr=1,
                moduleAxialSpacing=0.0, rsectorAxialNr=1, radius=radius, firstCrystalAxis=1,
                NrCrystalsPerRing=nt, NrRings=nr, min_rsector_difference=0)
    tm = PETTOFMeta(bins, 2.2 * radius, 40.0) if bins else None
    sm = PETSinogramSystemMatrix(ObjectMeta(list(vox), shape),
                                 PETSinogramPolygonProjMeta(info, tm))
    tof = None if tm is None else (bins, float(tm.bin_width), float(tm.sigma),
                                   float(tm.center_offset), float(tm.n_sigmas))
    o = oracle.PetLMOracle(shape, vox, sm.proj_meta.scanner_lut.numpy(), tof=tof)
    xs, xe = (t.numpy() for t in sm._get_xyz_sinogram_coordinates(None))
    rng = np.random.default_rng(9)
    img = rng.random(shape) + 0.2
    it = torch.tensor(img, dtype=torch.float32, device=cuda)
    fwd, names = _kernels(lambda: sm.forward(it))
    assert ("k_sino_fwd_line" in names) == line_fwd, names
    ref = o.lor_forward_tof(img, xs, xe) if bins else o.lor_forward(img, xs, xe)
    assert rel_l2(fwd.cpu().numpy().reshape(-1), ref.reshape(-1)) < TOL
    g = rng.random(ref.shape) * (rng.random(ref.shape) < 0.7)
    gt = torch.tensor(g.reshape(tuple(fwd.shape)), dtype=torch.float32, device=cuda)
    bwd, names = _kernels(lambda: sm.backward(gt))
    assert ("k_sino_bwd_line" in names) == line_bwd, names
    refb = o.lor_backward_tof(g, xs, xe) if bins else o.lor_backward(g, xs, xe)
    assert rel_l2(bwd.cpu().numpy(), refb) < TOL
