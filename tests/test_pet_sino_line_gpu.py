"""Line kernels of the sinogram projectors at the edges of their tiles against the float64
oracle: slices not divisible by four, more planes than a block has threads and than are
staged at once, unequal transaxial extents, LORs whose principal axis is z, an even number of
TOF bins, few lines (ring pairs split over blocks) and more slices than the line kernels hold.

Tolerance: 1e-5 relative L2, as in the other sinogram tests."""
import numpy as np
import pytest
import torch

import oracle
from conftest import rel_l2

pytestmark = pytest.mark.gpu
TOL = 1e-5

# image shape, voxel (mm), crystals, rings, radius (mm), TOF bins, subsets
CASES = [
    ((40, 40, 7), (4.0, 4.0, 4.0), 60, 8, 120.0, 0, 1),
    ((36, 150, 12), (4.0, 1.5, 3.0), 48, 6, 130.0, 0, 3),
    ((150, 33, 12), (1.5, 4.0, 3.0), 48, 6, 130.0, 9, 3),
    ((24, 24, 40), (4.0, 4.0, 4.0), 24, 30, 55.0, 0, 2),   # steep LORs
    ((24, 24, 40), (4.0, 4.0, 4.0), 24, 30, 55.0, 8, 6),
    ((130, 130, 250), (1.0, 1.0, 0.5), 16, 5, 90.0, 0, 4),  # columns staged in two rounds
    ((12, 12, 420), (8.0, 8.0, 0.5), 16, 4, 90.0, 0, 1),    # beyond the line kernels
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(map(str, c[0])) + f"-tof{c[5]}")
def test_line_kernels_match_oracle(case, cuda):
    from pytomography_gb300.metadata import ObjectMeta
    from pytomography_gb300.metadata.PET import PETSinogramPolygonProjMeta, PETTOFMeta
    from pytomography_gb300.projectors.PET import PETSinogramSystemMatrix
    shape, vox, nt, nr, radius, bins, subsets = case
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
    sub = None
    if subsets > 1:
        sm.set_n_subsets(subsets)
        sub = subsets - 1
    xs, xe = (t.numpy() for t in sm._get_xyz_sinogram_coordinates(sub))
    rng = np.random.default_rng(8)
    img = rng.random(shape) + 0.2
    fwd = sm.forward(torch.tensor(img, dtype=torch.float32, device=cuda), sub)
    ref = o.lor_forward_tof(img, xs, xe) if bins else o.lor_forward(img, xs, xe)
    assert rel_l2(fwd.cpu().numpy().reshape(-1), ref.reshape(-1)) < TOL
    g = rng.random(ref.shape) * (rng.random(ref.shape) < 0.7)  # some empty bins
    bwd = sm.backward(torch.tensor(g.reshape(tuple(fwd.shape)), dtype=torch.float32,
                                   device=cuda), sub)
    refb = o.lor_backward_tof(g, xs, xe) if bins else o.lor_backward(g, xs, xe)
    assert rel_l2(bwd.cpu().numpy(), refb) < TOL
