"""Patch layout of the listmode projectors (one 16-byte cell per plane of a LOR) at the edges of
its arrays against the float64 oracle: unequal transaxial extents, one slice, odd slice
counts, LORs that graze the image or run along z, an even number of TOF bins; enough events
per voxel for the layout to be taken, and a subset with too few.

Tolerance: 1e-5 relative L2, as in the other listmode tests."""
import numpy as np
import pytest
import torch

import oracle
from conftest import rel_l2

pytestmark = pytest.mark.gpu
TOL = 1e-5

# image shape, voxel (mm), crystals, rings, radius (mm), TOF bins, events, subsets
CASES = [
    ((20, 31, 7), (6.0, 4.0, 4.0), 40, 8, 90.0, 0, 6000, 1),
    ((31, 20, 8), (4.0, 6.0, 4.0), 40, 8, 90.0, 9, 6000, 2),
    ((16, 16, 1), (8.0, 8.0, 8.0), 32, 2, 90.0, 8, 4000, 1),
    ((12, 12, 33), (6.0, 6.0, 4.0), 16, 40, 50.0, 0, 8000, 1),   # steep LORs
    ((33, 40, 5), (4.0, 3.0, 4.0), 48, 4, 90.0, 13, 9000, 60),   # subsets below the rule
    # the smallest lists that the forward takes the layout for, and one event less
    ((21, 30, 7), (6.0, 4.0, 4.0), 40, 8, 90.0, 0, 40000, 1),
    ((31, 20, 8), (4.0, 6.0, 4.0), 40, 8, 90.0, 9, 80001, 2),
    ((16, 15, 1), (8.0, 8.0, 8.0), 32, 2, 90.0, 8, 39999, 1),
    ((12, 13, 33), (6.0, 6.0, 4.0), 16, 40, 50.0, 13, 40001, 1),
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(map(str, c[0])) + f"-tof{c[5]}")
def test_patch_layout_matches_oracle(case, cuda):
    from pytomography_gb300.likelihoods import PoissonLogLikelihood
    from pytomography_gb300.metadata import ObjectMeta
    from pytomography_gb300.metadata.PET import PETLMProjMeta, PETTOFMeta
    from pytomography_gb300.projectors.PET import PETLMSystemMatrix
    shape, vox, nt, nr, radius, bins, n, subsets = case
    info = dict(crystalTransNr=1, crystalTransSpacing=4.0, submoduleTransNr=1,
                submoduleTransSpacing=0.0, moduleTransNr=1, moduleTransSpacing=0.0,
                rsectorTransNr=nt, crystalAxialNr=nr, crystalAxialSpacing=4.0,
                submoduleAxialNr=1, submoduleAxialSpacing=0.0, moduleAxialNr=1,
                moduleAxialSpacing=0.0, rsectorAxialNr=1, radius=radius, firstCrystalAxis=1,
                NrCrystalsPerRing=nt, NrRings=nr)
    rng = np.random.default_rng(11)
    i = rng.integers(0, nt * nr, n)
    j = rng.integers(0, nt * nr - 1, n)
    cols = [i, j + (j >= i)] + ([rng.integers(0, bins, n)] if bins else [])
    ev = np.stack(cols, 1)
    tm = PETTOFMeta(bins, 2.2 * radius, 40.0) if bins else None
    pairs = torch.as_tensor(ev[:, :2].copy())
    sm = PETLMSystemMatrix(ObjectMeta(list(vox), shape),
                           PETLMProjMeta(torch.as_tensor(ev), info=info, tof_meta=tm,
                                         detector_ids_sensitivity=pairs))
    lut = sm.proj_meta.scanner_lut.numpy()
    tof = None if tm is None else (bins, float(tm.bin_width), float(tm.sigma),
                                   float(tm.center_offset), float(tm.n_sigmas))
    o = oracle.PetLMOracle(shape, vox, lut, tof=tof)
    img = rng.random(shape) + 0.2
    it = torch.tensor(img, dtype=torch.float32, device=cuda)
    # sensitivity over explicit pairs (never TOF)
    sens = oracle.PetLMOracle(shape, vox, lut).backward(np.full(n, 1 + 1e-11), ev[:, :2])
    sens[sens < 1e-7] = 1e7
    assert rel_l2(sm.norm_BP.cpu().numpy(), sens) < TOL
    sub = None
    if subsets > 1:
        sm.set_n_subsets(subsets)
        sub = 1
    es = ev if sub is None else ev[sub::subsets]
    assert rel_l2(sm.forward(it, sub).cpu().numpy(), o.forward(img, es)) < TOL
    w = rng.random(len(es)) * (rng.random(len(es)) < 0.8)
    bwd = sm.backward(torch.tensor(w, dtype=torch.float32, device=cuda), sub)
    assert rel_l2(bwd.cpu().numpy(), o.backward(w, es)) < TOL
    # the fused sub-iteration
    lik = PoissonLogLikelihood(sm, additive_term=torch.full((n,), 0.3, device=cuda))
    lik._set_n_subsets(subsets)
    f = it.clone()
    sm.osem_step(f, lik.projections, lik.additive_term, lik._get_normBP(sub), sub)
    nb = sens * len(es) / n
    bp = o.backward(1 / (o.forward(img, es) + 0.3 + 1e-11), es)
    ref = np.maximum(img + img / (nb + 1e-11) * (bp - nb), 0)
    assert rel_l2(f.cpu().numpy(), ref) < TOL


def test_calls_on_two_streams_take_turns(cuda):
    """Forward and back projections of one plan enqueued on two streams, and a forward recorded
    in a graph, give what one stream gives (1e-5: the additions' order differs)."""
    from pytomography_gb300.metadata import ObjectMeta
    from pytomography_gb300.metadata.PET import PETLMProjMeta
    from pytomography_gb300.projectors.PET import PETLMSystemMatrix
    nt, nr, n, shape = 64, 16, 200_000, (60, 60, 24)
    info = dict(crystalTransNr=1, crystalTransSpacing=4.0, submoduleTransNr=1,
                submoduleTransSpacing=0.0, moduleTransNr=1, moduleTransSpacing=0.0,
                rsectorTransNr=nt, crystalAxialNr=nr, crystalAxialSpacing=4.0,
                submoduleAxialNr=1, submoduleAxialSpacing=0.0, moduleAxialNr=1,
                moduleAxialSpacing=0.0, rsectorAxialNr=1, radius=150.0, firstCrystalAxis=1,
                NrCrystalsPerRing=nt, NrRings=nr)
    rng = np.random.default_rng(5)
    i = rng.integers(0, nt * nr, n)
    j = rng.integers(0, nt * nr - 1, n)
    pairs = torch.as_tensor(np.stack([i, j + (j >= i)], 1))
    sm = PETLMSystemMatrix(ObjectMeta([3.0] * 3, shape),
                           PETLMProjMeta(pairs, info=info,
                                         detector_ids_sensitivity=pairs[:100].clone()))
    imgs = [torch.rand(shape, device=cuda) + k for k in range(8)]
    want = [sm.forward(x) for x in imgs]
    back = [sm.backward(y) for y in want]
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    got, gback = [], []
    for k, x in enumerate(imgs):
        with torch.cuda.stream(streams[k % 2]):
            got.append(sm.forward(x))
            gback.append(sm.backward(want[k]))
    torch.cuda.synchronize()
    gr = torch.cuda.CUDAGraph()
    with torch.cuda.graph(gr, stream=streams[0]):
        rec = sm.forward(imgs[0])
    gr.replay()
    torch.cuda.synchronize()
    for a, b in zip(got + gback + [rec], want + back + [want[0]]):
        assert rel_l2(a.cpu().numpy(), b.cpu().numpy()) < TOL
