"""The plane-at-a-time PSF kernels, which plans of the PSF-before-attenuation order and plans of
more than 128 rows run: every tile tuning against the float64 oracle, and batches of such plans
alone and beside strip plans against each plan's own projections (1e-5 relative L2, as in every
parity test)."""
import numpy as np
import pytest
import torch

import oracle
from conftest import rel_l2

pytestmark = pytest.mark.gpu
TOL = 1e-5


def _plan(n, nz, angles, order, seed=1):
    from pytomography_gb300.metadata.SPECT import SPECTObjectMeta, SPECTProjMeta, SPECTPSFMeta
    from pytomography_gb300.projectors.SPECT import SPECTSystemMatrix
    from pytomography_gb300.transforms.SPECT import SPECTAttenuationTransform, SPECTPSFTransform
    rng = np.random.default_rng(seed)
    dr = 0.442
    ang = [float(np.float32(a)) for a in np.linspace(5.0, 365.0, angles, endpoint=False)]
    f, mu = rng.random((n, n, nz)), 0.15 * rng.random((n, n, nz))
    made = {"a": lambda: SPECTAttenuationTransform(torch.tensor(mu, dtype=torch.float32)),
            "p": lambda: SPECTPSFTransform(SPECTPSFMeta((0.03, 0.11)))}
    H = SPECTSystemMatrix([made[c]() for c in order], [], SPECTObjectMeta([dr] * 3, (n, n, nz)),
                          SPECTProjMeta((n, nz), [dr] * 2, ang, radii=[22.0] * angles))
    o = oracle.SpectOracle((n, n, nz), (dr,) * 3, ang, [22.0] * angles,
                           mu=mu if "a" in order else None, psf=(0.03, 0.11), order=order)
    return H, o, f


# PSF first (quads and single values in z), and more than 128 rows
@pytest.mark.parametrize("n,nz,order", [(48, 40, "pa"), (40, 37, "pa"), (132, 32, "ap")])
def test_every_tuning_of_the_plane_kernels(n, nz, order, cuda):
    H, o, f = _plan(n, nz, 6, order)
    ft = torch.tensor(f, dtype=torch.float32, device=cuda)
    ref = o.forward(f)
    g = np.random.default_rng(2).random(ref.shape)
    gt = torch.tensor(g, dtype=torch.float32, device=cuda)
    refb, refa = o.backward(g), o.adjoint(g)
    seen = set()
    for tpb in (512, 768):
        for zt in (0, 16, 24):
            for items in (1, 2):
                try:
                    H.set_tuning(fwd_tpb=tpb, fwd_zt=zt, fwd_items=items, b1_zt=zt,
                                 b1_items=items)
                except RuntimeError:
                    continue  # the tile does not fit
                seen.add((tpb, zt, items))
                fwd = H.forward(ft).cpu().numpy()
                for a in range(len(ref)):
                    assert rel_l2(fwd[a], ref[a]) < TOL, (tpb, zt, items, a)
                assert rel_l2(H.backward(gt).cpu().numpy(), refb) < TOL, (tpb, zt, items)
                assert rel_l2(H.backward_adjoint(gt).cpu().numpy(), refa) < TOL, (tpb, zt, items)
    assert {s[0] for s in seen} == {512, 768} and {s[1] for s in seen} == {0, 16, 24}
    assert H.device_status() == 0


# (n, nz, angles, order) of each entry: plane-at-a-time plans alone, and mixed with strip plans
BATCHES = {"plane": [(32, 24, 18, "pa"), (24, 40, 9, "pa")],
           "mixed": [(40, 36, 18, "ap"), (32, 24, 18, "pa"), (24, 64, 9, "p"), (48, 20, 40, "pa")]}


@pytest.mark.parametrize("kind", list(BATCHES))
def test_batches_of_plane_kernels(kind, cuda):
    from pytomography_gb300.batched import SpectBatch, common_psf_bucket
    made = [_plan(*e, seed=k) for k, e in enumerate(BATCHES[kind])]
    Hs = [m[0] for m in made]
    common_psf_bucket(Hs)
    for H in Hs:
        H.set_n_subsets(3)
    b = SpectBatch(Hs)
    fs = [torch.tensor(m[2], dtype=torch.float32, device=cuda) for m in made]
    for sub in (None, 2):
        proj = b.forward(fs, sub)
        for (H, o, f), x, p in zip(made, fs, proj):
            own = H.forward(x, sub).cpu().numpy()
            assert rel_l2(p.cpu().numpy(), own) < TOL
            if sub is None:
                assert rel_l2(own, o.forward(f)) < TOL
        gp = [torch.rand_like(p) for p in proj]
        for adj in (False, True):
            back = b.backward(gp, sub, adjoint=adj)
            for H, g, x in zip(Hs, gp, back):
                own = (H.backward_adjoint if adj else H.backward)(g, sub)
                assert rel_l2(x.cpu().numpy(), own.cpu().numpy()) < TOL, (sub, adj)


def test_batched_osem_of_mixed_plans(cuda):
    from pytomography_gb300.algorithms import OSEM
    from pytomography_gb300.batched import BatchedOSEM
    from pytomography_gb300.likelihoods import PoissonLogLikelihood
    made = [_plan(*e, seed=k) for k, e in enumerate(BATCHES["mixed"])]
    liks = lambda: [PoissonLogLikelihood(H, H.forward(torch.tensor(  # noqa: E731
        f, dtype=torch.float32, device=cuda))) for H, _, f in made]
    refs = [OSEM(k, fused=True)(2, 3).clone() for k in liks()]
    batch = BatchedOSEM(liks(), n_subsets=3)
    assert batch.mode == "persistent"
    for a, r in zip(batch(2), refs):
        assert torch.isfinite(a).all()
        assert rel_l2(a.cpu().numpy(), r.cpu().numpy()) < TOL


def test_batch_of_1d_and_2d_plans(cuda):
    """Strip plans of a 1-D and a 2-D PSF in one batch."""
    from pytomography_gb300.batched import SpectBatch, common_psf_bucket
    from test_spect_strip_gpu import _pair
    made = [_pair(n, nz, 6, (0.03, 0.11), "ap", two_d, 0.0)
            for n, nz, two_d in ((40, 36, False), (32, 64, True), (24, 100, False))]
    Hs = [m[0] for m in made]
    common_psf_bucket(Hs)
    for H in Hs:
        H.set_n_subsets(2)
    b = SpectBatch(Hs)
    fs = [torch.tensor(m[2], dtype=torch.float32, device=cuda) for m in made]
    gs = [torch.tensor(m[3], dtype=torch.float32, device=cuda) for m in made]
    for (H, o, f, g), p, x in zip(made, b.forward(fs, None), b.backward(gs, None)):
        assert rel_l2(p.cpu().numpy(), o.forward(f)) < TOL
        assert rel_l2(x.cpu().numpy(), o.backward(g)) < TOL
