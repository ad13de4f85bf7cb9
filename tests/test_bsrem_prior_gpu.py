"""The relative-difference prior inside the fused BSREM step against its float64 formula, for
objects whose denominators lie above, around and far below the range of the kernel's fast
reciprocal, with both boundary quads and inner ones.

With projections of zero the step is f (1 - beta rdp(f)).  Tolerance: 1e-5 of each voxel, as in
the other tests of the prior."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rdp(f, gamma, delta, dr):
    p = np.pad(f, 1, mode="edge")
    out = np.zeros_like(f)
    nx, ny, nz = f.shape
    for i in (-1, 0, 1):
        for j in (-1, 0, 1):
            for k in (-1, 0, 1):
                if i == j == k == 0:
                    continue
                s = p[1 + i:1 + i + nx, 1 + j:1 + j + ny, 1 + k:1 + k + nz]
                w = dr[0] / np.sqrt((dr[0] * i) ** 2 + (dr[1] * j) ** 2 + (dr[2] * k) ** 2)
                d = f - s
                a = gamma * np.abs(d)
                out += w * d * (a + 3 * s + f + 2 * delta) / (f + s + a + delta) ** 2
    return out


@pytest.mark.parametrize("low,delta", [(1e-17, 0.0), (1e-17, 1e-17), (4e-16, 0.0), (0.0, 1e-11),
                                       (1e-3, 1e-11)])
@pytest.mark.parametrize("shape,psf,gamma", [((10, 10, 12), True, 2.0), ((9, 9, 4), False, 0.0)])
def test_prior_term(low, delta, shape, psf, gamma, cuda):
    from pytomography_gb300.metadata.SPECT import SPECTObjectMeta, SPECTProjMeta, SPECTPSFMeta
    from pytomography_gb300.priors import RelativeDifferencePrior
    from pytomography_gb300.projectors.SPECT import SPECTSystemMatrix
    from pytomography_gb300.transforms.SPECT import SPECTPSFTransform
    dr = [0.5, 0.5, 0.4]
    om = SPECTObjectMeta(dr, shape)
    pm = SPECTProjMeta(shape[1:], dr[:2], [0.0, 90.0, 210.0], radii=[20.0] * 3)
    tr = [SPECTPSFTransform(SPECTPSFMeta((0.03, 0.11)))] if psf else []
    H = SPECTSystemMatrix(tr, [], om, pm)
    prior = RelativeDifferencePrior(beta=0.01, gamma=gamma, delta=delta)
    prior.set_object_meta(om)
    rng = np.random.default_rng(3)
    f = rng.random(shape) + 0.5
    f[:, shape[1] // 2:] *= low
    f = f.astype(np.float32)
    x = torch.tensor(f, device=cuda)
    out = torch.empty_like(x)
    g = torch.zeros(3, *shape[1:], device=cuda)
    H.bsrem_step(x, out, g, torch.ones_like(g), torch.zeros_like(x), torch.ones_like(x), 1.0, 1.0,
                 prior=prior, floor_value=0.0)
    f = f.astype(np.float64)
    ref = f * (1 - 0.01 * _rdp(f, gamma, delta, dr))
    assert (ref >= 0).all()
    assert (np.abs(out.cpu().numpy() - ref) <= 1e-5 * ref).all()
