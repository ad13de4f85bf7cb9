"""The relative-difference prior in the fused BSREM step for rows whose last z quad is partial
(strip plans of any nz) and for the one-kernel back projection without PSF, whose sample table
must fit its block: against the float64 formula, for denominators above, around and far below
the range of the fast reciprocal.  As test_bsrem_prior_gpu: projections of zero, so that the
step is f (1 - beta rdp(f)); tolerance 1e-5 of each voxel."""
import numpy as np
import pytest
import torch

from test_bsrem_prior_gpu import _rdp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("low,delta", [(1e-17, 0.0), (4e-16, 0.0), (0.0, 1e-11), (1e-3, 1e-11)])
@pytest.mark.parametrize("shape,psf,gamma", [
    ((9, 9, 1), True, 2.0), ((8, 8, 2), True, 2.0), ((9, 9, 3), True, 0.0),
    ((10, 10, 5), True, 2.0), ((12, 12, 39), True, 2.0), ((11, 11, 66), True, 2.0),
    # without PSF: 64 rows x 3 angles, 32 x 3 and 8 x 3 entries of the 512 in a block's table
    ((9, 9, 16), False, 2.0), ((9, 9, 32), False, 0.0), ((10, 10, 132), False, 2.0)])
def test_prior_term_on_any_row(low, delta, shape, psf, gamma, cuda):
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
    rng = np.random.default_rng(4)
    f = rng.random(shape) + 0.5
    f[:, shape[1] // 2:] *= low
    f = f.astype(np.float32)
    x = torch.tensor(f, device=cuda)
    out = torch.full((x.numel() + 8,), -7.0, device=cuda)
    g = torch.zeros(3, *shape[1:], device=cuda)
    y = out[:x.numel()].view(shape)
    H.bsrem_step(x, y, g, torch.ones_like(g), torch.zeros_like(x), torch.ones_like(x), 1.0, 1.0,
                 prior=prior, floor_value=0.0)
    assert (out[x.numel():] == -7.0).all()
    f = f.astype(np.float64)
    ref = f * (1 - 0.01 * _rdp(f, gamma, delta, dr))
    assert (ref >= 0).all()
    assert (np.abs(y.cpu().numpy() - ref) <= 1e-5 * ref).all()
