"""Back projection of plans without PSF: the one-kernel form (whole z quads, 16-byte aligned
projections) against the two-kernel form, which a misaligned projection buffer takes, bit for
bit (the same products and sums), and both against the float64 oracle at 1e-5.  Sizes: one quad
per row (sample table too large, no fused form), rows that do and do not divide a warp, more
angles than a group, one angle, no attenuation."""
import numpy as np
import pytest
import torch

import oracle
from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nz,angles,att", [(16, 4, 12, True), (17, 12, 37, True),
                                             (24, 64, 5, True), (13, 36, 1, False),
                                             (20, 132, 3, True)])
def test_one_kernel_backward(n, nz, angles, att, cuda):
    from pytomography_gb300.metadata.SPECT import SPECTObjectMeta, SPECTProjMeta
    from pytomography_gb300.projectors.SPECT import SPECTSystemMatrix
    from pytomography_gb300.transforms.SPECT import SPECTAttenuationTransform
    rng = np.random.default_rng(n)
    shape, dx = (n, n, nz), 0.48
    mu = (rng.random(shape) * 0.2).astype(np.float32)
    ang = np.linspace(3.0, 363.0, angles, endpoint=False)
    om = SPECTObjectMeta([dx] * 3, shape)
    pm = SPECTProjMeta(shape[1:], [dx, dx], [float(a) for a in ang], radii=[20.0] * angles)
    H = SPECTSystemMatrix([SPECTAttenuationTransform(torch.tensor(mu))] if att else [], [], om, pm)
    g = rng.random((angles, n, nz)).astype(np.float32)
    flat = torch.zeros(g.size + 4, device=cuda)
    outs = []
    for off in (0, 1):
        p = flat[off:off + g.size].view(g.shape)
        p.copy_(torch.tensor(g))
        outs.append(H.backward(p).cpu().numpy())
    assert np.array_equal(outs[0], outs[1])
    assert outs[0].any()
    # the metadata keeps the angles in single precision
    o = oracle.SpectOracle(shape, (dx,) * 3, [float(np.float32(a)) for a in ang],
                           [20.0] * angles, mu=mu.astype(np.float64) if att else None,
                           order="a" if att else "")
    assert rel_l2(outs[0], o.backward(g.astype(np.float64))) < 1e-5
