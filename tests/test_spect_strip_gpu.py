"""Strip kernels of the PSF projectors (planes of at most 128 rows and 128 z values,
attenuation before the PSF) at the edges of their tiles, against the float64 oracle:
z extents around the 16-value groups, the lane widths (32 / 64 / 128 values) and odd ones,
the narrowest and widest taps, one angle, more angles than one group of 16, no attenuation,
a 1-D PSF, radii per angle and buffers that are not 16-byte aligned.

Tolerance: 1e-5 relative L2 per projection and per object, as in every parity test; the
samples' float32 coordinates (6 ulp of the position in a padded plane of at most 182 pixels)
bound the error at a few 1e-6."""
import numpy as np
import pytest
import torch

import oracle
from conftest import rel_l2

pytestmark = pytest.mark.gpu
TOL = 1e-5

# n, nz, angles, (a, b) of sigma(d), order, 2-D PSF, orbit amplitude
CASES = [
    (8, 1, 3, (0.03, 0.11), "ap", True, 0.0),
    (16, 15, 5, (0.03, 0.11), "ap", True, 0.0),
    (33, 16, 6, (0.03, 0.11), "ap", True, 2.0),
    (32, 17, 1, (0.03, 0.11), "ap", True, 0.0),
    (40, 33, 4, (0.03, 0.11), "p", True, 0.0),
    (64, 64, 18, (0.03, 0.11), "ap", True, 0.0),
    (65, 65, 3, (0.03, 0.11), "ap", False, 1.0),
    (97, 82, 2, (0.03, 0.11), "ap", True, 1.0),
    (128, 127, 2, (0.03, 0.11), "ap", True, 0.0),
    (48, 128, 2, (0.0, 0.05), "ap", True, 0.0),     # one tap carries the kernel
    (48, 40, 2, (0.0, 3.1), "ap", True, 0.0),       # 45 taps
    (128, 128, 1, (0.0, 2.6), "ap", True, 0.0),     # 37 taps, the largest plane
]


def _pair(n, nz, n_angles, ab, order, two_d, orbit):
    from pytomography_gb300.metadata.SPECT import SPECTObjectMeta, SPECTProjMeta, SPECTPSFMeta
    from pytomography_gb300.projectors.SPECT import SPECTSystemMatrix
    from pytomography_gb300.transforms.SPECT import SPECTAttenuationTransform, SPECTPSFTransform
    rng = np.random.default_rng(n * 1000 + nz)
    dr = 0.442
    angles = list(np.linspace(0, 360, n_angles + 1)[:-1] + 7.0)
    radii = [22.0 + round(orbit * (k % 3), 1) for k in range(n_angles)]
    f = rng.random((n, n, nz))
    mu = 0.15 * rng.random((n, n, nz))
    psf = SPECTPSFTransform(SPECTPSFMeta(ab, kernel_dimensions="2D" if two_d else "1D"))
    ts = ([SPECTAttenuationTransform(torch.tensor(mu, dtype=torch.float32))]
          if "a" in order else []) + [psf]
    H = SPECTSystemMatrix(ts, [], SPECTObjectMeta([dr] * 3, (n, n, nz)),
                          SPECTProjMeta((n, nz), [dr] * 2, angles, radii=radii))
    # the metadata keeps the angles in single precision
    o = oracle.SpectOracle((n, n, nz), (dr,) * 3, [float(np.float32(a)) for a in angles], radii,
                           mu=mu if "a" in order else None, psf=ab, order=order, psf_2d=two_d)
    return H, o, f, rng.random((n_angles, n, nz))


def _unaligned(a, cuda):
    """The array in device memory at an address that is 4 bytes past a 16-byte boundary."""
    buf = torch.zeros(a.size + 8, device=cuda)
    v = buf[1:1 + a.size].view(a.shape)
    v.copy_(torch.tensor(a, dtype=torch.float32))
    assert v.data_ptr() % 16 == 4 and v.is_contiguous()
    return v


@pytest.mark.parametrize("case", CASES, ids=lambda c: f"{c[0]}x{c[1]}-{c[2]}ang-{c[4]}")
def test_strip_projectors_match_oracle(case, cuda):
    H, o, f, g = _pair(*case)
    ft = torch.tensor(f, dtype=torch.float32, device=cuda)
    gt = torch.tensor(g, dtype=torch.float32, device=cuda)
    ref = o.forward(f)
    fwd = H.forward(ft)
    assert torch.isfinite(fwd).all()
    for a in range(len(ref)):
        assert rel_l2(fwd[a].cpu().numpy(), ref[a]) < TOL, a
    assert torch.equal(fwd, H.forward(ft))  # same sums in the same order
    assert rel_l2(H.backward(gt).cpu().numpy(), o.backward(g)) < TOL
    assert rel_l2(H.backward_adjoint(gt).cpu().numpy(), o.adjoint(g)) < TOL
    assert torch.equal(H.forward(_unaligned(f, cuda)), fwd)
    assert torch.equal(H.backward(_unaligned(g, cuda)), H.backward(gt))
    assert H.device_status() == 0
