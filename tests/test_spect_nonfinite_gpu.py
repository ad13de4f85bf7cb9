"""Infinities and NaN in the strip projectors stay where the blur can reach: a 1-D PSF leaves
every other slice as it is, bit for bit, a 2-D one the slices farther away than its taps; and a
1-D plan ignores z taps that its description holds all the same."""
import numpy as np
import pytest
import torch

from conftest import rel_l2
from test_spect_strip_gpu import _pair

pytestmark = pytest.mark.gpu
REACH = 4  # half width of the taps of sigma 0.05 cm at most, with the zeros that pad them


@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
@pytest.mark.parametrize("two_d", [False, True], ids=["1D", "2D"])
@pytest.mark.parametrize("shape", [(32, 17), (40, 64), (97, 83)])
def test_non_finite_slice_stays_local(shape, two_d, bad, cuda):
    H, _, f, g = _pair(*shape, 3, (0.0, 0.05), "ap", two_d, 0.0)
    n, nz = shape
    z0, reach = nz // 2, REACH if two_d else 0
    far = [z for z in range(nz) if abs(z - z0) > reach]
    ft = torch.tensor(f, dtype=torch.float32, device=cuda)
    gt = torch.tensor(g, dtype=torch.float32, device=cuda)
    fb, gb = ft.clone(), gt.clone()
    fb[n // 2, n // 2, z0] = bad
    gb[:, n // 2, z0] = bad
    for fn, x, xb in ((H.forward, ft, fb), (H.backward, gt, gb), (H.backward_adjoint, gt, gb)):
        a, b = fn(x), fn(xb)
        assert torch.isfinite(a).all()
        assert torch.equal(a[..., far], b[..., far])
        assert not torch.isfinite(b[..., z0]).all()


@pytest.mark.parametrize("shape", [(24, 20), (24, 33)])
def test_1d_plan_ignores_z_taps(shape, cuda):
    from pytomography_gb300 import _lib, reference_binding
    outs = []
    for z_taps in (False, True):
        H, o, f, g = _pair(*shape, 3, (0.03, 0.11), "ap", False, 1.0)
        d = reference_binding.describe(H)
        assert d["psf_2d"] == 0 and not np.any(d["psf_taps_z"])
        if z_taps:
            d["psf_taps_z"] = d["psf_taps_r"].copy()
        p = reference_binding.Plan(d, cuda)
        ft = torch.tensor(f, dtype=torch.float32, device=cuda)
        out = torch.empty(o.forward(f).shape, device=cuda)
        _lib.check(p.lib.gb_spect_forward(p.handle, _lib.ptr(ft), _lib.ptr(out), -1,
                                          _lib.stream_handle(ft.device)))
        gt = torch.tensor(g, dtype=torch.float32, device=cuda)
        back = torch.empty_like(ft)
        _lib.check(p.lib.gb_spect_backward(p.handle, _lib.ptr(gt), _lib.ptr(back), -1, 0,
                                           _lib.stream_handle(ft.device)))
        torch.cuda.synchronize()
        assert rel_l2(out.cpu().numpy(), o.forward(f)) < 1e-5
        assert rel_l2(back.cpu().numpy(), o.backward(g)) < 1e-5
        outs.append((out, back))
    assert all(torch.equal(a, b) for a, b in zip(*outs))
