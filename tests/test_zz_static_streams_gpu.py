"""gb_spect_forward_static keeps to its fixed arrays: it may run beside the plan's own projections
on another stream (interleaved calls with different objects give what one stream gives), and it
refuses what needs more partial sums whatever the groups."""
import numpy as np
import pytest
import torch

from conftest import rel_l2
from test_spect_strip_gpu import _pair
from test_zz_no_alloc import _static_fn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nz,angles", [(128, 128, 6), (128, 128, 5), (48, 33, 20)])
def test_static_beside_plan_calls(n, nz, angles, cuda):
    from pytomography_gb300 import _lib
    H, _, f, g = _pair(n, nz, angles, (0.03, 0.11), "ap", True, 0.0)
    fn = _static_fn(H._lib)
    objs = [torch.tensor(f, dtype=torch.float32, device=cuda) * (k + 1) + k for k in range(6)]
    want = [H.forward(x) for x in objs]
    back = [H.backward(y) for y in want]
    outs = [torch.full_like(want[0], float("nan")) for _ in objs]
    plan, gback = [], []
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    for k, x in enumerate(objs):
        _lib.check(fn(H._plan, _lib.ptr(x), _lib.ptr(outs[k]), -1, a.cuda_stream))
        with torch.cuda.stream(b):
            plan.append(H.forward(objs[-1 - k]))
            gback.append(H.backward(want[k]))
    torch.cuda.synchronize()
    for k in range(len(objs)):
        assert torch.equal(plan[k], want[-1 - k]) and torch.equal(gback[k], back[k])
        assert rel_l2(outs[k].cpu().numpy(), want[k].cpu().numpy()) < 1e-5


def test_static_limit_counts_every_angle(cuda):
    from pytomography_gb300 import _lib
    from pytomography_gb300.metadata.SPECT import SPECTObjectMeta, SPECTProjMeta, SPECTPSFMeta
    from pytomography_gb300.projectors.SPECT import SPECTSystemMatrix
    from pytomography_gb300.transforms.SPECT import SPECTPSFTransform
    n, nz, angles = 64, 128, 520  # 520 * 64 * 128 floats > 4,194,304, though 16 at a time fit
    om = SPECTObjectMeta([0.4] * 3, (n, n, nz))
    pm = SPECTProjMeta((n, nz), [0.4] * 2, list(np.linspace(0, 360, angles, endpoint=False)),
                       radii=[20.0] * angles)
    H = SPECTSystemMatrix([SPECTPSFTransform(SPECTPSFMeta((0.03, 0.11)))], [], om, pm)
    H.set_n_subsets(2)
    fn = _static_fn(H._lib)
    f = torch.ones((n, n, nz), device=cuda)
    out = torch.empty((angles, n, nz), device=cuda)
    assert fn(H._plan, _lib.ptr(f), _lib.ptr(out), -1, _lib.stream_handle(cuda)) == -2
    assert fn(H._plan, _lib.ptr(f), _lib.ptr(out), 0, _lib.stream_handle(cuda)) == 0
    assert rel_l2(out[:260].cpu().numpy(), H.forward(f, 0).cpu().numpy()) < 1e-5
