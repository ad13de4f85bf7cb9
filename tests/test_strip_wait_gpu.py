"""The bounded waits of the forward projector's copies when they run out: the strip form leaves
no sums behind (what the plan's partial sums held before stays), the plane-at-a-time form (N >
128) reports as well, and both work again afterwards.  Nothing is left in flight: every copy
that is issued is waited for."""
import numpy as np
import pytest
import torch

from test_spect_strip_gpu import _pair

pytestmark = pytest.mark.gpu


def _plan(shape, cuda):
    """A plan of three angles and an object."""
    H, _, f, _ = _pair(*shape, 3, (0.03, 0.11), "ap", True, 0.0)
    return H, torch.tensor(np.asarray(f), dtype=torch.float32, device=cuda)


def _rows(H, cuda):
    return torch.empty(tuple(int(v) for v in H.proj_meta.shape), device=cuda)


def _call(H, f, out):
    from pytomography_gb300 import _lib
    rc = H._lib.gb_spect_forward(H._plan, _lib.ptr(f), _lib.ptr(out), -1,
                                 _lib.stream_handle(f.device))
    assert rc == 0
    torch.cuda.synchronize()
    return H.device_status()


# (N, nz), polls until a wait gives up: one and several planes per work item, one or two
# warps of outputs, several row slabs
@pytest.mark.parametrize("shape", [(24, 16), (70, 33), (128, 128)])
@pytest.mark.parametrize("polls", [1, 7])
def test_strip_forward_that_gives_up_stores_nothing(shape, polls, cuda):
    H, f = _plan(shape, cuda)
    first, second = _rows(H, cuda), _rows(H, cuda)
    assert _call(H, f, first) == 0
    assert H._lib.gb_spect_set_debug(H._plan, 1, polls) == 0
    assert _call(H, f * 2 + 1, second) == 1
    assert torch.equal(first, second)  # the sums of the call before, added again
    H._lib.gb_spect_clear_device_status(H._plan)
    assert H._lib.gb_spect_set_debug(H._plan, 0, 0) == 0
    assert _call(H, f, second) == 0
    assert torch.equal(first, second)


def test_plane_kernel_that_gives_up_reports(cuda):
    H, f = _plan((132, 16), cuda)
    out, ref = _rows(H, cuda), _rows(H, cuda)
    assert _call(H, f, ref) == 0
    assert H._lib.gb_spect_set_debug(H._plan, 1, 16) == 0
    assert _call(H, f, out) == 1
    H._lib.gb_spect_clear_device_status(H._plan)
    assert H._lib.gb_spect_set_debug(H._plan, 0, 0) == 0
    assert _call(H, f, out) == 0
    assert torch.equal(out, ref)
