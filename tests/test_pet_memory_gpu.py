"""The patch layouts of a listmode plan give way to what the plan cannot do without: they are
allocated last, and an allocation that fails in a later call (injected on the host) takes their
memory and succeeds; the plan then projects without them."""
import pytest
import torch

from conftest import rel_l2
from test_pet_lease_gpu import _plan

pytestmark = pytest.mark.gpu
TOL = 1e-5


def _check(sm, img, fwd, bwd, sub=None, n=1):
    f = fwd if sub is None else fwd[sub::n]
    assert rel_l2(sm.forward(img, sub).cpu().numpy(), f.cpu().numpy()) < TOL
    if sub is None:
        assert rel_l2(sm.backward(fwd).cpu().numpy(), bwd.cpu().numpy()) < TOL


def test_split_takes_the_layouts_memory(cuda):
    sm, shape, n = _plan()
    img = torch.rand(shape, device=cuda) + 1
    fwd = sm.forward(img)
    bwd = sm.backward(fwd)
    assert sm._lib.gb_inject_fault(b"alloc", 1) == 0
    sm.set_n_subsets(2)  # its first allocation fails, once
    _check(sm, img, fwd, bwd, 1, 2)
    _check(sm, img, fwd, bwd)
    f = img.clone()
    sm.osem_step(f, torch.ones(1, device=cuda), None, torch.ones(shape, device=cuda), 0)
    sm2, _, _ = _plan()
    sm2.set_n_subsets(2)
    f2 = img.clone()
    sm2.osem_step(f2, torch.ones(1, device=cuda), None, torch.ones(shape, device=cuda), 0)
    assert rel_l2(f.cpu().numpy(), f2.cpu().numpy()) < TOL


def test_deterministic_image_takes_the_layouts_memory(cuda):
    sm, shape, n = _plan()
    img = torch.rand(shape, device=cuda) + 1
    fwd = sm.forward(img)
    bwd = sm.backward(fwd)
    assert sm._lib.gb_inject_fault(b"alloc", 1) == 0
    sm.set_deterministic(True)
    a, b = sm.backward(fwd), sm.backward(fwd)
    assert torch.equal(a, b) and rel_l2(a.cpu().numpy(), bwd.cpu().numpy()) < TOL
    sm.set_deterministic(False)
    _check(sm, img, fwd, bwd)


# allocations of a plan without TOF: LUT, events, ratio, image, tiles, four sort buffers and the
# sort's own, and then the layouts
@pytest.mark.parametrize("nth", [11, 12, 13, 14])
def test_plan_without_memory_for_the_layouts(nth, cuda):
    from pytomography_gb300 import _lib
    sm, shape, n = _plan()
    img = torch.rand(shape, device=cuda) + 1
    fwd = sm.forward(img)
    bwd = sm.backward(fwd)
    assert _lib.load().gb_inject_fault(b"alloc", nth) == 0
    sm2, _, _ = _plan()
    assert _lib.load().gb_inject_fault(b"alloc", 0) == 0
    _check(sm2, img, fwd, bwd)


@pytest.mark.parametrize("nth", [2, 5, 10])
def test_what_the_plan_needs_is_still_an_error(nth, cuda):
    from pytomography_gb300 import _lib
    assert _lib.load().gb_inject_fault(b"alloc", nth) == 0
    with pytest.raises(RuntimeError, match="out of memory"):
        _plan()
    _lib.load().gb_inject_fault(b"alloc", 0)
    _plan()
