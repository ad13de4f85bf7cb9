"""The patch layout of a listmode plan is lent to one call at a time also when equal stream
handles name different streams: two host threads on the per-thread default stream, and a stream
created after another was destroyed."""
import ctypes
import threading

import numpy as np
import pytest
import torch

from conftest import rel_l2

pytestmark = pytest.mark.gpu
PER_THREAD = 2  # cudaStreamPerThread
TOL = 1e-5      # the order of the back projection's additions differs


def _plan():
    from pytomography_gb300.metadata import ObjectMeta
    from pytomography_gb300.metadata.PET import PETLMProjMeta
    from pytomography_gb300.projectors.PET import PETLMSystemMatrix
    nt, nr, n, shape = 64, 16, 300_000, (80, 80, 32)
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
    sm = PETLMSystemMatrix(ObjectMeta([2.5] * 3, shape),
                           PETLMProjMeta(pairs, info=info,
                                         detector_ids_sensitivity=pairs[:100].clone()))
    return sm, shape, n


def _run(sm, imgs, projs, fwd, bwd, stream):
    from pytomography_gb300 import _lib
    for x, y, a, b in zip(imgs, projs, fwd, bwd):
        _lib.check(sm._lib.gb_pet_forward(sm._plan, _lib.ptr(x), _lib.ptr(a), -1, stream))
        _lib.check(sm._lib.gb_pet_backward(sm._plan, _lib.ptr(y), _lib.ptr(b), -1, stream))


def test_two_threads_on_the_per_thread_stream(cuda):
    sm, shape, n = _plan()
    imgs = [torch.rand(shape, device=cuda) + k for k in range(12)]
    want = [sm.forward(x) for x in imgs]
    back = [sm.backward(y) for y in want]
    fwd = [torch.zeros(n, device=cuda) for _ in imgs]
    bwd = [torch.zeros(shape, device=cuda) for _ in imgs]
    torch.cuda.synchronize()
    th = [threading.Thread(target=_run, args=(sm, imgs[k::2], want[k::2], fwd[k::2], bwd[k::2],
                                              ctypes.c_void_p(PER_THREAD))) for k in range(2)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    torch.cuda.synchronize()
    for a, b in zip(fwd + bwd, want + back):
        assert rel_l2(a.cpu().numpy(), b.cpu().numpy()) < TOL


def test_stream_created_after_another_was_destroyed(cuda):
    sm, shape, n = _plan()
    rt = ctypes.CDLL("libcudart.so.13")
    imgs = [torch.rand(shape, device=cuda) + k for k in range(12)]
    want = [sm.forward(x) for x in imgs]
    back = [sm.backward(y) for y in want]
    fwd = [torch.zeros(n, device=cuda) for _ in imgs]
    bwd = [torch.zeros(shape, device=cuda) for _ in imgs]
    torch.cuda.synchronize()
    for k in range(len(imgs)):
        st = ctypes.c_void_p()
        assert rt.cudaStreamCreateWithFlags(ctypes.byref(st), 1) == 0
        _run(sm, imgs[k:k + 1], want[k:k + 1], fwd[k:k + 1], bwd[k:k + 1], st)
        assert rt.cudaStreamDestroy(st) == 0  # its work goes on
    torch.cuda.synchronize()
    for a, b in zip(fwd + bwd, want + back):
        assert rel_l2(a.cpu().numpy(), b.cpu().numpy()) < TOL
