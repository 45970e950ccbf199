"""The scratch that the stateless entry points keep between calls (csrc/vpt_scratch.cu): calls from several threads
on streams of their own do not disturb one another, what is kept is bounded, and a destroyed context gives it back."""
import ctypes
import threading

import numpy as np
import pytest
import torch

from cloudrendering_b200 import _lib
from cloudrendering_b200._lib import VptSparseInfo
from tests.harness import Core

pytestmark = pytest.mark.gpu

KEPT = 256 << 20  # bytes a device's pool may hold across synchronisations
SLACK = 64 << 20  # the driver's own granularity (32 MiB blocks) and what a context's first launches load


def eaw(lib, color, out, stream):
    h, w = color.shape[:2]
    st = lib.vpt_eaw_denoise_rgba(ctypes.c_void_p(color.data_ptr()), None, None, w, h, 3, 5.0, 0.1, 0.1, 0,
                                  ctypes.c_void_p(out.data_ptr()), ctypes.c_void_p(stream.cuda_stream))
    assert st == 0


def test_threads_and_streams_share_the_pool():
    lib = _lib.load()
    g = torch.Generator().manual_seed(5)
    sizes = [(64, 96), (1, 1), (333, 257), (720, 1280)]
    images = [torch.rand((h, w, 4), generator=g).cuda() for h, w in sizes]
    want = []
    for c in images:
        out = torch.empty_like(c)
        eaw(lib, c, out, torch.cuda.current_stream())
        torch.cuda.synchronize()
        want.append(out)
    got = [[torch.full_like(c, float("nan")) for c in images] for _ in range(4)]
    torch.cuda.synchronize()
    errors = []

    def work(outs, shift):
        try:
            torch.cuda.set_device(0)
            stream = torch.cuda.Stream()
            for rep in range(8):
                for k in range(len(images)):
                    i = (k + shift) % len(images)
                    eaw(lib, images[i], outs[i], stream)
                if rep % 3 == shift % 3:
                    stream.synchronize()  # what is free may be given back here
            stream.synchronize()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(got[i], i)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    torch.cuda.synchronize()
    for outs in got:
        for a, b in zip(outs, want):
            assert torch.equal(a, b)


@pytest.mark.parametrize("size", [(3000, 3000), (3000, 8000)], ids=["below_the_bound", "above_the_bound"])
def test_kept_scratch_is_bounded_and_given_back(size):
    lib = _lib.load()
    c = torch.rand(size + (4,), device="cuda")
    out = torch.empty_like(c)
    ctx = ctypes.c_void_p()
    assert lib.vpt_create(ctypes.byref(ctx), 0) == 0
    eaw(lib, c, out, torch.cuda.current_stream())  # loads the kernels
    torch.cuda.synchronize()
    lib.vpt_destroy(ctx)
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    assert lib.vpt_create(ctypes.byref(ctx), 0) == 0
    eaw(lib, c, out, torch.cuda.current_stream())
    torch.cuda.synchronize()
    held = free0 - torch.cuda.mem_get_info()[0]
    assert held <= KEPT + SLACK
    if size[0] * size[1] * 16 <= KEPT:  # the image is kept across the synchronisation ...
        assert held >= size[0] * size[1] * 16
        assert lib.vpt_release_scratch() == 0  # ... until it is asked for
        assert free0 - torch.cuda.mem_get_info()[0] <= SLACK
        eaw(lib, c, out, torch.cuda.current_stream())
        torch.cuda.synchronize()
        assert free0 - torch.cuda.mem_get_info()[0] >= size[0] * size[1] * 16
    lib.vpt_destroy(ctx)
    assert free0 - torch.cuda.mem_get_info()[0] <= SLACK  # less than the image


def test_allocations_take_the_kept_scratch():
    """With the device's memory used up, an allocation of a context finds the memory that the scratch keeps."""
    lib = _lib.load()
    core = Core()
    n = 192
    grid = np.random.default_rng(3).random((n, n, n), np.float32)
    core("vpt_set_dense_grid", grid.ctypes.data_as(ctypes.c_void_p), n, n, n, 0)

    def sparse(on):
        core("vpt_set_use_sparse_grid", on)
        info = VptSparseInfo()
        if on:
            core("vpt_get_sparse_grid_info", ctypes.byref(info))
        return info.leaves

    leaves = sparse(1)  # loads the kernels
    assert leaves * 2048 > 24 << 20  # bytes of values
    sparse(0)
    core("vpt_set_dense_grid", grid.ctypes.data_as(ctypes.c_void_p), n, n, n, 0)  # drops the sparse copy
    c = torch.rand((3000, 3000, 4), device="cuda")
    out = torch.empty_like(c)
    eaw(lib, c, out, torch.cuda.current_stream())
    torch.cuda.synchronize()
    hog = torch.empty(torch.cuda.mem_get_info()[0] - (16 << 20), dtype=torch.uint8, device="cuda")
    try:
        assert torch.cuda.mem_get_info()[0] <= 20 << 20
        assert sparse(1) == leaves
    finally:
        del hog
        torch.cuda.empty_cache()
        core.close()
