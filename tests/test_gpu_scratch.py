"""The scratch that the stateless entry points keep between calls (csrc/vpt_scratch.cu): calls from several threads
on streams of their own do not disturb one another, what is kept is bounded, and a destroyed context gives it back."""
import ctypes
import threading

import pytest
import torch

from cloudrendering_b200 import _lib

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


@pytest.mark.parametrize("size", [(720, 1280), (3000, 8000)], ids=["below_the_bound", "above_the_bound"])
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
    assert free0 - torch.cuda.mem_get_info()[0] <= KEPT + SLACK
    lib.vpt_destroy(ctx)
    assert free0 - torch.cuda.mem_get_info()[0] <= SLACK
