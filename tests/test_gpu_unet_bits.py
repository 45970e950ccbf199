"""The learned denoiser's sums in their recorded order, bit for bit.

A convolution's fp32 sum depends on its order in the last place, and a network amplifies that: one flipped bf16
rounding or ReLU mask in an early layer moves a training step's gradient by several per cent, which is as far as it is
from its 64-bit value.  So the order is part of the results: whichever kernel takes a shape adds the same products in
the same order.  The digests below are of results recorded on a B200 (148 SMs, which fixes the number of
partial sums) with the kernels that defined the order."""
import ctypes
import hashlib

import numpy as np
import pytest
import torch

from cloudrendering_b200 import _lib
from cloudrendering_b200 import learned_denoiser as ld
from oracle import unet_oracle as uo

pytestmark = pytest.mark.gpu


def ptr(t):
    return ctypes.c_void_p(t.data_ptr()) if t is not None else None


def normal(seed, *shape, scale=1.0):
    return (np.random.default_rng(seed).standard_normal(shape) * scale).astype(np.float32)


def f32(a):
    return torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda()


def bf16(a):
    return torch.from_numpy(uo.bf16(np.asarray(a, np.float32))).to(torch.bfloat16).cuda().contiguous()


def digest(*tensors):
    h = hashlib.sha256()
    for t in tensors:
        h.update((t.float() + 0.0).contiguous().cpu().numpy().tobytes())  # (+ 0: -0 and 0 are one value)
    return h.hexdigest()[:16]


def call(lib, name, *args):
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    assert getattr(lib, name)(*args, ptr(err), None) == 0, name
    torch.cuda.synchronize()
    assert int(err.item()) == 0, name


# ---- the kernel head ----
def head_digest(lib, n, h, w, ks):
    hc = (ks * ks + 7) // 8 * 8
    g = np.random.default_rng(40)
    rad = f32(g.exponential(1.0, (n, 3, h, w)) * (g.random((n, 3, h, w)) < 0.7))
    target = f32(g.exponential(1.0, (n, 3, h, w)))
    logits = f32(normal(41, n, h, w, hc, scale=2.0))
    out = torch.empty((n, 3, h, w), device="cuda")
    dl = torch.empty((n, h, w, hc), dtype=torch.bfloat16, device="cuda")
    lp = torch.empty(lib.vpt_unet_head_blocks(n, h, w), device="cuda")
    assert lib.vpt_unet_kpn_head(ptr(logits), hc, ks, ptr(rad), ptr(target), ptr(out), ptr(dl), ptr(lp), n, h, w,
                                 ctypes.c_float(1e-2), None) == 0
    torch.cuda.synchronize()
    return digest(out, dl)


# ---- convolutions: forward (bias, fp32) and input gradient (mask) ----
def conv_digest(lib, n, h, w, cin, cout):
    x, dy = bf16(normal(51, n, h, w, cin)), bf16(normal(52, n, h, w, cout))
    wt, b = bf16(normal(53, cout, 9, cin, scale=1.0 / np.sqrt(9 * cin))), f32(normal(54, cout, scale=0.1))
    y = torch.empty((n, h, w, cout), device="cuda")
    call(lib, "vpt_unet_conv3x3", ptr(x), ptr(wt), ptr(b), None, ptr(y), n, h, w, cin, cout, 0, 1)
    wrot = torch.empty((cin, 9, cout), dtype=torch.bfloat16, device="cuda")
    assert lib.vpt_unet_rotate_weights(ptr(wt), ptr(wrot), cin, cout, None) == 0
    dx = torch.empty((n, h, w, cin), device="cuda")
    call(lib, "vpt_unet_conv3x3", ptr(dy), ptr(wrot), None, ptr(x), ptr(dx), n, h, w, cout, cin, 0, 1)
    return digest(y, dx)


# ---- weight gradients ----
def split_pixels(lib, pixels, cin):
    """The training loop's pixels per split."""
    tiles = lib.vpt_unet_wgrad_rows(cin) // 128
    splits = max(1, min((pixels + 63) // 64, (2 * 148 + tiles - 1) // tiles))
    return ((pixels + splits - 1) // splits + 63) // 64 * 64


def wgrad_digest(lib, n, h, w, cin, cout):
    x, dy = bf16(normal(61, n, h, w, cin)), bf16(normal(62, n, h, w, cout))
    pps = split_pixels(lib, n * h * w, cin)
    splits, rows = lib.vpt_unet_wgrad_splits(n, h, w, cin, cout, pps), lib.vpt_unet_wgrad_rows(cin)
    part = torch.zeros((splits, rows, cout), device="cuda")
    call(lib, "vpt_unet_conv3x3_wgrad", ptr(x), ptr(dy), ptr(part), n, h, w, cin, cout, pps)
    return digest(part[:, :9 * cin])


# ---- training steps ----
def train_digest(lib, n, h, w):
    g = np.random.default_rng(70)
    net = ld.KpnUNet(seed=5)
    scene = 0.5 + 0.4 * np.sin(np.arange(w)[None, None, None] / 9.0 + np.arange(h)[None, None, :, None] / 13.0)
    batch = dict(radiance=scene * g.exponential(1.0, (n, 3, h, w)), target=np.broadcast_to(scene, (n, 3, h, w)),
                 albedo=g.random((n, 3, h, w)), normal=g.standard_normal((n, 3, h, w)), depth=g.random((n, h, w)),
                 transmittance=g.random((n, h, w)), noise_level=np.full(n, 0.5))
    batch = {k: f32(v) for k, v in batch.items()}
    for _ in range(2):
        net.train_step(batch, 1e-4)
    net.check_errors()
    return digest(net.grad, net.param, *net.logits)


COMPUTE = {"head": head_digest, "conv": conv_digest, "wgrad": wgrad_digest, "train": train_digest}
# (what, sizes): the digest
RECORDED = {
    ("head", 2, 9, 130, 13): "43e0284da028c99d",
    ("head", 1, 33, 70, 5): "96607ab2ed513255",
    ("head", 1, 6, 64, 15): "0a8f679207c8b013",
    ("wgrad", 8, 96, 256, 96, 32): "a0dcfe46e0ade327",
    ("wgrad", 2, 80, 224, 96, 32): "68d25f01401e2d07",
    ("wgrad", 1, 37, 130, 64, 64): "1b001b1a681183d3",
    ("wgrad", 1, 64, 128, 160, 64): "d4636b2e89e0de43",
    ("wgrad", 2, 50, 200, 32, 176): "3f2207bf578b20f5",
    ("wgrad", 2, 64, 256, 32, 32): "ff406f1095b659ae",
    ("wgrad", 1, 96, 150, 16, 32): "297b0026b330b4d6",
    ("wgrad", 4, 40, 112, 64, 64): "5af21771fd023618",
    ("wgrad", 8, 32, 32, 128, 128): "1a14c8b49fae70ea",
    ("conv", 2, 80, 224, 96, 32): "045841120c058184",
    ("conv", 4, 64, 256, 32, 176): "d8dffbe203856862",
    ("conv", 1, 64, 128, 96, 32): "552c9e589121c6f3",
    ("conv", 1, 200, 128, 96, 32): "664d0fc73bc91969",
    ("conv", 8, 128, 128, 160, 64): "992ae3ff36a47072",
    ("conv", 1, 40, 128, 160, 64): "d7316fae95089f40",
    ("conv", 2, 40, 128, 176, 32): "1a95d6f0b52d491c",
    ("conv", 2, 128, 256, 48, 48): "c56e0299a6be8a97",
    ("conv", 1, 70, 128, 48, 48): "def1d5a670812b25",
    ("conv", 2, 128, 128, 96, 96): "d2ed80b7fc5fef4b",
    ("conv", 4, 128, 256, 96, 96): "660af0682e04cd93",
    ("conv", 2, 256, 128, 224, 96): "73aee32fff885770",
    ("conv", 1, 90, 150, 112, 80): "17c51028e31a1aef",
    ("conv", 1, 60, 130, 272, 64): "ffaaad767f8c14b0",
    ("conv", 2, 512, 128, 32, 112): "752103d811e0d68c",
    ("conv", 1, 16, 16, 160, 160): "374f6b27e502437f",
    ("conv", 2, 16, 16, 288, 128): "c9e7bb8999ac40ae",
    ("conv", 8, 16, 16, 128, 160): "0a24f18ddbb0f591",
    ("conv", 2, 32, 32, 96, 128): "e15f52e99f00e947",
    ("conv", 1, 64, 64, 224, 96): "8229df357683fc6a",
    ("conv", 2, 64, 64, 48, 96): "3d998bb577afc99f",
    ("conv", 8, 64, 64, 96, 96): "d75ce6e4cc6f08aa",
    ("conv", 1, 28, 56, 96, 96): "ffe6c21e8c7caf55",
    ("conv", 1, 4, 4, 128, 160): "b08638116ed22ef2",
    ("conv", 3, 8, 8, 16, 272): "25462c92d966b521",
    ("train", 2, 80, 224): "91b0c6a78fa4ca6d",
    ("train", 3, 64, 96): "757e0ae5ac3a2b1f",
    ("train", 2, 256, 256): "45c2496e8e506686",
    ("train", 1, 192, 512): "988742b8fbf7da8f",
}


@pytest.fixture(scope="module")
def lib():
    torch.cuda.init()
    return _lib.load()


@pytest.mark.parametrize("key", RECORDED, ids=lambda k: "-".join(map(str, k)))
def test_results_as_recorded(lib, key):
    assert COMPUTE[key[0]](lib, *key[1:]) == RECORDED[key]
