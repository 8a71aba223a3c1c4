"""Outputs that begin 16 bytes past a 32-byte boundary: the kernels that store 32 bytes at a time store 16 there, with the same values and nothing
beside them."""
import ctypes as C

import pytest
import torch

from oracle.bindings import same_pads
from smallframework_b200 import _lib
from smallframework_b200._lib import Layer, check, lib

pytestmark = pytest.mark.gpu


def _both(elems, dtype, run):
    """The output of run(pointer) on a 32-byte boundary and 16 bytes past one, the second with its kernel and what lies around it."""
    size = torch.empty(0, dtype=dtype).element_size()
    aligned, wide = torch.full((elems,), 77, dtype=dtype, device="cuda"), torch.full((elems + 64 // size,), 77, dtype=dtype, device="cuda")
    shift = 16 // size
    assert aligned.data_ptr() % 32 == 0 and wide.data_ptr() % 32 == 0
    run(aligned.data_ptr())
    first = _lib.last_kernel()
    run(wide.data_ptr() + 16)
    torch.cuda.synchronize()
    assert _lib.device_status() == 0
    assert bool((wide[:shift] == 77).all()) and bool((wide[shift + elems:] == 77).all())
    return aligned, wide[shift:shift + elems], first, _lib.last_kernel()


def _rand(*shape):
    return torch.randn(*shape, device="cuda", generator=torch.Generator("cuda").manual_seed(4))


def _layer(c, k, h, w, f, s, n, act=1, pads=None, **q):
    pads = same_pads(h, w, f, f, s) if pads is None else pads
    return Layer(n, c, k, h, w, f, f, s, *pads, 0, act, 0.0, q.get("zi", 0), q.get("zf", 0), 0, q.get("rs", 0), q.get("mult", 0), 0)


STREAM = lambda: torch.cuda.current_stream().cuda_stream

TENSOR_CORE = [
    # C, K, H, W, kernel, stride, images, pool, kernel's name
    (16, 16, 32, 32, 3, 1, 3, False, "conv_f16x3_kernel"), (64, 32, 20, 20, 3, 1, 9, False, "conv_f16x3_kernel"),
    (32, 64, 20, 20, 3, 1, 3, False, "conv_f16x3_kernel"), (128, 16, 26, 26, 3, 1, 4, False, "conv_f16x3_kernel"),
    (16, 32, 80, 80, 3, 1, 2, True, "conv_f16x3_kernel"), (32, 64, 80, 80, 3, 1, 2, True, "conv_f16x3_kernel"),
    (48, 64, 29, 31, 3, 2, 4, False, "conv_gather_f32_kernel"),
]


@pytest.mark.parametrize("case", TENSOR_CORE, ids=lambda c: "C{}_K{}_{}x{}_k{}_s{}_n{}{}".format(*c[:7], "_pool" if c[7] else ""))
def test_fp32_tensor_core_convolutions(case):
    c, k, h, w, f, s, n, pool, name = case
    L, P = _layer(c, k, h, w, f, s, n), _layer(k, k, h, w, 2, 2, n, 0, (0, 0, 0, 0))
    x, filt, bias = _rand(n * c * h * w), _rand(k * c * f * f), _rand(k)
    prepared = torch.empty(2 * filt.numel(), device="cuda")
    if s == 1:
        check(lib().small_b200_filter_prepare_tf32x3(C.byref(L), filt.data_ptr(), prepared.data_ptr(), STREAM()))
    ho, wo = (P if pool else L).out_hw()

    def run(out):
        if pool:
            check(lib().small_b200_conv2d_maxpool_f32_tf32x3(C.byref(L), C.byref(P), x.data_ptr(), prepared.data_ptr(), bias.data_ptr(), out, STREAM()))
        elif s == 2:
            check(lib().small_b200_conv2d_f32(C.byref(L), x.data_ptr(), filt.data_ptr(), bias.data_ptr(), out, STREAM()))
        else:
            check(lib().small_b200_conv2d_f32_tf32x3(C.byref(L), x.data_ptr(), prepared.data_ptr(), bias.data_ptr(), out, STREAM()))

    a, b, ka, kb = _both(n * k * ho * wo, torch.float32, run)
    assert torch.equal(a, b) and float(a.abs().max()) > 0 and ka == kb == name


def test_fp32_first_layer_with_its_pool():
    L, P = _layer(3, 16, 64, 64, 3, 1, 4), _layer(16, 16, 64, 64, 2, 2, 4, 0, (0, 0, 0, 0))
    x, filt, bias = _rand(4 * 3 * 64 * 64), _rand(16 * 27), _rand(16)
    assert lib().small_b200_conv2d_maxpool_f32_supported(C.byref(L), C.byref(P))
    run = lambda out: check(lib().small_b200_conv2d_maxpool_f32(C.byref(L), C.byref(P), x.data_ptr(), filt.data_ptr(), bias.data_ptr(), out, STREAM()))
    a, b, ka, kb = _both(4 * 16 * 32 * 32, torch.float32, run)
    assert torch.equal(a, b) and float(a.abs().max()) > 0 and ka == kb


@pytest.mark.parametrize("c,k", [(16, 16), (64, 64)])
def test_fp32_separable_blocks(c, k):
    """16 channels: the kernel on the FMA pipe stores 32 bytes only, other outputs are the tensor cores'."""
    D, L = _layer(c, c, 24, 24, 3, 1, 8), _layer(c, k, 24, 24, 1, 1, 8)
    x, dw, pw, b1, b2 = _rand(8 * c * 576), _rand(c * 9), _rand(c * k), _rand(c), _rand(k)
    prepared = torch.empty(2 * pw.numel(), device="cuda")
    check(lib().small_b200_filter_prepare_dwconv2d_conv2d_f32(C.byref(L), pw.data_ptr(), prepared.data_ptr(), STREAM()))
    run = lambda out: check(lib().small_b200_dwconv2d_conv2d_f32(C.byref(D), C.byref(L), x.data_ptr(), dw.data_ptr(), b1.data_ptr(),
                                                                 prepared.data_ptr(), b2.data_ptr(), out, STREAM()))
    a, b, ka, kb = _both(8 * k * 576, torch.float32, run)
    assert kb == "dwpw_f32_kernel" and ka == ("dwpw_direct_f32_kernel" if c == 16 else kb)
    if ka == kb:
        assert torch.equal(a, b)
    # sums of 16 products in fp32 and in pairs of tf32 words (2^-21 of a product)
    assert float((a - b).abs().max()) <= 1e-5 * float(a.abs().max())


@pytest.mark.parametrize("size,s", [(96, 2), (64, 1), (65, 1)])
def test_uint8_first_layer_on_three_channels(size, s):
    n = -(-210000 // (size // s) ** 2)
    L = _layer(3, 32, size, size, 3, s, n, zi=-113, zf=-121, rs=8, mult=1 << 30)
    gen = torch.Generator("cuda").manual_seed(4)
    byte = lambda e: torch.randint(0, 256, (e,), dtype=torch.uint8, device="cuda", generator=gen)
    x, filt = byte(n * 3 * size * size), byte(32 * 27)
    ho, wo = L.out_hw()
    run = lambda out: check(lib().small_b200_conv2d_u8(C.byref(L), x.data_ptr(), filt.data_ptr(), None, out, STREAM()))
    a, b, ka, kb = _both(n * 32 * ho * wo, torch.uint8, run)
    assert torch.equal(a, b) and int(a.max()) > int(a.min()) and ka == kb == "conv_u8_rgb_kernel"
