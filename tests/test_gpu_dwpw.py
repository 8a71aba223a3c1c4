"""Depthwise 3x3 + 1x1 convolution as one kernel (small_b200_dwconv2d_conv2d_f32) against the oracle's two layers."""
import ctypes as C

import numpy as np
import pytest

from oracle.bindings import same_pads, shape
from smallframework_b200 import _lib
from smallframework_b200 import interface as S
from smallframework_b200 import packing as P
from smallframework_b200._lib import Layer, check, lib
from tests.gpu_util import CB, fbuf, oracle_conv_batch, rel_max_err

CASES = [
    # channels in, out, H, W, stride, images
    (16, 16, 12, 12, 1, 3),      # one channel block
    (16, 32, 24, 24, 2, 5),      # stride 2, pads (0, 1)
    (32, 32, 20, 16, 1, 150),    # more tiles than CTAs
    (64, 128, 7, 12, 1, 9),      # 128 output channels
    (128, 128, 6, 6, 1, 40),     # strips of three, several images per tile
    (128, 256, 6, 6, 2, 9),      # two channel tiles; output width 3
    (256, 256, 3, 3, 1, 50),     # two hi*hi accumulators, filter streamed
    (384, 16, 4, 4, 1, 2),       # the longest reduction covered
    (48, 144, 9, 8, 1, 4),       # a partial channel tile of 16
    (16, 48, 5, 2, 1, 7),        # images narrower than a strip
    (32, 16, 2, 1, 1, 3),
    (32, 64, 17, 37, 1, 3),      # ragged: partial tiles on both sides
    (16, 16, 45, 29, 2, 2),
    (32, 32, 48, 48, 1, 9),      # tiles of 8 x 16
    (144, 160, 6, 12, 2, 70),    # two accumulators, partial channel tile
]


def _layers(c, k, h, w, s, n):
    pads = same_pads(h, w, 3, 3, s)
    dw = Layer(n, c, c, h, w, 3, 3, s, *pads, 0, S.ACT_RELU, 0.0, 0, 0, 0, 0, 0, 0)
    ho, wo = dw.out_hw()
    return dw, Layer(n, c, k, ho, wo, 1, 1, 1, 0, 0, 0, 0, 0, S.ACT_LEAKY, 0.1, 0, 0, 0, 0, 0, 0), pads, ho, wo


@pytest.mark.gpu
@pytest.mark.parametrize("case", CASES, ids=lambda c: "C{}_K{}_{}x{}_s{}_n{}".format(*c))
@pytest.mark.parametrize("bias", [False, True])
def test_depthwise_then_pointwise_one_kernel(oracle, case, bias):
    c, k, h, w, s, n = case
    dw, pw, pads, ho, wo = _layers(*case)
    assert lib().small_b200_dwconv2d_conv2d_f32_supported(C.byref(dw), C.byref(pw))
    rng = np.random.default_rng(c + k + h)
    x = P.pack_activation(rng.uniform(-1, 1, (n, c, h, w)).astype(np.float32))
    wd = P.pack_dw_filter(rng.normal(0, 0.4, (c, 3, 3)).astype(np.float32))
    wp = P.pack_conv_filter(rng.normal(0, np.sqrt(2.0 / c), (k, c, 1, 1)).astype(np.float32))
    b1 = rng.uniform(-0.5, 0.5, c).astype(np.float32) if bias else None
    b2 = rng.uniform(-0.5, 0.5, k).astype(np.float32) if bias else None
    X, WD, WP, O = fbuf(x), fbuf(wd), fbuf(wp), S.FloatBuffer(n * k * ho * wo)
    FP, ptr = S.FloatBuffer(2 * WP.size()), lambda b: None if b is None else b.ptr()
    B1, B2 = (fbuf(b1), fbuf(b2)) if bias else (None, None)
    st = S._stream(None)
    check(lib().small_b200_filter_prepare_dwconv2d_conv2d_f32(C.byref(pw), WP.ptr(), FP.ptr(), st))
    check(lib().small_b200_dwconv2d_conv2d_f32(C.byref(dw), C.byref(pw), X.ptr(), WD.ptr(), ptr(B1), FP.ptr(), ptr(B2), O.ptr(), st))
    got = O.numpy().reshape(n, -1)
    assert _lib.device_status() == 0
    mid = oracle_conv_batch(oracle, shape(c, c, h, w, 3, 3, s, pads, CB), x, wd, bias=b1, act=1, depthwise=True)
    want = oracle_conv_batch(oracle, shape(c, k, ho, wo, 1, 1, 1, (0, 0, 0, 0), CB), mid, wp, bias=b2, act=2, slope=0.1)
    assert rel_max_err(got, want) <= 1e-5


def test_pairs_that_are_refused():
    ok = lambda d, p: bool(lib().small_b200_dwconv2d_conv2d_f32_supported(C.byref(d), C.byref(p)))
    dw, pw, *_ = _layers(32, 32, 12, 12, 1, 1)
    assert ok(dw, pw)
    dw5 = Layer(1, 32, 32, 12, 12, 5, 5, 1, 2, 2, 2, 2, 0, 0, 0.0, 0, 0, 0, 0, 0, 0)
    assert not ok(dw5, pw)                                        # another window
    assert not ok(*_layers(400, 128, 12, 12, 1, 1)[:2])           # more accumulator columns than tensor memory has
    acc = Layer(1, 32, 32, 12, 12, 1, 1, 1, 0, 0, 0, 0, 1, 0, 0.0, 0, 0, 0, 0, 0, 0)
    assert not ok(dw, acc)                                        # PartialConv2D
