"""Depthwise-separable blocks of few channels on the FMA pipe (csrc/dwpw_direct_f32.cu) against the oracle's two layers: rows cut
into parts, ragged last strips and tiles, images of a pixel, both strides, 16 and 32 channels; infinities come out as the layers'."""
import ctypes as C

import numpy as np
import pytest

from oracle.bindings import same_pads, shape
from smallframework_b200 import _lib
from smallframework_b200 import interface as S
from smallframework_b200 import packing as P
from smallframework_b200._lib import Layer, check, lib
from tests.gpu_util import CB, fbuf, oracle_conv_batch, rel_max_err

pytestmark = pytest.mark.gpu

CASES = [
    # C, K, H, W, stride, pads, images
    (16, 16, 48, 48, 1, "same", 3), (16, 16, 5, 130, 1, "same", 2), (16, 16, 45, 65, 1, "same", 2), (16, 32, 13, 7, 1, "same", 5),
    (16, 16, 1, 1, 1, "same", 9), (16, 16, 200, 3, 1, "same", 2), (32, 32, 33, 37, 1, "same", 15), (32, 16, 129, 130, 1, "same", 1),
    (16, 32, 48, 48, 2, "same", 3), (16, 32, 51, 133, 2, "same", 2), (16, 32, 9, 64, 2, (1, 1, 1, 1), 4), (16, 16, 20, 20, 1, (0, 0, 0, 0), 3),
]


def _run(oracle, case, x, wd, wp, b1, b2):
    c, k, h, w, s, pm, n = case
    pads = same_pads(h, w, 3, 3, s) if pm == "same" else pm
    dw = Layer(n, c, c, h, w, 3, 3, s, *pads, 0, S.ACT_LEAKY, 0.2, 0, 0, 0, 0, 0, 0)
    ho, wo = dw.out_hw()
    pw = Layer(n, c, k, ho, wo, 1, 1, 1, 0, 0, 0, 0, 0, S.ACT_LEAKY, 0.1, 0, 0, 0, 0, 0, 0)
    X, WD, WP, O = fbuf(P.pack_activation(x)), fbuf(P.pack_dw_filter(wd)), fbuf(P.pack_conv_filter(wp)), S.FloatBuffer(n * k * ho * wo)
    FP, B1, B2 = S.FloatBuffer(2 * WP.size()), fbuf(b1), fbuf(b2)
    st = S._stream(None)
    check(lib().small_b200_filter_prepare_dwconv2d_conv2d_f32(C.byref(pw), WP.ptr(), FP.ptr(), st))
    check(lib().small_b200_dwconv2d_conv2d_f32(C.byref(dw), C.byref(pw), X.ptr(), WD.ptr(), B1.ptr(), FP.ptr(), B2.ptr(), O.ptr(), st))
    got = O.numpy().reshape(n, -1)
    assert _lib.device_status() == 0
    mid = oracle_conv_batch(oracle, shape(c, c, h, w, 3, 3, s, pads, CB), P.pack_activation(x), P.pack_dw_filter(wd), bias=b1, act=2, slope=0.2,
                            depthwise=True)
    return got, oracle_conv_batch(oracle, shape(c, k, ho, wo, 1, 1, 1, (0, 0, 0, 0), CB), mid, P.pack_conv_filter(wp), bias=b2, act=2, slope=0.1)


def _operands(case):
    c, k, h, w, s, pm, n = case
    rng = np.random.default_rng(c + k + h + w)
    f = lambda *a: a[-1].astype(np.float32)
    return (f(rng.uniform(-1, 1, (n, c, h, w))), f(rng.normal(0, 0.4, (c, 3, 3))), f(rng.normal(0, np.sqrt(2.0 / c), (k, c, 1, 1))),
            f(rng.uniform(-0.5, 0.5, c)), f(rng.uniform(-0.5, 0.5, k)))


@pytest.mark.parametrize("case", CASES, ids=lambda c: "C{}_K{}_{}x{}_s{}_{}_n{}".format(*c[:5], "".join(map(str, c[5])), c[6]))
def test_against_the_two_layers(oracle, case):
    got, want = _run(oracle, case, *_operands(case))
    assert rel_max_err(got, want) <= 1e-6  # two fp32 sums of 9 and at most 32 products in the same precision


LINES = [
    # to either side of the lines between the two kernels
    (32, 16, 18, 5, 1, "same", 200, "dwpw_f32_kernel"), (32, 16, 24, 24, 1, "same", 30, "dwpw_direct_f32_kernel"),
    (32, 32, 126, 5, 1, "same", 40, "dwpw_direct_f32_kernel"), (32, 32, 5, 126, 1, "same", 40, "dwpw_f32_kernel"),
    (16, 32, 12, 13, 2, "same", 1, "dwpw_direct_f32_kernel"), (16, 32, 12, 11, 2, "same", 1, "dwpw_f32_kernel"),
]


@pytest.mark.parametrize("case", LINES, ids=lambda c: "C{}_K{}_{}x{}_s{}_{}_n{}".format(*c[:7]))
def test_which_kernel(oracle, case):
    got, want = _run(oracle, case[:7], *_operands(case[:7]))
    assert _lib.last_kernel() == case[7]
    assert rel_max_err(got, want) <= (1e-6 if "direct" in case[7] else 1e-5)  # as above; pairs of tf32 words, 2^-21 of a product


@pytest.mark.parametrize("value", [np.inf, np.nan, 1e38], ids=str)
def test_values_without_a_finite_sum(oracle, value):
    case = CASES[0]
    x, wd, wp, b1, b2 = _operands(case)
    x[1, 3, 20:22, 20] = value
    wd, wp = np.abs(wd) + 0.1, np.abs(wp) + (100 if value == 1e38 else 0.1)  # infinities of one sign
    got, want = _run(oracle, case, x, wd, wp, b1, b2)
    assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(np.isinf(got), np.isinf(want))
    assert not np.isfinite(want).all()
    fin = np.isfinite(want)
    assert rel_max_err(got[fin], want[fin]) <= 1e-6
