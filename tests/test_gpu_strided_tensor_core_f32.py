"""The kernels that small_b200_conv2d_f32 takes for strided windows, the gathering tensor-core one and the first layer's, against
the oracle."""
import ctypes as C

import numpy as np
import pytest
import torch

from oracle.bindings import same_pads, shape
from smallframework_b200 import interface as S
from smallframework_b200 import packing as P
from smallframework_b200._lib import Layer, check, device_status, lib
from tests.gpu_util import CB, fbuf, oracle_conv_batch, rel_max_err

pytestmark = pytest.mark.gpu

CASES = [
    # C, K, H, W, Fh, Fw, stride, pads, batch
    (96, 80, 31, 29, 3, 3, 2, "same", 6),       # a last tile of 32 pixels, a second filter tile of 16 channels
    (16, 192, 64, 64, 1, 1, 2, (0, 0, 0, 0), 20),  # one step a tile: every other tile leaves an MMA warp without work
    (64, 16, 33, 35, 5, 3, 2, (4, 1, 0, 2), 4),
    (48, 48, 19, 3, 3, 3, 2, "same", 60),       # 27 steps, images shorter than a tile
    (336, 64, 9, 9, 3, 3, 2, "same", 6),        # 189 of at most 192 steps
    (368, 32, 11, 11, 3, 3, 2, "same", 6),      # 207: the other kernel
    # first layers, in blocks of 1x2 outputs
    (3, 16, 96, 96, 3, 3, 2, "same", 8),        # rows by 16-byte loads
    (3, 32, 95, 95, 3, 3, 2, (1, 1, 1, 1), 6),
    (3, 16, 97, 95, 3, 3, 2, (1, 1, 1, 1), 8),  # an odd number of rows
    (3, 16, 92, 92, 3, 3, 2, (2, 3, 0, 5), 9),  # blocks of nothing but padding
]


def run(oracle, case, bias, part, x_edit=None):
    c, k, h, w, fh, fw, s, pm, n = case
    pads = same_pads(h, w, fh, fw, s) if pm == "same" else pm
    rng = np.random.default_rng(c * k + h)
    x = rng.uniform(-1, 1, (n, c, h, w)).astype(np.float32)
    if x_edit:
        x_edit(x)
    x = P.pack_activation(x)
    wt = P.pack_conv_filter(rng.normal(0, np.sqrt(2.0 / (c * fh * fw)), (k, c, fh, fw)).astype(np.float32))
    sh = shape(c, k, h, w, fh, fw, s, pads, CB)
    ho, wo = sh.out_hw()
    seed = rng.uniform(-1, 1, (n, k * ho * wo)).astype(np.float32)
    b = rng.uniform(-0.5, 0.5, k).astype(np.float32) if bias else None
    L = Layer(n, c, k, h, w, fh, fw, s, *pads, int(part), S.ACT_LEAKY if part else 0, 0.1, 0, 0, 0, 0, 0, 0)
    assert not lib().small_b200_conv2d_f32_small_preferred(C.byref(L))
    X, W, O = fbuf(x), fbuf(wt), fbuf(seed)
    B = fbuf(b) if bias else None
    check(lib().small_b200_conv2d_f32(C.byref(L), X.ptr(), W.ptr(), B.ptr() if bias else None, O.ptr(), S._stream(None)))
    want = oracle_conv_batch(oracle, sh, x, wt, bias=b, **(dict(act=2, slope=0.1, seed=seed) if part else {}))
    assert device_status() == 0
    return O.numpy().reshape(n, -1), want


@pytest.mark.parametrize("case", CASES, ids=lambda c: "C{}_K{}_{}x{}_k{}x{}_s{}_n{}".format(*c[:7], c[8]))
@pytest.mark.parametrize("mode", ["plain", "partial_bias_leaky"])
def test_strided_convolution(oracle, case, mode):
    got, want = run(oracle, case, mode != "plain", mode != "plain")
    assert rel_max_err(got, want) <= 1e-5


# C, K, H, W, window, images: filters that stay in shared memory, of 1, 2, 3, 4 and 9 steps, and three tiles or more an SM
RESIDENT = [(16, 32, 64, 64, 1, 60), (32, 64, 49, 51, 1, 100), (48, 16, 64, 64, 1, 60), (64, 64, 40, 40, 1, 150), (16, 64, 64, 64, 3, 60)]


@pytest.mark.parametrize("case", RESIDENT, ids=lambda c: "C{}_K{}_{}x{}_k{}_n{}".format(*c))
def test_resident_filters_through_many_tiles(case):
    """Every image, against fp64, of launches whose filters differ.  With an odd number of steps a step is issued by one warp in a CTA's
    first tile and by the other in its second.  (Bound: the fp32 gate of the other tests.)"""
    c, k, h, w, f, n = case
    pads = same_pads(h, w, f, f, 2)
    rng = np.random.default_rng(c + k + f)
    ho, wo = shape(c, k, h, w, f, f, 2, pads, CB).out_hw()
    assert n * ho * wo > 3 * 148 * 128
    x = rng.uniform(-1, 1, (n, c, h, w)).astype(np.float32)
    X, O = fbuf(P.pack_activation(x)), S.FloatBuffer(n * k * ho * wo)
    L = Layer(n, c, k, h, w, f, f, 2, *pads, 0, 0, 0.1, 0, 0, 0, 0, 0, 0)
    xp = torch.nn.functional.pad(torch.from_numpy(x.astype(np.float64)), (pads[2], pads[3], pads[0], pads[1]))
    for _ in range(4):
        wt = rng.normal(0, np.sqrt(2.0 / (c * f * f)), (k, c, f, f)).astype(np.float32)
        W = fbuf(P.pack_conv_filter(wt))
        check(lib().small_b200_conv2d_f32(C.byref(L), X.ptr(), W.ptr(), None, O.ptr(), S._stream(None)))
        got = P.unpack_activation(O.numpy().reshape(n, -1), k, ho, wo)
        assert device_status() == 0
        want = torch.nn.functional.conv2d(xp, torch.from_numpy(wt.astype(np.float64)), stride=2).numpy()
        assert rel_max_err(got, want) <= 1e-5


def test_values_outside_the_words_range(oracle):
    """Infinities, NaN and values next to the largest float give what the products themselves sum to."""
    def edit(x):
        x[0, 3, 4, 4] = np.inf
        x[1, 40, 10, 7] = np.nan
        x[2, 5, 8, 8] = np.finfo(np.float32).max
    got, want = run(oracle, CASES[0], False, False, edit)
    odd = ~np.isfinite(want)
    assert odd.any() and np.array_equal(got[odd], want[odd], equal_nan=True)
    assert np.isfinite(got[~odd]).all()
    tame = np.abs(want) < 1e3
    assert rel_max_err(got[tame], want[tame]) <= 1e-5
