"""uint8 kernels that work on tiles of several images or planes, at the edges of their tiles: bit-exact against the oracle."""
import numpy as np
import pytest

from oracle.bindings import Quant, same_pads, shape
from smallframework_b200 import _lib
from smallframework_b200 import interface as S
from smallframework_b200 import packing as P
from tests.gpu_util import CB, qbuf
from tests.test_gpu_uint8 import _out, _quant

pytestmark = pytest.mark.gpu

DW_CASES = [
    # C, H, W, pads (None: same), batch
    (32, 3, 3, None, 70),                # whole planes, an odd number of rows, a last CTA that is not full
    (128, 6, 6, None, 40),
    (16, 48, 48, None, 3),               # runs of rows
    (48, 45, 37, None, 2),               # a short last run with an odd number of rows, a last strip that is not full
    (16, 1, 1, None, 5),
    (16, 2, 300, None, 1),
    (16, 9, 7, (0, 0, 0, 0), 2),
    (16, 5, 6, (2, 4, 3, 1), 2),         # rows and columns of nothing but padding
]


@pytest.mark.parametrize("case", DW_CASES, ids=lambda c: "C{}_{}x{}_p{}_n{}".format(*c))
@pytest.mark.parametrize("zp", [(0, -128), (-128, -128), (-113, -121), (-255, -250), (3, -7)], ids=lambda z: "zi{}_zf{}".format(*z))
def test_depthwise_3x3_tiles(oracle, case, zp):
    import torch
    C, H, W, pads, N = case
    pads = pads or same_pads(H, W, 3, 3, 1)
    rng = np.random.default_rng(C * H + W + zp[0] + 1000)
    q = _quant(rng, 9, zp)
    x = P.pack_activation(rng.integers(0, 256, (N, C, H, W)).astype(np.uint8))
    w = P.pack_dw_filter(rng.integers(0, 256, (C, 3, 3)).astype(np.uint8))
    bias = rng.integers(-4096, 4097, C).astype(np.int32)
    sh = shape(C, C, H, W, 3, 3, 1, pads, CB)
    ho, wo = sh.out_hw()
    I, F, O = qbuf(x, zp[0]), qbuf(w, zp[1]), _out(N * C * ho * wo, q)
    S.DepthwiseConv2D_Bias_Activation(3, 3, 1, *pads, C, H, W, I, F, torch.from_numpy(bias).cuda(), O, batch=N)
    want = np.stack([oracle.conv2d_u8(sh, q, x[n], w, bias=bias, depthwise=True) for n in range(N)])
    assert _lib.device_status() == 0
    assert np.array_equal(O.numpy().reshape(N, -1), want)
    assert want.min() < want.max()


# rows that do not fit a tile as a whole: a last piece of one strip, of few columns and of one; runs of rows with an odd
# one at the end; a single row; columns of nothing but padding; the widest
WIDE_CASES = [
    (16, 37, 416, None, 2), (16, 5, 700, None, 1), (48, 34, 1001, None, 1), (16, 1, 900, None, 2), (16, 9, 511, (0, 0, 0, 0), 2),
    (32, 6, 640, (2, 4, 3, 1), 1), (2048, 3, 190, None, 1), (16, 3, 5003, None, 1),
]


@pytest.mark.parametrize("case", WIDE_CASES, ids=lambda c: "C{}_{}x{}_p{}_n{}".format(*c))
@pytest.mark.parametrize("zp", [(0, -128), (-113, -121), (-255, -250)], ids=lambda z: "zi{}_zf{}".format(*z))
def test_depthwise_3x3_tiles_of_wide_images(oracle, case, zp):
    test_depthwise_3x3_tiles(oracle, case, zp)


@pytest.mark.parametrize("zp", [(-128, -128), (-113, -121)], ids=lambda z: "zi{}_zf{}".format(*z))
def test_depthwise_3x3_of_wide_images_is_as_fast_as_of_narrow_ones(zp):
    """A pixel of a row that does not fit a tile takes no longer than one of a row that does (0.9 of its time; 2.1 to 2.3
    on the kernel for any window): half as long again is left for the clock."""
    import torch

    def us(W):
        C, H, N = 16, 416, 64
        x = qbuf(np.random.default_rng(W).integers(0, 256, N * C * H * W), zp[0])
        w, o = qbuf(np.arange(C * 9) % 256, zp[1]), _out(N * C * H * W, Quant(*zp, 0, 8, 1 << 30, 0))
        ev = [torch.cuda.Event(enable_timing=True) for _ in range(7)]
        for e in ev:
            for _ in range(10):
                S.DepthwiseConv2D(3, 3, 1, 1, 1, 1, 1, C, H, W, x, w, o, batch=N)
            e.record()
        torch.cuda.synchronize()
        return min(a.elapsed_time(b) for a, b in zip(ev, ev[1:])) / W

    assert us(416) <= 1.5 * us(368)


@pytest.mark.parametrize("case", [(32, 16, 8, 8, 5), (256, 256, 3, 3, 31), (64, 128, 6, 6, 8), (128, 32, 1, 2, 130), (96, 48, 5, 13, 4),
                                  (32, 64, 12, 12, 17), (64, 32, 24, 24, 3), (32, 16, 3, 43, 140)],
                         ids=lambda c: "C{}_K{}_{}x{}_n{}".format(*c))
@pytest.mark.parametrize("zp", [(0, -128), (-113, -121)], ids=lambda z: "zi{}_zf{}".format(*z))
def test_pointwise_tiles_of_several_images(oracle, case, zp):
    C, K, H, W, N = case
    rng = np.random.default_rng(C + K + N)
    q = _quant(rng, C, zp)
    x = P.pack_activation(rng.integers(0, 256, (N, C, H, W)).astype(np.uint8))
    w = P.pack_conv_filter(rng.integers(0, 256, (K, C, 1, 1)).astype(np.uint8))
    sh = shape(C, K, H, W, 1, 1, 1, (0, 0, 0, 0), CB)
    I, F, O = qbuf(x, zp[0]), qbuf(w, zp[1]), _out(N * K * H * W, q)
    S.Conv2D(1, 1, 1, 0, 0, 0, 0, K, C, H, W, I, F, O, batch=N, path="tensor_core")
    want = np.stack([oracle.conv2d_u8(sh, q, x[n], w) for n in range(N)])
    assert _lib.device_status() == 0
    assert np.array_equal(O.numpy().reshape(N, -1), want)
    assert want.min() < want.max()


@pytest.mark.parametrize("hw", [(1, 1), (8, 8), (5, 13), (16, 16), (1, 257)], ids=lambda s: "{}x{}".format(*s))
def test_global_average_pool_sizes(oracle, hw):
    H, W = hw
    C, N = 48, 7
    rng = np.random.default_rng(H * W)
    x = rng.integers(0, 256, (N, C, H, W)).astype(np.uint8)
    x[0] = 255                           # the largest sum
    x = P.pack_activation(x)
    rshift = int(np.floor(np.log2(H * W)))
    q = Quant(0, 0, 0, rshift, min(int(2.0 ** (31 + rshift) / (H * W) * 0.99), (1 << 31) - 1), 0)
    sh = shape(C, C, H, W, H, W, 1, (0, 0, 0, 0), CB)
    I, O = qbuf(x, 0), _out(N * C, q)
    S.AveragePool2D(H, W, 1, 0, 0, 0, 0, C, H, W, I, O, batch=N)
    want = np.stack([oracle.pool2d_u8(sh, q, x[n], average=True) for n in range(N)])
    assert np.array_equal(O.numpy().reshape(N, -1), want)


@pytest.mark.parametrize("case", [
    # C, K, H, W, Fh, Fw, stride, pads, batch
    (16, 32, 24, 24, 1, 1, 1, (0, 0, 0, 0), 3),
    (16, 128, 9, 9, 1, 1, 2, (1, 1, 1, 1), 2),
    (16, 16, 300, 300, 1, 1, 1, (0, 0, 0, 0), 2),   # two pixels a thread, the last ones past the end
    (32, 16, 7, 5, 1, 1, 1, (0, 0, 0, 0), 3),
    (3, 16, 15, 17, 3, 3, 1, (1, 1, 1, 1), 3),
    (3, 16, 400, 401, 3, 3, 2, (2, 3, 2, 3), 2),    # windows of nothing but padding
    (2, 32, 11, 9, 3, 4, 1, (3, 0, 0, 3), 2),
], ids=lambda c: "C{}_K{}_{}x{}_k{}x{}_s{}_p{}_n{}".format(*c))
@pytest.mark.parametrize("zp", [(0, -128), (-113, -121), (-255, -250)], ids=lambda z: "zi{}_zf{}".format(*z))
def test_reductions_of_one_step(oracle, case, zp):
    C, K, H, W, Fh, Fw, s, pads, N = case
    rng = np.random.default_rng(C + K + H)
    q = _quant(rng, C * Fh * Fw, zp)
    x = P.pack_activation(rng.integers(0, 256, (N, C, H, W)).astype(np.uint8))
    w = P.pack_conv_filter(rng.integers(0, 256, (K, C, Fh, Fw)).astype(np.uint8))
    sh = shape(C, K, H, W, Fh, Fw, s, pads, CB)
    ho, wo = sh.out_hw()
    I, F, O = qbuf(x, zp[0]), qbuf(w, zp[1]), _out(N * K * ho * wo, q)
    S.Conv2D(Fh, Fw, s, *pads, K, C, H, W, I, F, O, batch=N, path="cuda_cores")
    want = np.stack([oracle.conv2d_u8(sh, q, x[n], w) for n in range(N)])
    assert np.array_equal(O.numpy().reshape(N, -1), want)
    assert want.min() < want.max()


@pytest.mark.parametrize("case", [
    # C, K, H, W, Fh, Fw, stride, pads, batch
    (48, 176, 9, 14, 3, 3, 1, (1, 1, 1, 1), 2),     # a second block of 48 channels of 128
    (16, 80, 11, 7, 3, 3, 2, (0, 1, 0, 1), 3),      # one block of 80 of 128
    (32, 48, 5, 5, 5, 3, 1, (2, 2, 1, 1), 12),      # one block of 48 of 64, several tiles
    (3, 48, 9, 8, 5, 5, 2, (2, 2, 2, 2), 5),
], ids=lambda c: "C{}_K{}_{}x{}_k{}x{}_s{}_p{}_n{}".format(*c))
@pytest.mark.parametrize("zp", [(0, -128), (-113, -121), (4, -7)], ids=lambda z: "zi{}_zf{}".format(*z))
def test_implicit_gemm_with_a_partial_block_of_channels(oracle, case, zp):
    C, K, H, W, Fh, Fw, s, pads, N = case
    rng = np.random.default_rng(C + K + H)
    q = _quant(rng, C * Fh * Fw, zp)
    x = P.pack_activation(rng.integers(0, 256, (N, C, H, W)).astype(np.uint8))
    w = P.pack_conv_filter(rng.integers(0, 256, (K, C, Fh, Fw)).astype(np.uint8))
    sh = shape(C, K, H, W, Fh, Fw, s, pads, CB)
    ho, wo = sh.out_hw()
    I, F, O = qbuf(x, zp[0]), qbuf(w, zp[1]), _out(N * K * ho * wo, q)
    S.Conv2D(Fh, Fw, s, *pads, K, C, H, W, I, F, O, batch=N, path="tensor_core")
    want = np.stack([oracle.conv2d_u8(sh, q, x[n], w) for n in range(N)])
    assert _lib.device_status() == 0
    assert np.array_equal(O.numpy().reshape(N, -1), want)
    assert want.min() < want.max()
