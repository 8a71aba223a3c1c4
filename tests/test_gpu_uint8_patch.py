"""The uint8 convolution that fetches its pixels once (csrc/conv_u8_patch.cu) against the oracle, bit-exact: rows cut into
parts, ragged last tiles, several whole images a tile, strides of two with odd sizes, windows other than 3x3, odd numbers of
channel blocks, filters that stay in shared memory and filters that travel with the pixels, partial blocks of output channels,
and the zero points whose padding is a byte."""
import ctypes

import numpy as np
import pytest
import torch

from oracle.bindings import shape
from smallframework_b200 import _lib
from tests.test_gpu_uint8 import _case_id, _check_conv, _quant

pytestmark = pytest.mark.gpu

CASES = [
    # C, K, H, W, Fh, Fw, stride, pads, batch
    (64, 64, 45, 37, 3, 3, 1, "same", 5),       # three rows of the full width a tile
    (64, 128, 45, 37, 3, 3, 2, "same", 3),
    (32, 16, 33, 37, 3, 3, 1, "same", 45),      # several tiles a CTA
    (64, 128, 45, 37, 3, 3, 2, "same", 38),     # ... with two stages
    (144, 32, 20, 20, 3, 3, 1, "same", 112),    # ... in chunks of the channels
    (16, 16, 112, 112, 3, 3, 1, "same", 2),     # one block of channels: nine slabs, an odd step
    (16, 32, 11, 130, 3, 3, 1, "same", 1),      # wider than a tile
    (48, 48, 7, 7, 3, 3, 1, "same", 40),        # whole images a tile, odd blocks
    (32, 64, 3, 3, 3, 3, 1, "same", 37),        # many of them, the last tile partial
    (32, 32, 1, 1, 3, 3, 1, "same", 9),         # every tap but one outside
    (256, 256, 20, 19, 3, 3, 1, "same", 2),     # the filter travels
    (256, 128, 20, 19, 3, 3, 1, "same", 38),    # ... through several tiles a CTA
    (208, 336, 9, 10, 3, 3, 2, "same", 3),      # odd blocks, a partial block of output channels
    (256, 512, 14, 13, 3, 3, 2, "same", 2),
    (512, 64, 10, 6, 3, 3, 1, "same", 1),
    (32, 48, 9, 14, 5, 5, 1, "same", 2),
    (16, 16, 30, 9, 7, 7, 1, "same", 2),
    (80, 16, 17, 5, 2, 4, 2, "valid", 3),
    (64, 32, 6, 40, 1, 3, 1, "same", 2),
    (32, 32, 40, 6, 3, 1, 2, "same", 2),
    (16, 16, 3, 3, 7, 7, 1, (3, 3, 3, 3), 4),   # windows that cover the image
    (32, 64, 57, 57, 3, 3, 1, (1, 0, 0, 1), 1),
]


@pytest.mark.parametrize("case", CASES, ids=_case_id)
@pytest.mark.parametrize("zp", [(0, -128), (-113, -121), (-255, -130)], ids=lambda z: "zi{}_zf{}".format(*z))
def test_conv2d_u8_patch(oracle, case, zp):
    from oracle.bindings import same_pads
    C, K, H, W, Fh, Fw, s, pm, N = case
    pads = same_pads(H, W, Fh, Fw, s) if pm == "same" else (0, 0, 0, 0) if pm == "valid" else pm
    rng = np.random.default_rng(C * 100 + H * 10 + W + zp[0] + 1000)
    _check_conv(oracle, case, pads, _quant(rng, C * Fh * Fw, zp), rng, zp[0] != 0, None)


RING = [
    # what conv_u8_ring.cu does sooner (see ring_is_shorter), and windows of more taps than the patch kernel has room for
    (16, 16, 19, 19, 1, 3, 2, "same", 1, (-128, -128)),
    (32, 16, 7, 9, 2, 2, 2, "valid", 8, (-128, -128)),
    (32, 64, 3, 3, 1, 3, 1, "same", 2, (-128, -128)),
    (32, 16, 25, 25, 2, 2, 2, "valid", 300, (0, -128)),
    (64, 64, 8, 17, 7, 7, 2, "same", 592, (0, -128)),
    (16, 64, 11, 11, 2, 2, 1, (1, 1, 1, 1), 600, (-113, -121)),
    (256, 256, 8, 8, 1, 3, 2, (0, 0, 1, 1), 1024, (-128, -128)),
    (16, 16, 20, 20, 8, 8, 1, "same", 3, (0, -128)),
    (32, 48, 20, 11, 5, 12, 2, "same", 3, (-128, -128)),
    (16, 32, 20, 20, 10, 5, 1, "same", 2, (-113, -121)),
]


@pytest.mark.parametrize("case", RING, ids=lambda c: _case_id(c[:9]) + "_zi{}_zf{}".format(*c[9]))
def test_layers_that_stay_with_the_ring(oracle, case):
    from oracle.bindings import same_pads
    C, K, H, W, Fh, Fw, s, pm, N, zp = case
    pads = same_pads(H, W, Fh, Fw, s) if pm == "same" else (0, 0, 0, 0) if pm == "valid" else pm
    rng = np.random.default_rng(C + H + W + N)
    _check_conv(oracle, case[:9], pads, _quant(rng, C * Fh * Fw, zp), rng, zp[0] != 0, None)
    assert _lib.last_kernel() == "conv_u8_ring_kernel"


def test_biases_that_the_ring_does_not_take(oracle):
    """Four bytes past a 16-byte boundary: a layer that the ring does sooner stays on the tensor cores all the same."""
    rng = np.random.default_rng(8)
    C, K, H, W, N = 16, 32, 25, 19, 2
    x, w = rng.integers(0, 256, N * C * H * W).astype(np.uint8), rng.integers(0, 256, K * C * 3).astype(np.uint8)
    b = rng.integers(-1024, 1025, K + 1).astype(np.int32)
    q = _quant(rng, C * 3, (-128, -128))
    L = _lib.Layer(N, C, K, H, W, 1, 3, 2, 0, 0, 1, 1, 0, 0, 0.0, q.zero_in, q.zero_filt, q.lshift, q.rshift, q.multiplier, q.k_zero)
    ho, wo = L.out_hw()
    xd, wd, bd = (torch.from_numpy(v).cuda() for v in (x, w, b))
    out = torch.empty(N, K * ho * wo, dtype=torch.uint8, device="cuda")
    for skip, kernel in ((0, "conv_u8_ring_kernel"), (1, "conv_u8_patch_kernel")):
        _lib.check(_lib.lib().small_b200_conv2d_u8(ctypes.byref(L), xd.data_ptr(), wd.data_ptr(), bd.data_ptr() + 4 * skip, out.data_ptr(),
                                                   torch.cuda.current_stream().cuda_stream))
        torch.cuda.synchronize()
        assert _lib.last_kernel() == kernel
        sh = shape(C, K, H, W, 1, 3, 2, (0, 0, 1, 1), 16)
        want = np.stack([oracle.conv2d_u8(sh, q, v, w, bias=b[skip:skip + K]) for v in x.reshape(N, -1)])
        assert np.array_equal(out.cpu().numpy(), want) and want.min() < want.max()


@pytest.mark.parametrize("shift", [0, 1], ids=lambda r: f"rshift{r}")
def test_quantisers_outside_the_common_form(oracle, shift):
    from oracle.bindings import Quant, same_pads
    case = (32, 32, 9, 11, 3, 3, 1, "same", 2)
    rng = np.random.default_rng(3)
    q = Quant(-3, -120, 2 - 2 * shift, shift, 1 << 14, 0)
    _check_conv(oracle, case, same_pads(9, 11, 3, 3, 1), q, rng, True, None)


@pytest.mark.parametrize("case", [
    # C, H, W, Fh, Fw, stride, images: a filter and a patch whose bytes wrap to next to nothing in 32 bits; tiles of more than 2^32 bytes
    (139811 * 16, 7, 7, 7, 7, 1, 1),
    (838860 * 16, 8, 10, 1, 2, 2, 6),
], ids=["filter", "tile"])
def test_sizes_beyond_32_bits(oracle, case):
    """Millions of channels, of which three blocks have pixels other than zero."""
    C, H, W, Fh, Fw, s, N = case
    blocks, taps, used = C // 16, Fh * Fw, [0, C // 48, C // 16 - 1]
    ho, wo = (H - Fh) // s + 1, (W - Fw) // s + 1
    gen = torch.Generator("cuda").manual_seed(5)
    x = torch.zeros(N, blocks, H * W * 16, dtype=torch.uint8, device="cuda")
    x[:, used] = torch.randint(0, 256, (N, 3, H * W * 16), dtype=torch.uint8, device="cuda", generator=gen)
    w = torch.randint(0, 256, (blocks, taps * 256), dtype=torch.uint8, device="cuda", generator=gen)
    out = torch.empty(N, ho * wo * 16, dtype=torch.uint8, device="cuda")
    q = _quant(np.random.default_rng(5), 48 * taps, (0, -121))
    L = _lib.Layer(N, C, 16, H, W, Fh, Fw, s, 0, 0, 0, 0, 0, 0, 0.0, q.zero_in, q.zero_filt, q.lshift, q.rshift, q.multiplier, q.k_zero)
    stream = torch.cuda.current_stream()
    _lib.check(_lib.lib().small_b200_conv2d_u8(ctypes.byref(L), x.data_ptr(), w.data_ptr(), None, out.data_ptr(), stream.cuda_stream))
    stream.synchronize()
    assert _lib.device_status() == 0 and _lib.last_kernel() == "conv_u8_patch_kernel"
    sh = shape(48, 16, H, W, Fh, Fw, s, (0, 0, 0, 0), 16)
    few, xs = w[used].cpu().numpy().ravel(), x[:, used].cpu().numpy()
    want = np.stack([oracle.conv2d_u8(sh, q, xs[n].ravel(), few) for n in range(N)])
    assert np.array_equal(out.cpu().numpy(), want.reshape(N, -1)) and want.min() < want.max()
