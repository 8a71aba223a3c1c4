"""uint8 pointwise layers on 16, 32 and 64 channels as one or two MMAs a tile (csrc/conv_u8_thin.cu) against the oracle, bit-exact: tiles across
images, ragged last tiles, several blocks and parts of output channels, more tiles a CTA than stages, any zero points."""
import ctypes as C_

import numpy as np
import pytest
import torch

from oracle.bindings import Quant, shape
from smallframework_b200 import _lib
from smallframework_b200 import packing as P
from tests.test_gpu_uint8 import _case_id, _check_conv, _quant

pytestmark = pytest.mark.gpu

CASES = [
    # C, K, H, W, Fh, Fw, stride, pads, batch
    (16, 16, 48, 48, 1, 1, 1, "valid", 320),
    (16, 64, 1, 1, 1, 1, 1, "valid", 1),
    (16, 32, 24, 24, 1, 1, 1, "valid", 240),
    (16, 64, 37, 7, 1, 1, 1, "valid", 133),    # parts of the output channels
    (16, 48, 5, 5, 1, 1, 1, "valid", 3600),    # many images a tile
    (32, 32, 24, 24, 1, 1, 1, "valid", 200),   # four and a half tiles an image
    (32, 16, 16, 8, 1, 1, 1, "valid", 601),
    (32, 64, 16, 8, 1, 1, 1, "valid", 240),
    (32, 64, 31, 33, 1, 1, 1, "valid", 90),
    (32, 128, 111, 113, 1, 1, 1, "valid", 3),
    (32, 48, 23, 45, 1, 1, 1, "valid", 60),
    (32, 64, 12, 12, 1, 1, 1, "valid", 231),   # tiles across images: two or three of them a tile
    (32, 16, 13, 5, 1, 1, 1, "valid", 827),
    (64, 64, 12, 12, 1, 1, 1, "valid", 1999),  # two reduction steps
    (64, 48, 8, 8, 1, 1, 1, "valid", 1320),
    (64, 128, 17, 4, 1, 1, 1, "valid", 1150),
]


@pytest.mark.parametrize("case", CASES, ids=_case_id)
@pytest.mark.parametrize("zp", [(0, -128), (-113, -121), (-255, -130)], ids=lambda z: "zi{}_zf{}".format(*z))
def test_conv2d_u8_thin(oracle, case, zp):
    rng = np.random.default_rng(case[0] + case[1] + case[2] + zp[0] + 1000)
    _check_conv(oracle, case, (0, 0, 0, 0), _quant(rng, case[0], zp), rng, zp[0] != 0, None)


@pytest.mark.parametrize("C", [16, 32, 64])
@pytest.mark.parametrize("shift", [0, 1], ids=lambda r: f"rshift{r}")
def test_quantisers_outside_the_common_form(oracle, shift, C):
    rng = np.random.default_rng(3)
    _check_conv(oracle, (C, 32, 32, 32, 1, 1, 1, "valid", 130), (0, 0, 0, 0), Quant(-3, -120, 2 - 2 * shift, shift, 1 << 19, 0), rng, True, None)


@pytest.mark.parametrize("case", [(16, 64, 8, 16, 1, 1, 1, "valid", 1), (16, 64, 3, 43, 1, 1, 1, "valid", 1), (16, 96, 2, 2, 1, 1, 1, "valid", 32),
                                  (16, 128, 5, 26, 1, 1, 1, "valid", 1)], ids=_case_id)
def test_where_a_few_pixels_go(oracle, case):
    """16 channels to 64 and more: from 129 pixels on this kernel."""
    rng = np.random.default_rng(case[1] + case[2])
    _check_conv(oracle, case, (0, 0, 0, 0), _quant(rng, 16, (-113, -121)), rng, True, None)
    assert (_lib.last_kernel() == "conv_u8_thin_kernel") == (case[2] * case[3] * case[8] > 128)


def test_planes_beyond_a_fifteenth_of_31_bits(oracle):
    """One image of 143 million pixels (4.6 GB): the runs of a tile that lie in other images are counted in 32 bits."""
    C, K, H, W = 32, 16, 11970, 11969
    assert 15 * H * W >= 1 << 31
    rng = np.random.default_rng(9)
    gen = torch.Generator("cuda").manual_seed(9)
    x = torch.randint(0, 256, (C // 16, H * W, 16), dtype=torch.uint8, device="cuda", generator=gen)
    out = torch.empty(K // 16, H * W, 16, dtype=torch.uint8, device="cuda")
    q = _quant(rng, C, (-113, -121))
    w = P.pack_conv_filter(rng.integers(0, 256, (K, C, 1, 1)).astype(np.uint8))
    wd = torch.from_numpy(w.reshape(-1)).cuda()
    L = _lib.Layer(1, C, K, H, W, 1, 1, 1, 0, 0, 0, 0, 0, 0, 0.0, q.zero_in, q.zero_filt, q.lshift, q.rshift, q.multiplier, q.k_zero)
    stream = torch.cuda.current_stream()
    _lib.check(_lib.lib().small_b200_conv2d_u8(C_.byref(L), x.data_ptr(), wd.data_ptr(), None, out.data_ptr(), stream.cuda_stream))
    stream.synchronize()
    assert _lib.device_status() == 0 and _lib.last_kernel() == "conv_u8_thin_kernel"
    at = np.unique(np.concatenate([np.arange(3000), rng.integers(0, H * W, 30000), H * W - 1 - np.arange(3000)]))
    some = torch.from_numpy(at).cuda()
    want = oracle.conv2d_u8(shape(C, K, 1, len(at), 1, 1, 1, (0, 0, 0, 0), 16), q, x[:, some].cpu().numpy().ravel(), w)
    assert np.array_equal(out[:, some].cpu().numpy().ravel(), want) and want.min() < want.max()
