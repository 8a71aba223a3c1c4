"""First uint8 layers on three-channel images on the tensor cores (csrc/conv_u8_rgb.cu) against the oracle, bit-exact: both strides,
rows cut into parts, ragged last chunks and tiles, odd rows of bytes, images of a pixel, several blocks of output channels, windows other
than 3x3, the zero points whose padding is a byte."""
import numpy as np
import pytest

from smallframework_b200 import _lib
from tests.test_gpu_uint8 import _case_id, _check_conv, _quant

pytestmark = pytest.mark.gpu

CASES = [
    # C, K, H, W, Fh, Fw, stride, pads, batch: 200 000 outputs and more, fewer stay on the CUDA cores
    (3, 16, 96, 96, 3, 3, 2, "same", 90),
    (3, 16, 96, 96, 3, 3, 2, "same", 163),
    (3, 32, 33, 41, 3, 3, 2, "same", 565),      # two blocks of output channels a CTA, odd sizes
    (3, 48, 30, 31, 3, 3, 2, (1, 1, 1, 1), 840),
    (3, 16, 32, 32, 3, 3, 1, "same", 200),      # four outputs a GEMM row
    (3, 64, 29, 37, 3, 3, 1, "same", 190),
    (3, 16, 5, 700, 3, 3, 1, "same", 58),       # wider than a tile
    (3, 16, 11, 1201, 3, 3, 2, "valid", 67),
    (3, 16, 1, 300, 3, 3, 1, "same", 667),      # most taps outside
    (3, 16, 300, 1, 3, 3, 2, "same", 1340),
    (3, 16, 3, 200, 1, 3, 1, (0, 0, 2, 1), 335),
    (3, 32, 40, 44, 2, 5, 2, "valid", 505),
    (3, 16, 50, 30, 10, 1, 2, "same", 540),
    (3, 16, 40, 43, 2, 5, 1, (1, 0, 3, 1), 118),
    (3, 16, 447, 447, 3, 3, 1, "same", 1),      # one image: the line's other side
]


@pytest.mark.parametrize("case", CASES, ids=_case_id)
@pytest.mark.parametrize("zp", [(0, -128), (-113, -121), (-255, -130)], ids=lambda z: "zi{}_zf{}".format(*z))
def test_conv2d_u8_rgb(oracle, case, zp):
    from oracle.bindings import same_pads
    C, K, H, W, Fh, Fw, s, pm, N = case
    pads = same_pads(H, W, Fh, Fw, s) if pm == "same" else (0, 0, 0, 0) if pm == "valid" else pm
    rng = np.random.default_rng(K * 100 + H * 10 + W + zp[0] + 1000)
    _check_conv(oracle, case, pads, _quant(rng, C * Fh * Fw, zp), rng, zp[0] != 0, None)


@pytest.mark.parametrize("case", [
    (3, 48, 35, 38, 3, 3, 2, (1, 1, 1, 1), 640, "conv_u8_rgb_kernel"), (3, 48, 30, 31, 3, 3, 2, (1, 1, 1, 1), 840, "conv2d_u8_onestep_kernel"),
    (3, 16, 300, 3, 3, 3, 2, (1, 1, 1, 1), 700, "conv_u8_rgb_kernel"), (3, 16, 300, 1, 3, 3, 2, (1, 1, 1, 1), 1340, "conv2d_u8_onestep_kernel"),
    (3, 64, 18, 18, 3, 3, 1, (1, 1, 1, 1), 620, "conv_u8_rgb_kernel"), (3, 64, 38, 9, 3, 3, 1, (1, 1, 1, 1), 600, "conv2d_u8_onestep_kernel"),
], ids=lambda c: _case_id(c[:9]))
def test_how_full_tiles_are(oracle, case):
    rng = np.random.default_rng(case[1] + case[2])
    _check_conv(oracle, case[:9], case[7], _quant(rng, 27, (-113, -121)), rng, True, None)
    assert _lib.last_kernel() == case[9]


@pytest.mark.parametrize("shift", [0, 1], ids=lambda r: f"rshift{r}")
def test_quantisers_outside_the_common_form(oracle, shift):
    from oracle.bindings import Quant, same_pads
    case = (3, 16, 64, 64, 3, 3, 2, "same", 200)
    rng = np.random.default_rng(3)
    q = Quant(-3, -120, 2 - 2 * shift, shift, 1 << 14, 0)
    _check_conv(oracle, case, same_pads(64, 64, 3, 3, 2), q, rng, True, None)
