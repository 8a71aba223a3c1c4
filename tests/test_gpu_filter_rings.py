"""Filters of the tensor-core fp32 convolution that pass through a ring of two or three stages (windows of seven columns and more), through
many groups of taps: every image, against fp64, several filters one behind the other.  Bound as in test_gpu_operand_range.py, 2^-17
of the terms: a group here is a row of up to 16 taps, so the truncating additions take 2^-19 of it."""
import numpy as np
import pytest
import torch
import torch.nn.functional as F

from oracle.bindings import same_pads
from smallframework_b200 import _lib
from smallframework_b200 import interface as S
from smallframework_b200 import packing as P
from tests.gpu_util import fbuf

pytestmark = pytest.mark.gpu
CASES = [
    # C, K, size, Fh, Fw, images
    (32, 64, 30, 3, 15, 24),    # pixel-major, three stages beside one patch, 192 tiles of six groups
    (64, 64, 16, 16, 16, 40),   # channel-major, 64 groups to a tile
    (64, 64, 12, 5, 9, 200),    # pixel-major, 200 tiles
    (32, 128, 26, 7, 7, 12),    # channel-major, two stages, a cluster to a tile
    (64, 256, 13, 7, 7, 16),    # ... and two accumulators
    (64, 48, 26, 1, 11, 40),    # ... persistent
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "C{}_K{}_{}_k{}x{}_n{}".format(*c))
def test_filter_ring(case):
    C, K, H, fh, fw, N = case
    t, b, l, r = pads = same_pads(H, H, fh, fw, 1)
    assert S.tf32x3_supported(fh, fw, 1, *pads, K, C, H, H)
    rng = np.random.default_rng(C + K + fw)
    x = rng.uniform(-1, 1, (N, C, H, H)).astype(np.float32)
    I, FP, O = fbuf(P.pack_activation(x)), S.FloatBuffer(2 * K * C * fh * fw), S.FloatBuffer(N * K * H * H)
    xp = F.pad(torch.from_numpy(x.astype(np.float64)), (l, r, t, b))
    for _ in range(3):
        w = rng.normal(0, np.sqrt(2.0 / (C * fh * fw)), (K, C, fh, fw)).astype(np.float32)
        S.prepare_filter_3xTF32(fh, fw, K, C, fbuf(P.pack_conv_filter(w)), FP)
        S.Conv2D_3xTF32(fh, fw, 1, *pads, K, C, H, H, I, FP, None, O, batch=N)
        got = torch.from_numpy(P.unpack_activation(O.numpy().reshape(N, -1), K, H, H).astype(np.float64))
        assert _lib.device_status() == 0
        wt = torch.from_numpy(w.astype(np.float64))
        exact, terms = F.conv2d(xp, wt), F.conv2d(xp.abs(), wt.abs())
        worst = float(((got - exact).abs() / terms).max())
        assert worst <= 2.0 ** -17, f"2^{np.log2(worst):.2f}"
