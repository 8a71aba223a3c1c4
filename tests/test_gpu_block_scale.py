"""The tensor-core fp32 convolution scales every patch by a power of two, kept from patch to patch while it fits: images
whose magnitudes jump (so that a CTA meets patches outside the range of the scale at hand, and tiles with several images of them), all-zero images
between them, and an infinity, each held to the oracle on its own."""
import numpy as np
import pytest

from oracle.bindings import same_pads, shape
from smallframework_b200 import _lib
from smallframework_b200 import interface as S
from smallframework_b200 import packing as P
from tests.gpu_util import CB, fbuf, oracle_conv_batch, rel_max_err

pytestmark = pytest.mark.gpu

# C, K, H, W, window, images: pixel-major with 16 / 64 channels (persistent CTAs over many tiles), channel-major, 1x1
CASES = [(16, 16, 24, 24, 3, 160), (32, 64, 20, 20, 3, 120), (48, 128, 13, 13, 3, 7), (32, 48, 40, 40, 1, 40),
         (64, 32, 6, 6, 1, 90)]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "C{}_K{}_{}x{}_k{}_n{}".format(*c))
def test_magnitudes_that_jump_from_image_to_image(oracle, case):
    C, K, H, W, f, N = case
    pads = same_pads(H, W, f, f, 1)
    rng = np.random.default_rng(C + K)
    x = rng.uniform(-1, 1, (N, C, H, W)).astype(np.float32)
    scale = np.array([1.0, 1e-7, 3e9, 0.0, 1e-30, 1e12])[rng.integers(0, 6, N)].astype(np.float32)
    x *= scale[:, None, None, None]
    w = rng.normal(0, 1e-3, (K, C, f, f)).astype(np.float32)
    sh = shape(C, K, H, W, f, f, 1, pads, CB)
    ho, wo = sh.out_hw()
    xp, wp = P.pack_activation(x), P.pack_conv_filter(w)
    F, O = fbuf(wp), S.FloatBuffer(N * K * ho * wo)
    FP = S.FloatBuffer(2 * F.size())
    S.prepare_filter_3xTF32(f, f, K, C, F, FP)
    S.Conv2D_3xTF32(f, f, 1, *pads, K, C, H, W, fbuf(xp), FP, None, O, batch=N)
    got = O.numpy().reshape(N, -1)
    assert _lib.device_status() == 0
    want = oracle_conv_batch(oracle, sh, xp, wp)
    for n in range(N):  # each on its own, also where several images share a tile (1x1 on small images)
        assert rel_max_err(got[n], want[n]) <= 1e-5, (n, scale[n])
    assert rel_max_err(got, want) <= 1e-5


def test_an_infinity_stays_where_it_is(oracle):
    C, K, H, W = 32, 32, 18, 18
    rng = np.random.default_rng(3)
    x = rng.uniform(0.1, 1, (1, C, H, W)).astype(np.float32)
    x[0, 4, 2, 3] = np.inf
    w = rng.normal(0, 0.1, (K, C, 3, 3)).astype(np.float32)
    sh = shape(C, K, H, W, 3, 3, 1, (1, 1, 1, 1), CB)
    xp, wp = P.pack_activation(x), P.pack_conv_filter(w)
    F, O = fbuf(wp), S.FloatBuffer(K * H * W)
    FP = S.FloatBuffer(2 * F.size())
    S.prepare_filter_3xTF32(3, 3, K, C, F, FP)
    S.Conv2D_3xTF32(3, 3, 1, 1, 1, 1, 1, K, C, H, W, fbuf(xp), FP, None, O)
    want = oracle_conv_batch(oracle, sh, xp, wp)[0]
    got, fin = O.numpy(), np.isfinite(want)
    assert np.array_equal(np.isfinite(got), fin) and 0 < (~fin).sum() < fin.size
    assert rel_max_err(got[fin], want[fin]) <= 1e-5
