"""The channel-major tensor-core convolution lets the CTAs of a cluster share the reduction of a tile: by two, three, four, six or
eight, over a whole layer or over the tiles of its last, partial wave as a launch of their own.  Each of these that a layer
can get is held to the oracle here, parts of unequal length among them, bare and with everything an epilogue adds."""
import ctypes as C

import numpy as np
import pytest

from oracle.bindings import same_pads, shape
from smallframework_b200 import _lib
from smallframework_b200 import interface as S
from smallframework_b200 import packing as P
from tests.gpu_util import CB, fbuf, oracle_conv_batch, rel_max_err

pytestmark = pytest.mark.gpu

CASES = [
    # C, K, size, window, images, CTAs to a tile, CTAs to a tile of the remainder (on 148 SMs)
    (128, 144, 7, 3, 24, 2, 0),
    (96, 144, 7, 3, 12, 3, 0),
    (128, 144, 7, 3, 8, 4, 0),
    (96, 144, 7, 3, 2, 6, 0),
    (112, 144, 7, 3, 2, 4, 0),           # seven channel blocks to four
    (128, 144, 7, 3, 1, 8, 0),
    (176, 144, 13, 3, 1, 6, 0),          # eleven to six, two tiles to an image
    (512, 1024, 13, 3, 64, 1, 2),
    (512, 1024, 13, 1, 24, 1, 3),
    (192, 512, 7, 3, 40, 1, 6),
    (256, 512, 7, 3, 40, 1, 8),
]


def cut_of(C_, K, H, W, f, N):
    """(CTAs to a tile, CTAs to a tile of the remainder) of a same-padded layer on the current device."""
    L = S._layer(N, C_, K, H, W, f, f, 1, *same_pads(H, W, f, f, 1))
    v = (C.c_int * 3)()
    _lib.check(_lib.lib().small_b200_conv2d_f32_tf32x3_cut(C.byref(L), v))
    return v[1], v[2]


@pytest.mark.parametrize("full", [False, True], ids=["bare", "seed_bias_act"])
@pytest.mark.parametrize("case", CASES, ids=lambda c: "C{}_K{}_{}_k{}_n{}_cut{}_{}".format(*c))
def test_cut(oracle, case, full):
    import torch
    Cn, K, H, f, N, split, rem = case
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert cut_of(Cn, K, H, H, f, N) == (split, rem)
    pads = same_pads(H, H, f, f, 1)
    rng = np.random.default_rng(Cn + N)
    xp = P.pack_activation(rng.uniform(-1, 1, (N, Cn, H, H)).astype(np.float32))
    wp = P.pack_conv_filter(rng.normal(0, np.sqrt(2 / (Cn * f * f)), (K, Cn, f, f)).astype(np.float32))
    bias = rng.uniform(-0.5, 0.5, K).astype(np.float32) if full else None
    seed = rng.uniform(-1, 1, (N, K * H * H)).astype(np.float32)
    FP, O = S.FloatBuffer(2 * wp.size), fbuf(seed.reshape(-1))
    S.prepare_filter_3xTF32(f, f, K, Cn, fbuf(wp), FP)
    S.Conv2D_3xTF32(f, f, 1, *pads, K, Cn, H, H, fbuf(xp), FP, fbuf(bias) if full else None, O, batch=N, partial=full,
                    activation=S.ACT_LEAKY if full else S.ACT_NONE, negative_slope=0.1)
    got = O.numpy().reshape(N, -1)
    assert _lib.device_status() == 0
    some = sorted({0, N // 2, N - 2 if N > 1 else 0, N - 1})  # the remainder's tiles belong to the last images
    want = oracle_conv_batch(oracle, shape(Cn, K, H, H, f, f, 1, pads, CB), xp[some], wp, bias=bias,
                             act=S.ACT_LEAKY if full else 0, slope=0.1, seed=seed[some].copy() if full else None)
    for n, w in zip(some, want):
        assert rel_max_err(got[n], w) <= 1e-5, n
