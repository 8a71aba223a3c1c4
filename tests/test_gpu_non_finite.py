"""Infinities and NaN in the tensor-core fp32 convolutions, stride 1 and 2: they reach the outputs whose windows they lie in, with
the sign or the NaN that the products of the loop nest give, and no others.  (Operands enter the tensor core as two
words, and an infinity minus itself is none.)"""
import numpy as np
import pytest

from oracle.bindings import same_pads, shape
from smallframework_b200 import _lib
from smallframework_b200 import interface as S
from smallframework_b200 import packing as P
from tests.gpu_util import CB, fbuf, oracle_conv_batch, rel_max_err

pytestmark = pytest.mark.gpu

# C, K, H, W, window, stride, images, what follows (kernels as in test_gpu_operand_range.py; stride 2: the gathering kernel)
CASES = [
    (16, 16, 24, 24, 3, 1, 8, ""), (32, 32, 20, 20, 3, 1, 3, ""), (48, 64, 20, 20, 3, 1, 2, ""), (16, 32, 72, 70, 3, 1, 1, "pool"),
    (32, 48, 30, 30, 3, 1, 2, ""), (32, 48, 12, 12, 3, 1, 3, "partial"), (64, 128, 13, 13, 3, 1, 1, ""),
    (128, 144, 13, 13, 3, 1, 2, "partial"), (32, 256, 26, 26, 3, 1, 30, ""), (32, 48, 40, 40, 1, 1, 4, ""),
    (64, 32, 6, 6, 1, 1, 90, ""), (48, 64, 29, 31, 3, 2, 4, ""),
]
IDS = ["C{}_K{}_{}x{}_k{}_s{}_n{}{}".format(*c) for c in CASES]
NO_POOL = [c for c in CASES if c[-1] != "pool"]
NO_POOL_IDS = [i for c, i in zip(CASES, IDS) if c[-1] != "pool"]


def _run(case, x, w, bias, seed):
    C, K, H, W, f, s, N, what = case
    pads = same_pads(H, W, f, f, s)
    I, B = fbuf(P.pack_activation(x)), fbuf(bias)
    wp = P.pack_conv_filter(w)
    ho, wo = shape(C, K, H, W, f, f, s, pads, CB).out_hw()
    O = fbuf(P.pack_activation(seed)) if what == "partial" else S.FloatBuffer(N * K * (ho * wo // 4 if what == "pool" else ho * wo))
    if s == 2:
        S.Conv2D_Bias_Activation(f, f, s, *pads, K, C, H, W, I, fbuf(wp), B, O, batch=N)
    else:
        FP = S.FloatBuffer(2 * w.size)
        S.prepare_filter_3xTF32(f, f, K, C, fbuf(wp), FP)
        if what == "pool":
            S.Conv2D_Maxpool2D_3xTF32(f, f, pads, K, C, H, W, I, FP, B, O, batch=N)
        else:
            S.Conv2D_3xTF32(f, f, s, *pads, K, C, H, W, I, FP, B, O, partial=what == "partial", batch=N)
    assert _lib.device_status() == 0
    return O.numpy().reshape(N, -1)


def _same(oracle, case, x, w):
    C, K, H, W, f, s, N, what = case
    rng = np.random.default_rng(C * K)
    pads = same_pads(H, W, f, f, s)
    sh = shape(C, K, H, W, f, f, s, pads, CB)
    bias = rng.uniform(-0.1, 0.1, K).astype(np.float32)
    seed = rng.uniform(-1, 1, (N, K, *sh.out_hw())).astype(np.float32)
    got = _run(case, x, w, bias, seed)
    want = oracle_conv_batch(oracle, sh, P.pack_activation(x), P.pack_conv_filter(w), bias=bias,
                             seed=P.pack_activation(seed).reshape(N, -1) if what == "partial" else None)
    if what == "pool":
        want = np.stack([oracle.pool2d_f32(shape(K, K, H, W, 2, 2, 2, (0, 0, 0, 0), CB), v) for v in want])
    assert np.array_equal(np.isnan(got), np.isnan(want))
    assert np.array_equal(np.where(np.isinf(got), got, 0), np.where(np.isinf(want), want, 0))
    fin = np.isfinite(want)
    assert 0 < fin.sum() < fin.size
    assert rel_max_err(got[fin], want[fin]) <= 1e-5


def _operands(case):
    C, K, H, W, f, s, N, _ = case
    rng = np.random.default_rng(C + K + H)
    return rng.uniform(-1, 1, (N, C, H, W)).astype(np.float32), rng.normal(0, 0.1, (K, C, f, f)).astype(np.float32)


@pytest.mark.parametrize("case", CASES, ids=IDS)
def test_infinities_in_the_activations(oracle, case):
    C, K, H, W, f, s, N, _ = case
    x, w = _operands(case)
    x[0, 3, 2, 3] = np.inf
    x[N - 1, C - 1, H - 1, W - 1] = -np.inf
    if N > 2:                            # two that meet
        x[1, 0, 3, 3], x[1, C - 1, 3, 4 if f > 1 else 3] = np.inf, -np.inf
    w[K // 2] = np.abs(w[K // 2])
    if case[-1] != "pool":               # a NaN: which of four values the maximum passes over is the order's
        w[0, 3] = 0
    _same(oracle, case, x, w)


@pytest.mark.parametrize("case", CASES, ids=IDS)
def test_products_past_the_largest_number(oracle, case):
    """Finite operands whose products are not, beside zeros, which stay nothing whatever the scales are."""
    C, K, H, W, f, s, N, _ = case
    x, w = _operands(case)
    x = np.abs(x) * 1e38
    x[N // 2, :, H // 3:] = 0
    _same(oracle, case, x, (np.abs(w) + 0.01) * 1e12)


@pytest.mark.parametrize("case", NO_POOL, ids=NO_POOL_IDS)
def test_nan_in_the_activations(oracle, case):
    C, K, H, W, f, s, N, _ = case
    x, w = _operands(case)
    x[N // 2, C // 2, H // 2, 1] = np.nan
    _same(oracle, case, x, w)


@pytest.mark.parametrize("value", [np.inf, np.nan], ids=str)
@pytest.mark.parametrize("case", NO_POOL, ids=NO_POOL_IDS)
def test_one_weight(oracle, case, value):
    """At a corner of the window: the padding it meets is not there, so border pixels stay finite."""
    C, K, H, W, f, s, N, _ = case
    x, w = _operands(case)
    w[K - 2, C // 2, 0, 0] = value
    _same(oracle, case, x, w)
