"""16 and 32 output channels on the tensor cores with one and two sets of operand splitters (csrc/conv_f16x3.cu), to either side of
the line between them: images of magnitudes apart, so that a patch converted with another one's scale shows."""
import numpy as np
import pytest

from oracle.bindings import same_pads, shape
from smallframework_b200 import _lib
from smallframework_b200 import interface as S
from smallframework_b200 import packing as P
from tests.gpu_util import CB, fbuf, oracle_conv_batch, rel_max_err

pytestmark = pytest.mark.gpu

CASES = [
    # C, K, H, W, kernel, images, pool: a 16x16 or 32x32 image gives two and eight patches of 16 channels and 128 pixels
    (16, 16, 32, 32, 3, 16, False), (16, 16, 32, 32, 3, 47, False), (16, 16, 32, 32, 3, 90, False), (16, 32, 16, 16, 3, 301, False),
    (32, 32, 16, 16, 3, 1, False), (48, 16, 20, 20, 3, 7, False), (80, 32, 9, 20, 3, 131, False), (128, 16, 7, 7, 1, 40, False),
    (16, 32, 70, 90, 5, 9, False), (48, 32, 40, 130, 3, 4, True), (16, 32, 208, 208, 3, 5, True), (16, 32, 208, 208, 3, 51, True),
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "C{}_K{}_{}x{}_k{}_n{}{}".format(*c[:6], "_pool" if c[6] else ""))
def test_against_the_oracle(oracle, case):
    c, k, h, w, f, n, pool = case
    pads = same_pads(h, w, f, f, 1)
    rng = np.random.default_rng(c + k + h + n)
    x = rng.uniform(-1, 1, (n, c, h, w)).astype(np.float32) * (8.0 ** (np.arange(n) % 5 - 2)).astype(np.float32)[:, None, None, None]
    x, wt = P.pack_activation(x), P.pack_conv_filter(rng.normal(0, np.sqrt(2.0 / (c * f * f)), (k, c, f, f)).astype(np.float32))
    I, F = fbuf(x), fbuf(wt)
    Fp, O = S.FloatBuffer(2 * F.size()), S.FloatBuffer(n * k * h * w // (4 if pool else 1))
    S.prepare_filter_3xTF32(f, f, k, c, F, Fp)
    if pool:
        S.Conv2D_Maxpool2D_3xTF32(f, f, pads, k, c, h, w, I, Fp, None, O, batch=n)
    else:
        S.Conv2D_3xTF32(f, f, 1, *pads, k, c, h, w, I, Fp, None, O, batch=n)
    got = O.numpy().reshape(n, -1)
    assert _lib.device_status() == 0
    some = np.unique(np.linspace(0, n - 1, 12).astype(int))
    want = oracle_conv_batch(oracle, shape(c, k, h, w, f, f, 1, pads, CB), x[some], wt)
    for i, ref in zip(some, want):
        if pool:
            ref = oracle.pool2d_f32(shape(k, k, h, w, 2, 2, 2, (0, 0, 0, 0), CB), ref)
        assert rel_max_err(got[i], ref) <= 1e-5  # pairs of 11-bit words: a product is off by 2^-21 at most, the rest is fp32 sums


TRAVELLING = [
    # C, K, H, W, kernel, images, onto what is there: more patches than filter stages, two tiles a CTA and more
    (128, 32, 26, 35, 3, 90, False), (144, 16, 26, 35, 3, 90, False), (96, 16, 20, 60, 5, 70, False), (64, 32, 16, 60, 7, 70, False),
    (256, 16, 30, 33, 1, 90, False), (128, 16, 26, 35, 3, 90, True), (112, 32, 26, 35, 3, 2, True),
]


@pytest.mark.parametrize("case", TRAVELLING, ids=lambda c: "C{}_K{}_{}x{}_k{}_n{}{}".format(*c[:6], "_onto" if c[6] else ""))
def test_filters_that_travel(oracle, case):
    """Two sets of splitters with four patch slots beside a ring of filter stages, and the forms that find their pixel late."""
    c, k, h, w, f, n, onto = case
    pads = same_pads(h, w, f, f, 1)
    rng = np.random.default_rng(c + k + f)
    x = rng.uniform(-1, 1, (n, c, h, w)).astype(np.float32) * (8.0 ** (np.arange(n) % 5 - 2)).astype(np.float32)[:, None, None, None]
    x, wt = P.pack_activation(x), P.pack_conv_filter(rng.normal(0, np.sqrt(2.0 / (c * f * f)), (k, c, f, f)).astype(np.float32))
    seed = rng.uniform(-1, 1, (n, k * h * w)).astype(np.float32) if onto else None
    I, F, O = fbuf(x), fbuf(wt), fbuf(seed) if onto else S.FloatBuffer(n * k * h * w)
    Fp = S.FloatBuffer(2 * F.size())
    S.prepare_filter_3xTF32(f, f, k, c, F, Fp)
    S.Conv2D_3xTF32(f, f, 1, *pads, k, c, h, w, I, Fp, None, O, partial=onto, batch=n)
    got = O.numpy().reshape(n, -1)
    assert _lib.device_status() == 0
    some = np.unique(np.linspace(0, n - 1, 8).astype(int))
    want = oracle_conv_batch(oracle, shape(c, k, h, w, f, f, 1, pads, CB), x[some], wt, seed=seed[some] if onto else None)
    for i, ref in zip(some, want):
        assert rel_max_err(got[i], ref) <= 1e-5  # as above


def test_pooled_with_wide_tiles_and_infinities(oracle):
    """The pooled form with two sets of splitters (an input beyond L2): images with a pixel 2^30 and more above its neighbours, whose tiles are
    summed on the FMA pipe, and with an infinity, beside ordinary ones."""
    c, k, h, n = 16, 32, 208, 51
    rng = np.random.default_rng(3)
    x = rng.uniform(-1, 1, (n, c, h, h)).astype(np.float32)
    spots = {4: (57, 91), 23: (0, 0), 50: (207, 130)}
    for i, (r, q) in spots.items():
        x[i] *= 1e-5
        x[i, 3, r, q] = 3e4
    x[30, 5, 100, 33], x[31, 0, 207, 207] = np.inf, -np.inf
    wt = rng.normal(0, np.sqrt(2.0 / (c * 9)), (k, c, 3, 3)).astype(np.float32)
    I, F = fbuf(P.pack_activation(x)), fbuf(P.pack_conv_filter(wt))
    Fp, O = S.FloatBuffer(2 * F.size()), S.FloatBuffer(n * k * h * h // 4)
    S.prepare_filter_3xTF32(3, 3, k, c, F, Fp)
    S.Conv2D_Maxpool2D_3xTF32(3, 3, (1, 1, 1, 1), k, c, h, h, I, Fp, None, O, batch=n)
    got = P.unpack_activation(O.numpy().reshape(n, -1), k, h // 2, h // 2)
    assert _lib.device_status() == 0
    some = [3, *spots, 24, 30, 31, 32]
    want = oracle_conv_batch(oracle, shape(c, k, h, h, 3, 3, 1, (1, 1, 1, 1), CB), P.pack_activation(x[some]), P.pack_conv_filter(wt))
    for i, ref in zip(some, want):
        ref = P.unpack_activation(oracle.pool2d_f32(shape(k, k, h, h, 2, 2, 2, (0, 0, 0, 0), CB), ref)[None], k, h // 2, h // 2)[0]
        mine, fin = got[i], np.isfinite(ref)
        assert np.array_equal(np.isposinf(mine), np.isposinf(ref)) and np.array_equal(np.isfinite(mine), fin)
        assert fin.all() == (i not in (30, 31))
        if i in spots:
            r, q = (v // 2 for v in spots[i])
            near = np.zeros_like(fin)
            near[:, max(0, r - 1):r + 2, max(0, q - 1):q + 2] = True
            assert rel_max_err(mine[near], ref[near]) <= 1e-5
            fin = ~near # to the size of the sums around, 10^9 below
        assert rel_max_err(mine[fin], ref[fin]) <= 1e-5
