"""The tensor-core fp32 convolution (stride 1) holds an operand as two half-precision words under a power of two: one for each
output channel of the filter, one for each patch of activations.  Whatever the magnitudes beside it, an output channel, an
image and a pixel keep the precision of their own: every output is held on its own to a bound on its own terms,
    |got - exact| <= 2^-17 * (sum |x||w| + |bias| + |seed|),
of which the words take 2^-21 for each operand (11 + 11 bits, cut), the product of the second words that is left out 2^-20, the
tensor core's truncating additions (at most nine full-size ones to a group, sixteen products each) some 2^-19, and the rest
is for the magnitudes within one pixel's channels (a factor of two here) and the fp32 additions of the groups."""
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
BOUND = 2.0 ** -17

# C, K, H, W, window, images, what follows
CASES = [
    (16, 16, 24, 24, 3, 20, ""),          # pixel-major, whole windows, filter resident
    (32, 32, 20, 20, 3, 6, ""),
    (256, 32, 12, 12, 3, 2, ""),          # pixel-major, a filter ring
    (48, 64, 20, 20, 3, 3, ""),           # pixel-major, 64 channels
    (16, 32, 72, 70, 3, 1, "pool"),
    (64, 64, 66, 68, 3, 1, "pool"),
    (32, 48, 30, 30, 3, 2, ""),           # channel-major, persistent
    (32, 48, 12, 12, 3, 3, "partial"),
    (64, 128, 13, 13, 3, 1, ""),          # a cluster shares the reduction of a tile
    (128, 144, 13, 13, 3, 2, "partial"),  # ... with a partial last channel tile, seeded
    (32, 256, 26, 26, 3, 30, ""),         # one CTA a tile
    (32, 48, 40, 40, 1, 4, ""),           # runs of pixels
    (64, 32, 6, 6, 1, 90, ""),            # images share tiles
    (128, 256, 3, 3, 1, 60, ""),
    (48, 32, 9, 11, 5, 2, "partial"),
]
IDS = ["C{}_K{}_{}x{}_k{}_n{}{}".format(*c) for c in CASES]


def _signed(rng, shape):
    """Magnitudes in [0.5, 1)."""
    return rng.uniform(0.5, 1, shape) * rng.choice([-1.0, 1.0], shape)


def _run(case, x, w, bias, seed):
    C, K, H, W, f, N, what = case
    pads = same_pads(H, W, f, f, 1)
    I, FP = fbuf(P.pack_activation(x)), S.FloatBuffer(2 * w.size)
    S.prepare_filter_3xTF32(f, f, K, C, fbuf(P.pack_conv_filter(w)), FP)
    B = fbuf(bias)
    if what == "pool":
        O = S.FloatBuffer(N * K * (H // 2) * (W // 2))
        S.Conv2D_Maxpool2D_3xTF32(f, f, pads, K, C, H, W, I, FP, B, O, batch=N)
    else:
        O = fbuf(P.pack_activation(seed))
        S.Conv2D_3xTF32(f, f, 1, *pads, K, C, H, W, I, FP, B, O, partial=what == "partial", batch=N)
    assert _lib.device_status() == 0
    return P.unpack_activation(O.numpy().reshape(N, -1), K, *((H // 2, W // 2) if what == "pool" else (H, W)))


def _check(case, x, w, bias, seed):
    C, K, H, W, f, N, what = case
    x, w, bias, seed = (a.astype(np.float32) for a in (x, w, bias, seed))
    got = torch.from_numpy(_run(case, x, w, bias, seed).astype(np.float64))
    t = lambda a: torch.from_numpy(a.astype(np.float64))
    b = t(bias)[None, :, None, None]
    exact = F.conv2d(t(x), t(w), padding=f // 2) + b
    terms = F.conv2d(t(x).abs(), t(w).abs(), padding=f // 2) + b.abs()
    if what == "partial":
        exact, terms = exact + t(seed), terms + t(seed).abs()
    if what == "pool":  # the maximum of four is off by no more than the one of them that is off most
        exact, terms = F.max_pool2d(exact, 2), F.max_pool2d(terms, 2)
    worst = float(((got - exact).abs() / terms).max())
    print(f"\nworst error over its terms: 2^{np.log2(max(worst, 1e-30)):.2f}", end="")
    assert worst <= BOUND, f"2^{np.log2(worst):.2f}"


@pytest.mark.parametrize("case", CASES, ids=IDS)
def test_output_channels_far_apart(case):
    C, K, H, W, f, N, _ = case
    rng = np.random.default_rng(C + K + H)
    own = 2.0 ** -rng.integers(0, 60, (K, 1, 1, 1))
    _check(case, _signed(rng, (N, C, H, W)), _signed(rng, (K, C, f, f)) * own, _signed(rng, K) * own[:, 0, 0, 0],
           _signed(rng, (N, K, H, W)) * own[None, :, 0])


@pytest.mark.parametrize("case", [c for c in CASES if c[0] > 16], ids=[i for c, i in zip(CASES, IDS) if c[0] > 16])
def test_weights_of_a_channel_far_apart(case):
    """Half of the blocks of input channels 2^24 larger than the others, their weights as much smaller, in output channels
    2^11 below the largest: either half matters as much as the other."""
    C, K, H, W, f, N, _ = case
    rng = np.random.default_rng(C + K + H)
    block = np.repeat(np.where(np.arange(C // 16) % 2, 2.0 ** 24, 1.0), 16)
    own = np.full((K, 1, 1, 1), 2.0 ** -11)
    own[K // 2] = 1
    _check(case, _signed(rng, (N, C, H, W)) * block[:, None, None], _signed(rng, (K, C, f, f)) * own / block[:, None, None],
           _signed(rng, K) * own[:, 0, 0, 0], _signed(rng, (N, K, H, W)) * own[None, :, 0])


@pytest.mark.parametrize("bits", [20, 80], ids=lambda b: f"{b}bits")
@pytest.mark.parametrize("case", CASES, ids=IDS)
def test_images_far_apart(case, bits):
    C, K, H, W, f, N, _ = case
    rng = np.random.default_rng(C + K + H + bits)
    own = 2.0 ** -rng.integers(0, bits + 1, (N, 1, 1, 1))
    _check(case, _signed(rng, (N, C, H, W)) * own, _signed(rng, (K, C, f, f)), _signed(rng, K) * 2.0 ** -bits, _signed(rng, (N, K, H, W)) * own)


@pytest.mark.parametrize("bits", [16, 30, 80], ids=lambda b: f"{b}bits")
@pytest.mark.parametrize("case", CASES, ids=IDS)
def test_pixels_far_apart(case, bits):
    """A few large pixels in a small image: the outputs away from them see the small ones alone."""
    C, K, H, W, f, N, what = case
    rng = np.random.default_rng(C + K + H + bits)
    own = np.where(rng.random((N, 1, H, W)) < 0.01, 1.0, 2.0 ** -bits)
    if what != "partial":
        own[0, 0, H // 2] = 0  # and a row of zeros, which is no small row
    _check(case, _signed(rng, (N, C, H, W)) * own, _signed(rng, (K, C, f, f)), _signed(rng, K) * 2.0 ** -bits,
           _signed(rng, (N, K, H, W)) * 2.0 ** -bits)


# magnitudes of activations and filter that the tensor core is not given, or whose scales are far apart, or whose inverse scales
# (2^-110 and, as the kernel has it, 2^-30 or 2^-20 at least) multiply to next to nothing
EXTREMES = [(3e37, 1e-20), (1e-30, 1e30), (1e-18, 1e-16), (1e-35, 1e3), (1e-30, 1e-5), (1e-30, 1.25e-2)]


@pytest.mark.parametrize("scales", EXTREMES, ids=lambda s: "x{:g}_w{:g}".format(*s))
@pytest.mark.parametrize("case", CASES, ids=IDS)
def test_extreme_magnitudes(case, scales):
    C, K, H, W, f, N, what = case
    rng = np.random.default_rng(C + K + H)
    x = _signed(rng, (N, C, H, W)) * scales[0]
    x[N // 2, :, H // 2:] = 0
    out = scales[0] * scales[1]
    _check(case, x, _signed(rng, (K, C, f, f)) * scales[1], _signed(rng, K) * out, _signed(rng, (N, K, H, W)) * out)


def test_wide_tiles_past_the_tiles_of_one_launch():
    """A launch has at most 1024 tiles a CTA: images of one tile each, more than 148 CTAs take in one launch, a few of them wide."""
    C = K = 16
    H = W = 3
    N = 148 * 1024 + 3000
    rng = np.random.default_rng(9)
    w = _signed(rng, (K, C, 3, 3)).astype(np.float32)
    g = torch.Generator(device="cuda").manual_seed(9)
    x = torch.rand((N, H * W, C), device="cuda", generator=g) * 0.5 + 0.5
    sample = np.unique(np.concatenate([rng.integers(0, N, 300), [0, 147, 148, 148 * 1024 - 1, 148 * 1024, N - 1]]))
    at = torch.from_numpy(sample[::2].copy()).cuda()
    x[at, 1:] *= 2.0 ** -40
    I, FP, O = S.FloatBuffer(data=x.reshape(-1)), S.FloatBuffer(2 * w.size), S.FloatBuffer(N * K * H * W)
    S.prepare_filter_3xTF32(3, 3, K, C, fbuf(P.pack_conv_filter(w)), FP)
    S.Conv2D_3xTF32(3, 3, 1, 1, 1, 1, 1, K, C, H, W, I, FP, None, O, batch=N)
    pick = torch.from_numpy(sample).cuda()
    got = O.data().reshape(N, H * W, K)[pick].cpu().numpy().reshape(-1, H, W, K).transpose(0, 3, 1, 2).astype(np.float64)
    assert _lib.device_status() == 0
    xs = torch.from_numpy(x[pick].cpu().numpy().reshape(-1, H, W, C).transpose(0, 3, 1, 2).astype(np.float64))
    t = torch.from_numpy(w.astype(np.float64))
    exact, terms = F.conv2d(xs, t, padding=1), F.conv2d(xs.abs(), t.abs(), padding=1)
    assert float(((torch.from_numpy(got) - exact).abs() / terms).max()) <= BOUND
