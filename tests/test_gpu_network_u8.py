"""A keyword-spotting network as one kernel (csrc/net_u8_tc.cu) against the oracle's layer-by-layer result, bit-exact: both
splits of a CTA's warps over images (up to two images a CTA, up to four; several rounds), images up to the 128-pixel limit and down to one
pixel, windows of one to four chunks of the reduction, signed and unsigned operands, constants too large for the
in-accumulator form, quantisers outside the common form."""
import numpy as np
import pytest
import torch

from smallframework_b200 import _lib, networks
from smallframework_b200 import packing as P
from smallframework_b200.packing import calc_padding, output_dim
from tests.gpu_util import oracle_chain

pytestmark = pytest.mark.gpu

CASES = [
    # H, W, Fh, Fw, stride, blocks, batch, zero_in, zero_mid, classes, biases, quantiser
    (49, 10, 10, 4, 2, 4, 1, -128, 0, 12, 1024, "common"),
    (49, 10, 10, 4, 2, 4, 3, -128, 0, 12, 1024, "common"),
    (49, 10, 10, 4, 2, 4, 200, -128, 0, 12, 1024, "common"),     # two images a CTA
    (49, 10, 10, 4, 2, 4, 301, -128, 0, 12, 1024, "common"),     # four, some CTAs with fewer
    (49, 10, 10, 4, 2, 4, 1400, -128, 0, 12, 1024, "common"),    # several rounds
    (16, 8, 3, 3, 1, 1, 5, 0, 0, 128, 1024, "common"),           # 128 pixels
    (11, 11, 16, 1, 1, 2, 450, 0, -128, 16, 1024, "common"),     # one column of sixteen taps, signed intermediates
    (1, 1, 1, 1, 1, 1, 600, -128, 0, 3, 0, "common"),            # one pixel, no biases
    (9, 1, 5, 2, 1, 6, 7, -128, -128, 12, 1024, "common"),       # one column, six blocks
    (1, 40, 2, 4, 3, 5, 170, 0, 0, 12, 3_000_000, "common"),     # one row; constants beyond the digits
    (20, 12, 10, 4, 2, 2, 310, -128, 0, 12, 1024, "left shift"),
    (20, 12, 10, 4, 2, 2, 2, -128, -128, 12, 3_000_000, "small right shift"),
]


def _same(H, W, Fh, Fw, s):
    return (*calc_padding(H, Fh, s), *calc_padding(W, Fw, s))


def _layers(rng, H, W, Fh, Fw, s, blocks, zi, zm, classes, top, quantiser):
    """Random weights; multipliers calibrated on two images so that every layer's bytes spread over 0..255."""
    cur = rng.integers(0, 256, (2, 1, H, W)).astype(np.uint8)
    L = []

    def add(op, name, C, K, H, W, Fh, Fw, s, pads, zero):
        nonlocal cur
        dw = op == "dwconv"
        w = rng.integers(0, 256, (K, Fh, Fw) if dw else (K, C, Fh, Fw)).astype(np.uint8)
        b = rng.integers(-top, top + 1, K).astype(np.int32) if top else np.zeros(K, np.int32)
        acc = networks._calibrate(cur, w, b, zero, -128, s, pads, dw)
        scale = 255.0 / max(float(np.percentile(acc, 99)), 1.0)
        ls, rs, mult = networks._requant_params(scale)
        if quantiser == "left shift":
            ls, rs = 1, rs + 1
        elif quantiser == "small right shift":
            rs, mult = 1, max(int(round(scale * 2.0 ** 32)), 1)
        L.append(dict(op=op, name=name, C=C, K=K, H=H, W=W, Fh=Fh, Fw=Fw, stride=s, pads=pads, act=0, slope=0.0, w=w,
                      b=b if top else None, q=dict(zero_in=zero, zero_filt=-128, lshift=ls, rshift=rs, multiplier=mult)))
        cur = np.clip(np.rint(acc * scale), 0, 255).astype(np.uint8)

    pads = _same(H, W, Fh, Fw, s)
    h, v = output_dim(H, pads[0], pads[1], Fh, s), output_dim(W, pads[2], pads[3], Fw, s)
    add("conv", "stem", 1, 64, H, W, Fh, Fw, s, pads, zi)
    for i in range(blocks):
        add("dwconv", f"dw{i}", 64, 64, h, v, 3, 3, 1, (1, 1, 1, 1), zm)
        add("conv", f"pw{i}", 64, 64, h, v, 1, 1, 1, (0, 0, 0, 0), int(rng.integers(-20, 20)) if zm else 0)
    ls, rs, mult = networks._requant_params(1.0 / (h * v))
    L.append(dict(op="avgpool", name="pool", C=64, K=64, H=h, W=v, Fh=h, Fw=v, stride=1, pads=(0, 0, 0, 0),
                  q=dict(zero_in=0, zero_filt=0, lshift=ls, rshift=rs, multiplier=mult)))
    cur = np.clip(np.rint(cur.astype(np.float64).mean(axis=(2, 3), keepdims=True)), 0, 255).astype(np.uint8)
    add("conv", "dense", 64, classes, 1, 1, 1, 1, 1, (0, 0, 0, 0), 0)
    return L


@pytest.mark.parametrize("case", CASES, ids=lambda c: "{}x{}_k{}x{}_s{}_b{}_n{}_zi{}_zm{}_Kd{}_{}_{}".format(*c).replace(" ", ""))
def test_network_is_one_kernel(oracle, case):
    H, W, Fh, Fw, s, blocks, N, zi, zm, classes, top, quantiser = case
    rng = np.random.default_rng(H * 1000 + W * 10 + N)
    layers = _layers(rng, H, W, Fh, Fw, s, blocks, zi, zm, classes, top, quantiser)
    chain = networks.Chain(layers, N, "u8")
    x = P.pack_activation(rng.integers(0, 256, (N, 1, H, W), dtype=np.uint8))
    chain.x.copy_(torch.from_numpy(x.ravel()))
    chain.capture()
    for _ in range(2):
        chain.launch()
    chain.stream.synchronize()
    assert _lib.device_status() == 0
    assert chain.kernels_per_step == 1
    got = chain.y.cpu().numpy().reshape(N, -1)
    for n in sorted(set([0, N // 3, N // 2, N - 1])):
        want = oracle_chain(oracle, layers, x[n], "u8")
        assert np.array_equal(got[n], want), (n, got[n], want)
    assert len(np.unique(got[:, :classes])) > 1


@pytest.mark.parametrize("N", [1, 147, 149, 200, 296, 297], ids=lambda n: f"n{n}")
def test_every_image_of_a_batch(oracle, N):
    """All images, several batches one behind the other: groups of eight warps at one and at two images a CTA, where a warp may begin with
    half of a depthwise layer's sums, and the first batch of groups of four."""
    rng = np.random.default_rng(77)
    layers = _layers(rng, 25, 10, 4, 4, 2, 3, -128, 0, 12, 1024, "common")
    chain = networks.Chain(layers, N, "u8")
    chain.capture()
    for batch in range(3):
        x = P.pack_activation(rng.integers(0, 256, (N, 1, 25, 10), dtype=np.uint8))
        chain.stream.synchronize()
        chain.x.copy_(torch.from_numpy(x.ravel()))
        torch.cuda.current_stream().synchronize()
        for _ in range(5):
            chain.launch()
        chain.stream.synchronize()
        assert _lib.device_status() == 0
        got = chain.y.cpu().numpy().reshape(N, -1)
        want = np.stack([oracle_chain(oracle, layers, x[n], "u8") for n in range(N)])
        assert np.array_equal(got, want.reshape(N, -1)), np.flatnonzero((got != want.reshape(N, -1)).any(axis=1))


@pytest.mark.parametrize("how", ["written", "replaced", "replaced, then written", "untracked"])
def test_weights_changed_after_the_recording(oracle, how):
    """A launch computes with what the tensors of `params` hold then, as a network that runs layer by layer does."""
    rng = np.random.default_rng(11)
    old, new = (_layers(np.random.default_rng(s), 25, 10, 4, 4, 2, 2, -128, 0, 12, 1024, "common") for s in (1, 2))
    new = [dict(a, **{k: b[k] for k in ("w", "b") if k in b}) for a, b in zip(old, new)]  # other weights, the same quantisers
    chain = networks.Chain(old, 3, "u8")
    x = P.pack_activation(rng.integers(0, 256, (3, 1, 25, 10), dtype=np.uint8))
    chain.x.copy_(torch.from_numpy(x.ravel()))
    chain.capture()

    def run():
        torch.cuda.synchronize()
        chain.launch()
        chain.stream.synchronize()
        return chain.y.cpu().numpy().reshape(3, -1)

    want_old, want_new = (np.stack([oracle_chain(oracle, L, x[n], "u8") for n in range(3)]).reshape(3, -1) for L in (old, new))
    assert not np.array_equal(want_old, want_new)
    assert np.array_equal(run(), want_old)
    other = networks.Chain(new, 1, "u8").params
    if how.startswith("replaced"):
        chain.params[:] = [tuple(None if t is None else t.clone() for t in pair) for pair in other]
        chain.capture()
        assert np.array_equal(run(), want_new)
        if "written" in how:
            for mine, theirs in zip(chain.params, networks.Chain(old, 1, "u8").params):
                for a, b in zip(mine, theirs):
                    if a is not None:
                        a.copy_(b)
            assert np.array_equal(run(), want_old)
        return
    for mine, theirs in zip(chain.params, other):
        for a, b in zip(mine, theirs):
            if a is not None:
                (a.data if how == "untracked" else a).copy_(b)
    if how == "untracked":
        torch.cuda.synchronize()
        chain.prepare_whole()
    assert np.array_equal(run(), want_new)
    y = chain.enqueue()  # layer calls instead of the graph
    chain.stream.synchronize()
    assert np.array_equal(y.cpu().numpy().reshape(3, -1), want_new)


def test_networks_outside_the_one_kernel_form_run_layer_by_layer(oracle):
    """144 pixels do not fit a tile: the same list runs as its layers, with the same bytes."""
    rng = np.random.default_rng(5)
    layers = _layers(rng, 12, 12, 3, 3, 1, 1, -128, 0, 12, 1024, "common")
    chain = networks.Chain(layers, 2, "u8")
    assert chain.whole is None
    x = P.pack_activation(rng.integers(0, 256, (2, 1, 12, 12), dtype=np.uint8))
    chain.x.copy_(torch.from_numpy(x.ravel()))
    chain.capture()
    chain.launch()
    chain.stream.synchronize()
    got = chain.y.cpu().numpy().reshape(2, -1)
    for n in range(2):
        assert np.array_equal(got[n], oracle_chain(oracle, layers, x[n], "u8"))


@pytest.mark.parametrize("which", ["dense 3x3", "max pool"])
def test_other_operations_of_the_same_shapes_run_layer_by_layer(oracle, which):
    """A dense 3x3 layer has the descriptor of a depthwise one, a global max pool that of an average pool."""
    rng = np.random.default_rng(6)
    layers = _layers(rng, 25, 10, 4, 4, 2, 2, -128, 0, 12, 1024, "common")
    if which == "dense 3x3":
        layers[3].update(op="conv", w=rng.integers(0, 256, (64, 64, 3, 3)).astype(np.uint8))
    else:
        layers[-2] = {**layers[-2], "op": "maxpool"}
    chain = networks.Chain(layers, 2, "u8")
    assert chain.whole is None
    x = P.pack_activation(rng.integers(0, 256, (2, 1, 25, 10), dtype=np.uint8))
    chain.x.copy_(torch.from_numpy(x.ravel()))
    chain.capture()
    chain.launch()
    chain.stream.synchronize()
    got = chain.y.cpu().numpy().reshape(2, -1)
    for n in range(2):
        assert np.array_equal(got[n], oracle_chain(oracle, layers, x[n], "u8"))
