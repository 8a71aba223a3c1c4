"""The latency kernels: convolutions of a few million multiply-adds (small_b200_conv2d_f32_small) and the tail of a
classifier (small_b200_avgpool_dense_f32), against the oracle."""
import ctypes as C

import numpy as np
import pytest

from oracle.bindings import same_pads, shape
from smallframework_b200 import interface as S
from smallframework_b200 import packing as P
from smallframework_b200._lib import Layer, check, lib
from tests.gpu_util import CB, fbuf, oracle_conv_batch, oracle_layer, rel_max_err

CASES = [
    # C, K, H, W, Fh, Fw, stride, pads, batch
    (16, 16, 8, 8, 3, 3, 1, "same", 1),
    (32, 64, 16, 16, 3, 3, 2, "same", 3),
    (16, 32, 32, 32, 1, 1, 2, (0, 0, 0, 0), 2),
    (64, 64, 8, 8, 3, 3, 1, "same", 2),
    (48, 16, 11, 7, 5, 3, 1, (2, 2, 1, 1), 1),    # a last segment of 7 pixels, fewer pairs than a multiple of the warps
    (16, 48, 9, 17, 7, 7, 1, "same", 1),          # wider than the padding on both sides of a segment
    (256, 16, 1, 1, 1, 1, 1, (0, 0, 0, 0), 5),
    (3, 16, 32, 32, 3, 3, 1, "same", 2),          # first layers
    (3, 32, 33, 17, 3, 3, 2, "same", 2),
    (1, 16, 12, 10, 5, 4, 1, (2, 2, 1, 2), 1),
    (2, 16, 9, 9, 1, 1, 1, (0, 0, 0, 0), 1),
]


@pytest.mark.gpu
@pytest.mark.parametrize("case", CASES, ids=lambda c: "C{}_K{}_{}x{}_k{}x{}_s{}_n{}".format(*c[:7], c[8]))
@pytest.mark.parametrize("mode", ["plain", "partial_bias_leaky"])
def test_small_convolution(oracle, case, mode):
    c, k, h, w, fh, fw, s, pm, n = case
    pads = same_pads(h, w, fh, fw, s) if pm == "same" else pm
    rng = np.random.default_rng(c * k + h)
    x = P.pack_activation(rng.uniform(-1, 1, (n, c, h, w)).astype(np.float32))
    wt = P.pack_conv_filter(rng.normal(0, np.sqrt(2.0 / (c * fh * fw)), (k, c, fh, fw)).astype(np.float32))
    sh = shape(c, k, h, w, fh, fw, s, pads, CB)
    ho, wo = sh.out_hw()
    seed = rng.uniform(-1, 1, (n, k * ho * wo)).astype(np.float32)
    bias = rng.uniform(-0.5, 0.5, k).astype(np.float32)
    part = mode != "plain"
    L = Layer(n, c, k, h, w, fh, fw, s, *pads, int(part), S.ACT_LEAKY if part else 0, 0.1, 0, 0, 0, 0, 0, 0)
    assert lib().small_b200_conv2d_f32_small_preferred(C.byref(L))
    X, W, B, O = fbuf(x), fbuf(wt), fbuf(bias), fbuf(seed)
    check(lib().small_b200_conv2d_f32_small(C.byref(L), X.ptr(), W.ptr(), B.ptr() if part else None, O.ptr(), S._stream(None)))
    want = oracle_conv_batch(oracle, sh, x, wt, bias=bias, act=2, slope=0.1, seed=seed) if part else oracle_conv_batch(oracle, sh, x, wt)
    assert rel_max_err(O.numpy().reshape(n, -1), want) <= 1e-5


@pytest.mark.gpu
@pytest.mark.parametrize("case", [(64, 8, 8, 16, 3), (256, 3, 3, 16, 40), (16, 1, 1, 256, 2), (48, 5, 7, 32, 1)],
                         ids=lambda c: "C{}_{}x{}_K{}_n{}".format(*c))
@pytest.mark.parametrize("softmax", [0, 1])
def test_pool_dense_softmax(oracle, case, softmax):
    c, h, w, k, n = case
    rng = np.random.default_rng(c + k)
    x = P.pack_activation(rng.uniform(0, 1, (n, c, h, w)).astype(np.float32))
    wt = P.pack_conv_filter(rng.normal(0, np.sqrt(2.0 / c), (k, c, 1, 1)).astype(np.float32))
    bias = rng.uniform(-0.5, 0.5, k).astype(np.float32)
    pool = Layer(n, c, c, h, w, h, w, 1, 0, 0, 0, 0, 0, 0, 0.0, 0, 0, 0, 0, 0, 0)
    dense = Layer(n, c, k, 1, 1, 1, 1, 1, 0, 0, 0, 0, 0, 0, 0.0, 0, 0, 0, 0, 0, 0)
    assert lib().small_b200_avgpool_dense_f32_supported(C.byref(pool), C.byref(dense))
    X, W, B, O = fbuf(x), fbuf(wt), fbuf(bias), S.FloatBuffer(n * k)
    check(lib().small_b200_avgpool_dense_f32(C.byref(pool), C.byref(dense), softmax, X.ptr(), W.ptr(), B.ptr(), O.ptr(), S._stream(None)))
    got = O.numpy().reshape(n, -1)
    for i in range(n):
        want = oracle.pool2d_f32(shape(c, c, h, w, h, w, 1, (0, 0, 0, 0), CB), x[i], average=True)
        want = oracle.conv2d_f32(shape(c, k, 1, 1, 1, 1, 1, (0, 0, 0, 0), CB), want, wt, bias=bias)
        if softmax:
            want = oracle.softmax_f32(k, 1, 1, CB, want)
        assert rel_max_err(got[i], want) <= 1e-5


def test_layers_that_are_not_small():
    big = Layer(64, 64, 64, 32, 32, 3, 3, 1, 1, 1, 1, 1, 0, 0, 0.0, 0, 0, 0, 0, 0, 0)
    assert not lib().small_b200_conv2d_f32_small_preferred(C.byref(big))
    pool = Layer(1, 64, 64, 8, 8, 4, 4, 1, 0, 0, 0, 0, 0, 0, 0.0, 0, 0, 0, 0, 0, 0)
    dense = Layer(1, 64, 16, 1, 1, 1, 1, 1, 0, 0, 0, 0, 0, 0, 0.0, 0, 0, 0, 0, 0, 0)
    assert not lib().small_b200_avgpool_dense_f32_supported(C.byref(pool), C.byref(dense))  # not the whole image


@pytest.mark.gpu
@pytest.mark.parametrize("batch", [1, 21])
def test_residual_chain_never_works_in_place(oracle, batch):
    """A shortcut convolution behind an alias reads one buffer and writes another, and the chain gives what the oracle gives."""
    import torch
    from smallframework_b200 import networks
    layers = networks.resnet8(seed=0)
    chain = networks.Chain(layers, batch, "f32")
    assert all(io is None or L["op"] == "alias" or io[0].data_ptr() != io[1].data_ptr() for L, io in zip(layers, chain.io_plan()))
    x = np.random.default_rng(batch).uniform(0, 1, (batch, chain.x.numel() // batch)).astype(np.float32)
    chain.x.copy_(torch.from_numpy(x.reshape(-1)))
    torch.cuda.synchronize()
    chain.enqueue()
    torch.cuda.synchronize()
    got = chain.y.cpu().numpy().reshape(batch, -1)
    for n in (0, batch // 2, batch - 1):
        named, cur = {"in": x[n]}, None
        for i, L in enumerate(layers):
            if L["op"] == "alias":
                named[L["dst"]] = named[L["src"]]
                continue
            seed = named[L["dst"]].copy() if L.get("accumulate") else None
            cur = named[L["dst"]] = oracle_layer(oracle, L, i == 0, named[L["src"]], seed=seed)
        assert rel_max_err(got[n, :cur.size], cur) <= 2e-5
