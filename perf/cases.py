"""What this framework is timed on: whole networks through the graph executor and the Darknet
model, and single layers through the functional interface, at batch sizes from one image to the
configurations' own.

Inputs come from the seed; a network's weights are fixed, as they are in a deployed model, and are
laid out once in prepare().  Outputs are the tensors a caller reads: every head of a network, every
layer's tensor where layers are called one by one.
"""
import functools
import math

import numpy as np
import torch

from smallframework_b200 import darknet, networks
from smallframework_b200 import interface as S
from smallframework_b200.packing import calc_padding

# Largest batch of each network's configuration (Tiny-YOLOv2: its share of one GPU).
MAX_BATCH = {"resnet8": 1024, "dscnn": 4096, "mobilenet": 2048, "tinyyolov2": 64, "yolov3tiny": 16}
MOBILENET_SIZES = (64, 96, 128)


def listed():
    return [
        # One image at a time: a sensor or camera whose answer is waited for.
        dict(name="resnet8_f32_b1", kind="resnet8", dtype="f32", batch=1, size=32),
        dict(name="dscnn_u8_b1", kind="dscnn", dtype="u8", batch=1, size=49),
        dict(name="tinyyolov2_f32_b1", kind="tinyyolov2", dtype="f32", batch=1, size=416),
        # A few camera streams through a Darknet detector (routes, upsampling, two heads).
        dict(name="yolov3tiny_f32_b3", kind="yolov3tiny", dtype="f32", batch=3, size=416),
        # The configurations' own batches: throughput serving.
        dict(name="resnet8_f32_b1024", kind="resnet8", dtype="f32", batch=1024, size=32),
        dict(name="dscnn_u8_b4096", kind="dscnn", dtype="u8", batch=4096, size=49),
        dict(name="mobilenet_f32_b2048", kind="mobilenet", dtype="f32", batch=2048, size=96),
        dict(name="mobilenet_u8_b2048", kind="mobilenet", dtype="u8", batch=2048, size=96),
        dict(name="tinyyolov2_f32_b64", kind="tinyyolov2", dtype="f32", batch=64, size=416),
        # The 13 convolution shapes of YOLOv3-tiny, called one by one.
        dict(name="convs_f32_b32", kind="convs", dtype="f32", batch=32, size=416),
        # Layers called one by one on ragged images: depthwise, pools, activations, shortcut add,
        # upsampling, concatenation, a strided convolution.
        dict(name="layers_f32_c96_57x57_b32", kind="layers", dtype="f32", batch=32, C=96, H=57, W=57),
        # The same for uint8, with the zero points an asymmetric quantisation ends up with.
        dict(name="layers_u8_c64_45x37_b48", kind="layers", dtype="u8", batch=48, C=64, H=45, W=37,
             zero_in=-113, zero_filt=-121),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    known = [{k: v for k, v in c.items() if k != "name"} for c in listed()]
    while True:
        case = _draw(rng)
        if case not in known:
            return case


def _draw(rng):
    kind = rng.choice(["resnet8", "dscnn", "mobilenet", "mobilenet", "tinyyolov2", "tinyyolov2", "yolov3tiny",
                       "convs", "layers", "layers"])
    if kind == "layers":
        # up to the listed cases' elements per tensor
        C, H, W = 16 * _log_int(rng, 1, 16), _log_int(rng, 7, 112), _log_int(rng, 7, 112)
        case = dict(kind=kind, dtype=rng.choice(["f32", "u8"]), C=C, H=H, W=W)
        limit = 10e6 if case["dtype"] == "f32" else 5e6
        case["batch"] = _log_int(rng, 1, max(1, min(256, int(limit / (C * H * W)))))
        if case["dtype"] == "u8":
            case["zero_in"] = rng.choice([0, -128, -113, -7])
            case["zero_filt"] = rng.choice([-128, -128, -121, -133])
        return case
    case = dict(kind=kind, dtype="f32")
    if kind == "convs":
        case["size"] = rng.randint(96, 416)
        case["batch"] = _log_int(rng, 1, 32)
        return case
    case["batch"] = _log_int(rng, 1, MAX_BATCH[kind])
    case["size"] = 32
    if kind == "dscnn":
        case.update(dtype="u8", size=49)
    elif kind == "mobilenet":
        case.update(dtype=rng.choice(["f32", "u8"]), size=rng.choice(MOBILENET_SIZES))
        case["batch"] = min(case["batch"], MAX_BATCH[kind] * 96 ** 2 // case["size"] ** 2)
    elif kind in ("tinyyolov2", "yolov3tiny"):
        case["size"] = 32 * rng.randint(5, 13)
    return case


# --------------------------------------------------------------------------- networks
@functools.lru_cache(maxsize=None)
def _network(kind, dtype, size):
    if kind == "resnet8":
        return networks.resnet8(seed=0, size=size)
    if kind == "dscnn":
        return networks.ds_cnn(seed=1)
    if kind == "mobilenet":
        return networks.mobilenet_v1_025(seed=2, size=size, dtype=dtype)
    return networks.tiny_yolov2(seed=4, size=size)


@functools.lru_cache(maxsize=None)
def _convs(size):
    return [layers[0] for layers in networks.yolov3_tiny_convs(seed=3, size=size)]


@functools.lru_cache(maxsize=None)
def _serving_stream():
    """A serving process runs its requests in order on one stream."""
    return torch.cuda.Stream()


def _yolov3_tiny_cfg(size):
    """The YOLOv3-tiny graph: a pyramid of six convolutions with pools, a head on the coarse grid, and a
    second head behind an upsampling that is concatenated with the fifth convolution."""
    text = [f"[net]\nwidth={size}\nheight={size}\nchannels=3\n"]

    def conv(filters, kernel, linear=False):
        text.append("[convolutional]\n%sfilters=%d\nsize=%d\nstride=1\npad=1\nactivation=%s\n" % (
            "" if linear else "batch_normalize=1\n", filters, kernel, "linear" if linear else "leaky"))

    def yolo(mask):
        text.append("[yolo]\nmask = %s\nanchors = 10,14,  23,27,  37,58,  81,82,  135,169,  344,319\n"
                    "classes=80\nnum=6\n" % mask)

    for i, filters in enumerate((16, 32, 64, 128, 256, 512)):
        conv(filters, 3)                                            # records 0, 2, 4, 6, 8, 10
        text.append("[maxpool]\nsize=2\nstride=%d\n" % (2 if i < 5 else 1))
    conv(1024, 3)                                                   # 12
    conv(256, 1)                                                    # 13
    conv(512, 3)
    conv(255, 1, linear=True)
    yolo("3,4,5")
    text.append("[route]\nlayers = 13\n")
    conv(128, 1)
    text.append("[upsample]\nstride=2\n")
    text.append("[route]\nlayers = -1, 8\n")
    conv(256, 3)
    conv(255, 1, linear=True)
    yolo("0,1,2")
    return "\n".join(text)


@functools.lru_cache(maxsize=None)
def _darknet_weights():
    return darknet.random_weights(_yolov3_tiny_cfg(416), seed=3)


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _uniform(n, gen, lo=0.0, hi=1.0):
    return torch.rand(n, generator=gen, device="cuda") * (hi - lo) + lo


def _bytes(n, gen):
    return torch.randint(0, 256, (n,), generator=gen, device="cuda", dtype=torch.uint8)


def _prepare_network(case, gen):
    layers = _network(case["kind"], case["dtype"], case["size"])
    chain = networks.Chain(layers, case["batch"], case["dtype"])
    chain.stream = _serving_stream()
    n = chain.x.numel()
    chain.x.copy_(_uniform(n, gen) if case["dtype"] == "f32" else _bytes(n, gen))
    torch.cuda.synchronize()
    chain.capture()
    return dict(chain=chain)


def _prepare_darknet(case, gen):
    model = darknet.DarknetModel(_yolov3_tiny_cfg(case["size"]), _darknet_weights(), batch=case["batch"])
    return dict(model=model, x=_uniform(model.x.numel(), gen))


# --------------------------------------------------------------------------- layers called one by one
def _prepare_convs(case, gen):
    calls = []
    for i, L in enumerate(_convs(case["size"])):
        w, b = networks.padded_params(L, i == 0, "f32")
        k, c = networks.padded(L["K"]), L["C"]
        geo = (L["Fh"], L["Fw"], L["stride"], *L["pads"], k, c, L["H"], L["W"])
        x = S.FloatBuffer(data=_uniform(case["batch"] * c * L["H"] * L["W"], gen, -1.0, 1.0))
        filt, bias = S.FloatBuffer(data=w), S.FloatBuffer(data=b)
        out = S.FloatBuffer(case["batch"] * k * L["H"] * L["W"])
        tensor = c % 16 == 0 and S.tf32x3_supported(*geo)
        if tensor:
            packed, filt = filt, S.FloatBuffer(2 * filt.size())
            S.prepare_filter_3xTF32(L["Fh"], L["Fw"], k, c, packed, filt)
        act = dict(activation=L["act"], negative_slope=L["slope"], batch=case["batch"])
        calls.append((S.Conv2D_3xTF32 if tensor else S.Conv2D_Bias_Activation, geo, (x, filt, bias, out), act))
    return dict(calls=calls)


def _run_convs(state):
    for fn, geo, buffers, act in state["calls"]:
        fn(*geo, *buffers, **act)
    return [buffers[3].data() for _, _, buffers, _ in state["calls"]]


def _half(n):
    return n // 2


def _same(H, W, f, s):
    return (*calc_padding(H, f, s), *calc_padding(W, f, s))


def _strided(n):
    return -(-n // 2)


def _prepare_layers_f32(case, gen):
    n, C, H, W = case["batch"], case["C"], case["H"], case["W"]
    Hp, Wp, Hs, Ws = _half(H), _half(W), _strided(H), _strided(W)
    buf = lambda k: S.FloatBuffer(k)
    normal = lambda k, fan: S.FloatBuffer(data=torch.randn(k, generator=gen, device="cuda") * math.sqrt(2.0 / fan))
    return dict(case=case, x=S.FloatBuffer(data=_uniform(n * C * H * W, gen, -1.0, 1.0)),
                dw1=normal(C * 9, 9), dw2=normal(C * 9, 9), bias=S.FloatBuffer(data=_uniform(C, gen, -0.1, 0.1)),
                conv=normal(2 * C * C * 9, 9 * C), conv_bias=S.FloatBuffer(data=_uniform(2 * C, gen, -0.1, 0.1)),
                a=buf(n * C * H * W), act=buf(n * C * H * W), b=buf(n * C * Hs * Ws), d=buf(n * 2 * C * Hs * Ws),
                mx=buf(n * C * Hp * Wp), avg=buf(n * C * Hp * Wp), cat=buf(n * 2 * C * Hp * Wp),
                up=buf(n * C * 4 * Hp * Wp))


def _run_layers_f32(s):
    q = s["case"]
    n, C, H, W = q["batch"], q["C"], q["H"], q["W"]
    S.DepthwiseConv2D_Bias_Activation(3, 3, 1, *_same(H, W, 3, 1), C, H, W, s["x"], s["dw1"], s["bias"], s["a"],
                                      activation=S.ACT_RELU, batch=n)
    S.Accum(C, H, W, s["x"], s["a"], batch=n)
    S.LeakyReLUActivation(C, H, W, s["a"], 0.1, s["act"], batch=n)
    S.DepthwiseConv2D(3, 3, 2, *_same(H, W, 3, 2), C, H, W, s["act"], s["dw2"], s["b"], batch=n)
    S.Conv2D_Bias_ReLU(3, 3, 2, *_same(H, W, 3, 2), 2 * C, C, H, W, s["act"], s["conv"], s["conv_bias"], s["d"], batch=n)
    S.MaxPool2D(2, 2, 2, 0, 0, 0, 0, C, H, W, s["act"], s["mx"], batch=n)
    S.AveragePool2D(2, 2, 2, 0, 0, 0, 0, C, H, W, s["act"], s["avg"], batch=n)
    S.Concat(C, C, _half(H), _half(W), s["mx"], s["avg"], s["cat"], batch=n)
    S.UpSample2D(2, C, _half(H), _half(W), s["mx"], s["up"], batch=n)
    return {k: s[k].data() for k in ("a", "act", "b", "d", "mx", "avg", "cat", "up")}


def _quantise(buf, scale, zero=0):
    """A buffer's fields for a requantisation by `scale`: multiplier * 2^-31 * 2^(lshift - rshift)."""
    m, e = math.frexp(scale)
    buf.multiplier = min(int(round(m * (1 << 31))), (1 << 31) - 1)
    buf.lshift, buf.rshift = max(e, 0), max(-e, 0)
    buf.m_zero = zero
    return buf


def _prepare_layers_u8(case, gen):
    n, C, H, W = case["batch"], case["C"], case["H"], case["W"]
    Hp, Wp, Hs, Ws = _half(H), _half(W), _strided(H), _strided(W)
    zi, zf = case["zero_in"], case["zero_filt"]
    src = lambda k, zero: _quantise(S.QUInt8Buffer(data=_bytes(k, gen)), 1.0, zero)
    # sums of `taps` products of bytes of variance 74^2 land in 0..255
    dst = lambda k, taps: _quantise(S.QUInt8Buffer(k), 64.0 / (74.0 * 74.0 * math.sqrt(taps)), zi)
    return dict(case=case, x=src(n * C * H * W, zi), conv=src(C * C * 9, zf), pw=src(2 * C * C, zf), dw=src(C * 9, zf),
                down=src(2 * C * C * 9, zf),
                a=dst(n * C * H * W, 9 * C), b=dst(n * C * H * W, 9), c=dst(n * 2 * C * H * W, C),
                d=dst(n * 2 * C * Hs * Ws, 9 * C), mx=dst(n * C * Hp * Wp, 1), r=_quantise(S.QUInt8Buffer(n * C * H * W), 0.7))


def _run_layers_u8(s):
    q = s["case"]
    n, C, H, W = q["batch"], q["C"], q["H"], q["W"]
    S.Conv2D(3, 3, 1, *_same(H, W, 3, 1), C, C, H, W, s["x"], s["conv"], s["a"], batch=n)
    S.DepthwiseConv2D(3, 3, 1, *_same(H, W, 3, 1), C, H, W, s["a"], s["dw"], s["b"], batch=n)
    S.Conv2D(1, 1, 1, 0, 0, 0, 0, 2 * C, C, H, W, s["b"], s["pw"], s["c"], batch=n)
    S.Conv2D(3, 3, 2, *_same(H, W, 3, 2), 2 * C, C, H, W, s["b"], s["down"], s["d"], batch=n)
    S.MaxPool2D(2, 2, 2, 0, 0, 0, 0, C, H, W, s["a"], s["mx"], batch=n)
    S.ReLUActivation(C, H, W, s["x"], s["r"], batch=n)
    return {k: s[k].data() for k in ("a", "b", "c", "d", "mx", "r")}


# --------------------------------------------------------------------------- the interface of this file
def prepare(case, seed):
    gen = _generator(seed)
    if case["kind"] == "yolov3tiny":
        return dict(_prepare_darknet(case, gen), run=_run_darknet)
    if case["kind"] == "convs":
        return dict(_prepare_convs(case, gen), run=_run_convs)
    if case["kind"] == "layers":
        f32 = case["dtype"] == "f32"
        return dict((_prepare_layers_f32 if f32 else _prepare_layers_u8)(case, gen),
                    run=_run_layers_f32 if f32 else _run_layers_u8)
    return dict(_prepare_network(case, gen), run=_run_network)


def _run_network(state):
    state["chain"].launch()
    return state["chain"].y


def _run_darknet(state):
    return state["model"].inference(state["x"])


def run(state):
    return state["run"](state)


def _sum_work(layers, batch, elt, chained):
    """Every convolution's multiply-adds; first input and last output (all of them for layers that are
    called one by one), weights once."""
    flops = nbytes = 0
    for L in layers:
        f, a, w = networks.algorithmic_work(L, elt)
        flops += f * batch
        nbytes += w + (0 if chained else a * batch)
    if chained:
        k, ho, wo = networks.output_shape(layers)
        nbytes += batch * elt * (math.prod(networks.input_shape(layers)) + k * ho * wo)
    return dict(bytes=nbytes, flops=flops)


def work(case):
    n, elt = case["batch"], 4 if case["dtype"] == "f32" else 1
    if case["kind"] == "convs":
        return _sum_work(_convs(case["size"]), n, elt, False)
    if case["kind"] == "yolov3tiny":
        (c, h, w), plan, floats = darknet.build_plan(_yolov3_tiny_cfg(case["size"]))
        flops = sum(2 * r["Ho"] * r["Wo"] * r["K"] * r["C"] * r["size"] ** 2 for r in plan if r["op"] == "conv")
        heads = sum(r["preds"] * (r["classes"] + 5) for r in plan if r["op"] == "yolo")
        return dict(bytes=4 * (n * (c * h * w + heads) + floats), flops=n * flops)
    if case["kind"] == "layers":
        C, H, W = case["C"], case["H"], case["W"]
        full, strided, pooled = C * H * W, C * _strided(H) * _strided(W), C * _half(H) * _half(W)
        if case["dtype"] == "f32":
            return dict(bytes=4 * (n * (3 * full + 3 * strided + 8 * pooled) + 18 * C * C),
                        flops=n * (2 * 9 * full + 3 * full + 2 * 9 * strided + 2 * 2 * 9 * C * strided + 8 * pooled))
        return dict(bytes=n * (6 * full + 2 * strided + pooled) + 29 * C * C,
                    flops=n * (2 * 9 * C * full + 2 * 9 * full + 2 * 2 * C * full + 2 * 2 * 9 * C * strided + 4 * pooled))
    return _sum_work(_network(case["kind"], case["dtype"], case["size"]), n, elt, True)


def tolerance(case):
    if case["dtype"] == "u8":
        return "exact"  # bytes
    # one fp32 sum per value where layers are called one by one; some ten to thirty sums deep in a network
    return {"rel": 1e-5} if case["kind"] in ("convs", "layers") else {"rel": 2e-5}
