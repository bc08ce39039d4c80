"""The work a user of this package gives it, as measurable cases: single quantized operators over the range of sizes they are
called with, and the two whole networks of the package's benchmark (int8 ResNet-50 v1.5 and one layer of the int8
BERT-base-shaped encoder), each through the public entry points: `ngraph_b200.ops` where it has a wrapper, the C ABI
(`ngraph_b200.lib`) otherwise.

Data are synthetic and seeded: activations as the layers in question see them (post-ReLU codes, normally distributed hidden
states, normalised images), random weights quantised per output channel, and scales that spread the results over their range.
"""
import ctypes
import math

import torch

from ngraph_b200 import ops
from ngraph_b200.lib import F32, I8, LIB, U8, Epilogue, check

DTYPES = {"u8": torch.uint8, "i8": torch.int8, "f32": torch.float32}
CODES = {"u8": U8, "i8": I8, "f32": F32}
DIV, MUL, ADD, MAX_ABS = 3, 2, 0, 3          # b200_f32_op / b200_reduce_op
BLOCKS = ((3, 64, 256, 1), (4, 128, 512, 2), (6, 256, 1024, 2), (3, 512, 2048, 2))  # ResNet-50: blocks, mid, out, stride


def listed():
    return [
        # the activations of a small layer, one scale per tensor (the layer below takes 1024 features for 256 rows): latency
        {"name": "quantize_1mb", "kind": "quantize", "n": 1, "c": 64, "h": 64, "w": 64, "type": "i8", "per_channel": False, "mode": 4},
        # feature maps with an odd image size, one scale per channel: rows that start at any alignment
        {"name": "quantize_odd_channels", "kind": "quantize", "n": 24, "c": 64, "h": 113, "w": 113, "type": "u8", "per_channel": True, "mode": 4},
        # the streaming end of the range: 1 GB of f32, one scale per tensor, a half-way mode other than round-to-even
        {"name": "quantize_1gb", "kind": "quantize", "n": 64, "c": 64, "h": 256, "w": 256, "type": "u8", "per_channel": False, "mode": 0},
        # codes back to f32 at the edge of a quantized region, one scale per channel
        {"name": "dequantize_256mb", "kind": "dequantize", "n": 64, "c": 64, "h": 128, "w": 128, "type": "i8", "per_channel": True},
        # QuantizedDotBias + ReLU of a small fully connected layer, weights given at run time
        {"name": "dot_256_1024", "kind": "dot", "m": 256, "n": 1024, "k": 1024, "data": "i8", "out": "i8", "relu": True, "core": False, "packed": False},
        # the classifier of an image network (QuantizedDot with its own rounding), a width that no tile divides
        {"name": "dot_fc_1000", "kind": "dot", "m": 128, "n": 1000, "k": 2048, "data": "u8", "out": "i8", "relu": False, "core": True, "packed": True},
        # the wide product of a transformer's feed-forward block over a full batch, f32 results
        {"name": "dot_ffn", "kind": "dot", "m": 24576, "n": 3072, "k": 768, "data": "i8", "out": "f32", "relu": False, "core": False, "packed": True},
        # QuantizedConvolutionBias + ReLU, the single-layer configuration of the benchmark
        {"name": "conv3x3_64", "kind": "conv", "n": 32, "h": 56, "w": 56, "c": 64, "k": 64, "r": 3, "stride": 1, "residual": False},
        # a whole image network, one image at a time: an interactive service, where launches and host time count
        {"name": "resnet50_1", "kind": "resnet50", "n": 1, "h": 224, "w": 224},
        # the same network at the benchmark's batch: throughput
        {"name": "resnet50_128", "kind": "resnet50", "n": 128, "h": 224, "w": 224},
        # one layer of the encoder on one short sequence
        {"name": "encoder_1x128", "kind": "encoder", "n": 1, "seq": 128, "hidden": 768, "ffn": 3072},
        # one layer of the encoder at the benchmark's batch and sequence length
        {"name": "encoder_64x384", "kind": "encoder", "n": 64, "seq": 384, "hidden": 768, "ffn": 3072},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["quantize", "quantize", "dequantize", "dot", "dot", "conv", "conv", "resnet50", "encoder"])
    if kind in ("quantize", "dequantize"):
        # 1 MB to 1 GB of f32 in feature maps of 64 channels, square or not, odd sizes as they come
        elements = _log(rng, 1 << 18, 1 << 28)
        h = min(_log(rng, 14, 256), max(1, elements // 64))
        w = max(1, min(h + rng.randint(-3, 3), elements // (64 * h)))
        case = {"kind": kind, "n": max(1, elements // (64 * h * w)), "c": 64, "h": h, "w": w, "type": rng.choice(["u8", "i8"]),
                "per_channel": rng.random() < 0.5}
        if kind == "quantize":
            case["mode"] = 4 if rng.random() < 0.5 else rng.randrange(9)
        return case
    if kind == "dot":
        m, n, k = _log(rng, 1, 32768), _log(rng, 16, 4096), 16 * _log(rng, 4, 256)
        while m * n * k > 24576 * 3072 * 768 or m * n > 24576 * 3072:
            m = max(1, m // 2)
        core = rng.random() < 0.25
        return {"kind": "dot", "m": m, "n": n, "k": k, "data": rng.choice(["u8", "i8"]), "out": rng.choice(["u8", "i8"] if core else ["u8", "i8", "f32"]),
                "relu": not core and rng.random() < 0.5, "core": core, "packed": rng.random() < 0.5}
    if kind == "conv":
        h = _log(rng, 7, 56)
        r = rng.choice([1, 3])
        c, k = 64 * rng.choice([1, 2, 4, 8]), 16 * _log(rng, 2, 64)
        n = _log(rng, 1, 128)
        while n > 1 and n * h * h * max(k, c) > 128 * 56 * 56 * 256:
            n //= 2
        return {"kind": "conv", "n": n, "h": h, "w": max(7, h + rng.randint(-2, 2)), "c": c, "k": k, "r": r, "stride": rng.choice([1, 1, 2]),
                "residual": rng.random() < 0.4}
    if kind == "resnet50":
        return {"kind": "resnet50", "n": _log(rng, 1, 128), "h": 16 * rng.randint(6, 14), "w": 16 * rng.randint(6, 14)}
    # from about one short sequence (128 tokens) to the benchmark's 24576 tokens
    tokens, seq = _log(rng, 160, 24576), _log(rng, 24, 384)
    hidden, ffn = rng.choice([(768, 3072), (512, 2048)])
    return {"kind": "encoder", "n": max(-(-160 // seq), tokens // seq), "seq": seq, "hidden": hidden, "ffn": ffn}


# ------------------------------------------------------------------------------------------------ inputs
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _activations(shape, name, g):
    """codes as a quantized layer passes them on: half of them zero after a ReLU (u8), or both signs (i8)"""
    x = torch.randn(shape, generator=g, device="cuda") * 42.0
    return x.clamp_(0, 255).to(torch.uint8) if name == "u8" else x.clamp_(-127, 127).to(torch.int8)


def _weights(rows, cols, g):
    """(int8 [rows, cols] with the largest of each row at +-127, the per-row scale of normally distributed weights)"""
    w = torch.randn((rows, cols), generator=g, device="cuda")
    s = w.abs().amax(dim=1, keepdim=True) / 127.0
    return (w / s).round_().to(torch.int8), s.reshape(-1)


def _requant_scale(w, spread, mean_square):
    """per-row scale that brings sum(a * w) over activations of this mean square to a standard deviation of `spread` codes"""
    return (spread / (w.float().square().sum(dim=1) * mean_square).sqrt()).contiguous()


def _stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def _i64(v):
    return (ctypes.c_int64 * max(len(v), 1))(*v)


def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, _generator(seed))


def run(state):
    return state["run"](state)


# ------------------------------------------------------------------------------------------------ Quantize / Dequantize
def _scale_zp(case, g):
    if case["per_channel"]:
        u = torch.rand(case["c"], generator=g, device="cuda")
        scale = torch.exp(u * math.log(100.0) + math.log(1e-3))  # log-uniform in [1e-3, 1e-1]
    else:
        scale = torch.full((), 0.05, device="cuda")
    zp = torch.full(scale.shape, 128 if case["type"] == "u8" else 0, device="cuda").to(DTYPES[case["type"]])
    return scale, zp, (1,) if case["per_channel"] else ()


def _prepare_quantize(case, g):
    x = torch.randn((case["n"], case["c"], case["h"], case["w"]), generator=g, device="cuda")
    scale, zp, axes = _scale_zp(case, g)
    return {"run": _run_quantize, "x": x, "scale": scale, "zp": zp, "axes": axes, "mode": case["mode"]}


def _run_quantize(s):
    return ops.quantize(s["x"], s["scale"], s["zp"], axes=s["axes"], round_mode=s["mode"])


def _prepare_dequantize(case, g):
    shape = (case["n"], case["c"], case["h"], case["w"])
    lo, hi = (0, 256) if case["type"] == "u8" else (-128, 128)
    x = torch.randint(lo, hi, shape, generator=g, device="cuda", dtype=DTYPES[case["type"]])
    scale, zp, axes = _scale_zp(case, g)
    return {"run": _run_dequantize, "x": x, "scale": scale, "zp": zp, "axes": axes}


def _run_dequantize(s):
    return ops.dequantize(s["x"], s["scale"], s["zp"], axes=s["axes"])


# ------------------------------------------------------------------------------------------------ QuantizedDot / QuantizedDotBias
def _epilogue(scale, out, bias=None, relu=False, core=False, out_zp=0):
    e = Epilogue()
    e.scale, e.scale_count = scale.data_ptr(), scale.numel()
    e.bias = None if bias is None else bias.data_ptr()
    e.relu, e.round_half_away, e.out_zero_point, e.out_type = int(relu), int(core), out_zp, CODES[out]
    return e


def _prepare_dot(case, g):
    m, n, k = case["m"], case["n"], case["k"]
    a = _activations((m, k), case["data"], g)
    w, _ = _weights(n, k, g)
    scale = _requant_scale(w, 40.0, 42.0 ** 2 * (0.5 if case["data"] == "u8" else 1.0))
    if case["out"] == "f32":
        scale = scale * 0.025
    if case["core"]:
        scale = scale.mean().reshape(1)
    bias = None if case["core"] else torch.randint(-1000, 1001, (n,), generator=g, device="cuda", dtype=torch.int32)
    zp = 0 if case["out"] != "u8" or not case["core"] else 128
    s = {"a": a, "w": w, "scale": scale, "bias": bias, "relu": case["relu"], "core": case["core"], "zp": zp, "out": DTYPES[case["out"]], "case": case}
    if case["packed"]:
        s.update(run=_run_dot_packed, w=ops.pack_weights(w, 128), data=CODES[case["data"]], e=_epilogue(scale, case["out"], bias, case["relu"], case["core"], zp))
    else:
        s["run"] = _run_dot
    return s


def _run_dot(s):
    return ops.qgemm(s["a"], s["w"], s["scale"], s["out"], bias=s["bias"], relu=s["relu"], core=s["core"], out_zp=s["zp"])


def _run_dot_packed(s):
    c = s["case"]
    out = torch.empty((c["m"], c["n"]), dtype=s["out"], device="cuda")
    check(LIB.b200_qgemm_packed(s["a"].data_ptr(), s["data"], s["w"].data_ptr(), out.data_ptr(), c["m"], c["n"], c["k"], ctypes.byref(s["e"]), _stream()), "qgemm")
    return out


# ------------------------------------------------------------------------------------------------ QuantizedConvolutionBias (+Relu / +Add)
def _conv_layer(g, n, h, w, c, k, r, stride, mean_square, spread=60.0):
    """what a program keeps for one convolution: packed filters, scales, bias and geometry"""
    filt, _ = _weights(k, r * r * c, g)
    return {"filt": ops.pack_weights(filt, LIB.b200_qconv_weight_block(c)), "scale": _requant_scale(filt, spread, mean_square),
            "bias": torch.randint(-1000, 1001, (k,), generator=g, device="cuda", dtype=torch.int32),
            "cp": ops.conv_params((n, h, w, c), (k, r, r, c), (stride, stride), (r // 2, r // 2))}


def _prepare_conv(case, g):
    layer = _conv_layer(g, case["n"], case["h"], case["w"], case["c"], case["k"], case["r"], case["stride"], 42.0 ** 2 / 2)
    p, q = ops.conv_out_hw(layer["cp"])
    s = {"run": _run_conv, "x": _activations((case["n"], case["h"], case["w"], case["c"]), "u8", g), "layer": layer, "sum": None, "sum_scale": None}
    if case["residual"]:
        s["sum"], s["sum_scale"] = _activations((case["n"], p, q, case["k"]), "u8", g), torch.full((1,), 0.7, device="cuda")
    return s


def _conv(layer, x, out=torch.uint8, relu=True, sum_in=None, sum_scale=None):
    return ops.qconv(x, layer["filt"], layer["scale"], out, layer["cp"], bias=layer["bias"], relu=relu, sum_in=sum_in, sum_scale=sum_scale, packed="prepacked")


def _run_conv(s):
    return _conv(s["layer"], s["x"], sum_in=s["sum"], sum_scale=s["sum_scale"])


# ------------------------------------------------------------------------------------------------ int8 ResNet-50 v1.5
def _prepare_resnet50(case, g):
    n, h, w = case["n"], case["h"], case["w"]
    mean = torch.tensor([0.485, 0.456, 0.406], device="cuda").reshape(1, 3, 1, 1)
    std = torch.tensor([0.229, 0.224, 0.225], device="cuda").reshape(1, 3, 1, 1)
    x = ((torch.rand((n, 3, h, w), generator=g, device="cuda") - mean) / std).contiguous()
    p, q, _, _, rc = ops.stem_geometry(h, w, 7, 7, (3, 3), (3, 3))
    filt, _ = _weights(64, 3 * 49, g)
    kcrs = filt.reshape(64, 3, 7, 7).cpu().numpy()
    packed = torch.empty((64, rc * 64), dtype=torch.int8)
    check(LIB.b200_stem_pack_filter_host(kcrs.ctypes.data, packed.data_ptr(), 64, 3, 7, 7, 3, 3), "stem filter")
    scale = _requant_scale(filt, 60.0, 55.0 ** 2)
    bias = torch.randint(-1000, 1001, (64,), generator=g, device="cuda", dtype=torch.int32)
    s = {"run": _run_resnet50, "x": x, "case": case, "pq": (p, q), "stem": packed.cuda(), "stem_scale": scale, "stem_bias": bias,
         "stem_e": _epilogue(scale, "u8", bias, True), "x_scale": torch.full((1,), 2.64 / 127, device="cuda"),
         "x_zp": torch.zeros(1, dtype=torch.int8, device="cuda"), "sum_scale": torch.full((1,), 0.8, device="cuda"),
         "cells": torch.empty(LIB.b200_stem_cells_bytes(n, h, w, 7, 7, 3, 3, 3, 3), dtype=torch.uint8, device="cuda"), "blocks": []}
    h, w, cin, ms = (p + 1) // 2, (q + 1) // 2, 64, 60.0 ** 2  # after the 3x3 / stride 2 MaxPool the codes are larger
    for blocks, mid, cout, first in BLOCKS:
        for b in range(blocks):
            stride = first if b == 0 else 1
            block = {"down": _conv_layer(g, n, h, w, cin, cout, 1, stride, ms, 40.0) if b == 0 else None,
                     "c1": _conv_layer(g, n, h, w, cin, mid, 1, 1, ms), "c2": _conv_layer(g, n, h, w, mid, mid, 3, stride, 60.0 ** 2 / 2)}
            h, w = (h - 1) // stride + 1, (w - 1) // stride + 1
            block["c3"] = _conv_layer(g, n, h, w, mid, cout, 1, 1, 60.0 ** 2 / 2, 40.0)
            s["blocks"].append(block)
            cin, ms = cout, 55.0 ** 2
    fc, _ = _weights(1000, 2048, g)
    s.update(fc=fc, fc_scale=(40.0 / (fc.float().square().sum(dim=1).mean() * 60.0 ** 2).sqrt()).reshape(1), s_feat=torch.full((1,), 0.02, device="cuda"),
             s_pool=torch.full((1,), 0.01, device="cuda"), s_logits=torch.full((), 0.1, device="cuda"), zp=torch.zeros((), dtype=torch.int8, device="cuda"))
    return s


def _run_resnet50(s):
    n, h, w = s["case"]["n"], s["case"]["h"], s["case"]["w"]
    p, q = s["pq"]
    check(LIB.b200_stem_pack_input_f32(s["x"].data_ptr(), s["x_scale"].data_ptr(), s["x_zp"].data_ptr(), I8, 4, s["cells"].data_ptr(), n, 3, h, w, 7, 7,
                                       3, 3, 3, 3, _stream()), "stem input")
    a = torch.empty((n, p, q, 64), dtype=torch.uint8, device="cuda")
    check(LIB.b200_qconv_stem(s["cells"].data_ptr(), I8, s["stem"].data_ptr(), a.data_ptr(), n, h, w, 64, 7, 7, 3, 3, 3, 3, ctypes.byref(s["stem_e"]),
                              _stream()), "stem")
    a = ops.maxpool_nhwc(a, (3, 3), (2, 2), (1, 1))
    for block in s["blocks"]:
        y = _conv(block["c2"], _conv(block["c1"], a))
        if block["down"] is not None:  # the signed shortcut: QuantizedConvolutionBiasSignedAdd gives i8, the ReLU leaves it non-negative
            a = _conv(block["c3"], y, torch.int8, True, _conv(block["down"], a, torch.int8, False), s["sum_scale"]).view(torch.uint8)
        else:
            a = _conv(block["c3"], y, sum_in=a, sum_scale=s["sum_scale"])
    pooled = ops.global_avgpool_q(a, s["s_feat"], s["s_pool"])
    codes = ops.qgemm(pooled, s["fc"], s["fc_scale"], torch.int8, core=True)
    return {"codes": codes, "logits": ops.dequantize(codes, s["s_logits"], s["zp"])}


# ------------------------------------------------------------------------------------------------ one int8 encoder layer
def _prepare_encoder(case, g):
    """The launches of one layer as a compiled program keeps them: six QuantizedDotBias with per-channel weights and a dynamic
    activation scale (max |x| / 127), attention, LayerNorm and Gelu in f32, heads of 64."""
    batch, seq, hidden, ffn = case["n"], case["seq"], case["hidden"], case["ffn"]
    m, heads = batch * seq, hidden // 64
    keep, prog = [], []

    def new(*shape, dtype=torch.float32):
        t = torch.empty(shape, dtype=dtype, device="cuda")
        keep.append(t)
        return t

    def normal(n, sigma, mean=0.0):
        t = torch.randn(n, generator=g, device="cuda") * sigma + mean
        keep.append(t)
        return t

    def emit(fn, *args):
        prog.append((fn, tuple(a.data_ptr() if isinstance(a, torch.Tensor) else a for a in args)))

    zp, c127, rsqrt = torch.zeros((), dtype=torch.int8, device="cuda"), torch.full((1,), 127.0, device="cuda"), torch.full((1,), 0.125, device="cuda")
    keep += [zp, c127, rsqrt]

    def quantized(x, k):
        amax, s_x, xq = new(1), new(1), new(m, k, dtype=torch.int8)
        emit(LIB.b200_reduce_f32, MAX_ABS, x, amax, _i64([m, k]), 2, _i64([0, 1]), 2)
        emit(LIB.b200_f32_binary, DIV, amax, c127, s_x, 1)
        emit(LIB.b200_quantize, x, s_x, zp, xq, I8, _i64([m, k]), 2, _i64([]), 0, 4)
        return xq, s_x

    def linear(xq, s_x, k, n):
        w, s_w = _weights(n, k, g)
        s_w = (s_w * 0.02).contiguous()
        packed, scale, dot, y = ops.pack_weights(w, 128), new(n), new(m, n), new(m, n)
        zero, bias = torch.zeros(n, dtype=torch.int32, device="cuda"), normal(n, 0.02)
        e = _epilogue(scale, "f32", zero)
        keep.extend([s_w, packed, zero, e])
        emit(LIB.b200_f32_binary_periodic, MUL, s_w, s_x, scale, n, 1, 1)
        emit(LIB.b200_qgemm_packed, xq, I8, packed, dot, m, n, k, ctypes.byref(e))
        emit(LIB.b200_f32_binary_periodic, ADD, dot, bias, y, m * n, n, 0)
        return y

    def split_heads(x, order):
        y = new(m, hidden)
        emit(LIB.b200_permute_b32, x, y, _i64([batch, seq, heads, 64]), 4, _i64(order))
        return y

    def layer_norm(x, addend):
        y, gamma, beta = new(m, hidden), normal(hidden, 0.05, 1.0), normal(hidden, 0.05)
        emit(LIB.b200_layer_norm_rows_sum_f32, x, addend, gamma, beta, y, m, hidden, ctypes.c_float(1e-5))
        return y

    x = torch.randn((m, hidden), generator=g, device="cuda")
    xq, s_x = quantized(x, hidden)
    q = split_heads(linear(xq, s_x, hidden, hidden), (0, 2, 1, 3))
    kt = split_heads(linear(xq, s_x, hidden, hidden), (0, 2, 3, 1))
    v = split_heads(linear(xq, s_x, hidden, hidden), (0, 2, 1, 3))
    scores, probs, ctx, merged = new(batch * heads, seq, seq), new(batch * heads, seq, seq), new(m, hidden), new(m, hidden)
    emit(LIB.b200_bmm_f32, q, kt, scores, batch * heads, seq, 64, seq)
    emit(LIB.b200_softmax_rows_scaled_f32, scores, rsqrt, probs, batch * heads * seq, seq)
    emit(LIB.b200_bmm_f32, probs, v, ctx, batch * heads, seq, seq, 64)
    emit(LIB.b200_permute_b32, ctx, merged, _i64([batch, heads, seq, 64]), 4, _i64([0, 2, 1, 3]))
    x1 = layer_norm(x, linear(*quantized(merged, hidden), hidden, hidden))
    up = linear(*quantized(x1, hidden), hidden, ffn)
    h = new(m, ffn)
    emit(LIB.b200_gelu_f32, up, h, m * ffn)
    y = layer_norm(x1, linear(*quantized(h, ffn), ffn, hidden))
    return {"run": _run_encoder, "program": prog, "y": y, "keep": keep, "x": x}


def _run_encoder(s):
    stream = _stream()
    for fn, args in s["program"]:
        check(fn(*args, stream))
    return s["y"]


# ------------------------------------------------------------------------------------------------ what a pass cannot do without
def _out(n, r, stride):
    return (n + 2 * (r // 2) - r) // stride + 1


def work(case):
    kind = case["kind"]
    if kind in ("quantize", "dequantize"):
        elements = case["n"] * case["c"] * case["h"] * case["w"]
        return {"bytes": 5 * elements, "flops": 2 * elements}
    if kind == "dot":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": m * k + n * k + m * n * (4 if case["out"] == "f32" else 1), "flops": 2 * m * n * k}
    if kind == "conv":
        p, q = _out(case["h"], case["r"], case["stride"]), _out(case["w"], case["r"], case["stride"])
        taps, outputs = case["r"] ** 2 * case["c"], case["n"] * p * q * case["k"]
        return {"bytes": case["n"] * case["h"] * case["w"] * case["c"] + taps * case["k"] + outputs * (2 if case["residual"] else 1), "flops": 2 * taps * outputs}
    if kind == "resnet50":
        n, h, w = case["n"], _out(case["h"], 7, 2), _out(case["w"], 7, 2)
        macs, weights = h * w * 64 * 147, 64 * 147
        h, w, cin = _out(h, 3, 2), _out(w, 3, 2), 64
        for blocks, mid, cout, first in BLOCKS:
            for b in range(blocks):
                stride = first if b == 0 else 1
                macs += h * w * cin * mid
                h, w = _out(h, 3, stride), _out(w, 3, stride)
                each = mid * mid * 9 + mid * cout + (cin * cout if b == 0 else 0)
                macs, weights, cin = macs + h * w * each, weights + each + cin * mid, cout
        return {"bytes": n * case["h"] * case["w"] * 12 + weights + 2048 * 1000 + n * 5000, "flops": 2 * n * (macs + 2048 * 1000)}
    m, hidden, ffn = case["n"] * case["seq"], case["hidden"], case["ffn"]
    weights = 4 * hidden * hidden + 2 * hidden * ffn
    return {"bytes": 8 * m * hidden + weights, "flops": 2 * m * weights + 4 * m * case["seq"] * hidden}


def tolerance(case):
    """Bytes are the reference's bytes. Dequantize, f32 dots and the logits are one rounded product of exact values; the encoder
    layer chains sums and transcendental functions in f32."""
    if case["kind"] == "encoder":
        return {"rel": 1e-5}
    if case["kind"] in ("dequantize", "resnet50") or case.get("out") == "f32":
        return {"rel": 1e-6}
    return "exact"
