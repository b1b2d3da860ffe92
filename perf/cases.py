"""The work that is timed: what programs built on this library have it do, through its public calls, on device memory.

Sizes are those of the repository's own workloads (the BERT-base-shaped linear stack, the 8192 x 28672 feed-forward
products, the ResNet-50-shaped convolutions, the 256-channel 1-bit convolution, 16384 x 3072 activations) and, between
and around them, whatever draw() picks from the same ranges: odd sizes, short and long calls, every output type.

Every result is compared bit for bit.  All arithmetic on this path is integer accumulation followed by single binary32
(or binary16) operations whose order the library defines, so any correct implementation gives the same bits.
"""
import ctypes as C
import math

import torch

import bolt_b200 as B
from bolt_b200.linear_stack import Linear, LinearStack
from bolt_b200.workloads import RESNET50_LAYERS

OUT_DT = {"f32": (B.DT_F32, torch.float32), "s32": (B.DT_I32, torch.int32), "u8": (B.DT_U8_Q, torch.uint8)}


def listed():
    return [
        # the smallest call: one BERT-base projection of 128 tokens, fp32 in (quantized dynamically), fp32 out
        {"name": "linear_128x768x768", "kind": "linear", "m": 128, "k": 768, "n": 768, "out": "f32", "packed": True, "a_t": False},
        # sizes that are no multiple of anything: a sequence of 333 frames of 515 features against 1001 classes
        {"name": "linear_ragged", "kind": "linear", "m": 333, "k": 515, "n": 1001, "out": "f32", "packed": True, "a_t": False},
        # a BERT-base batch (32 x 128 tokens) through its 24 linear layers, 8-bit between layers
        {"name": "stack_4096", "kind": "stack", "m": 4096, "pairs": 12, "hidden": 768, "inter": 3072},
        # the same network answering one short query: launches and latency
        {"name": "stack_16", "kind": "stack", "m": 16, "pairs": 12, "hidden": 768, "inter": 3072},
        # feed-forward product of a large language model: prefill of 2048 tokens, u8 out, a scale for every token
        {"name": "ffn_2048", "kind": "ffn", "m": 2048, "k": 8192, "n": 28672, "out": "u8", "rows": True},
        # the same weight, 16 sequences decoded at once, fp32 out
        {"name": "ffn_16", "kind": "ffn", "m": 16, "k": 8192, "n": 28672, "out": "f32", "rows": True},
        # the same weight, one sequence decoded: matrix times vector
        {"name": "gemv_28672x8192", "kind": "gemv", "n": 28672, "k": 8192, "out": "f32"},
        # BERT-base attention of the 32 x 128 tokens: scores = Q K^T and context = P V, both operands fp32 activations
        {"name": "attention_32x12x128x64", "kind": "attention", "batch": 32, "heads": 12, "q": 128, "kv": 128, "dim": 64},
        # a ResNet-50-shaped network on a batch of 64: stem pooling and the 22 distinct convolutions, calibrated u8 outputs
        {"name": "resnet_64", "kind": "resnet", "batch": 64, "image": 224, "width": 64, "out": "u8"},
        # one image, Bolt's own output protocol: the u8 scale of every layer is found from its result
        {"name": "resnet_1_dynamic", "kind": "resnet", "batch": 1, "image": 224, "width": 64, "out": "dynamic"},
        # XNOR-Net convolution 256 -> 256, 3x3 on 28 x 28, fp16 in and out
        {"name": "bnn_128", "kind": "bnn", "batch": 128, "ic": 256, "oc": 256, "hw": 28, "kernel": 3, "stride": 1, "xnor": True},
        # conversions at the edges of a quantized region, on 16384 x 3072 activations
        {"name": "quantize_16384x3072", "kind": "quantize", "n": 16384 * 3072, "to": "u8"},
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng):
    kind = rng.choice(("linear", "linear", "stack", "ffn", "gemv", "attention", "resnet", "bnn", "quantize"))
    if kind == "linear":
        k = _log(rng, 16, 4096)
        if rng.random() < 0.5:
            k = (k + 15) // 16 * 16
        return {"kind": kind, "m": _log(rng, 2, 4096), "k": k, "n": _log(rng, 8, 4096), "out": rng.choice(("f32", "s32", "u8")),
                "packed": rng.random() < 0.8, "a_t": rng.random() < 0.1}
    if kind == "stack":
        hidden = 64 * rng.randint(4, 16)
        m, pairs = _log(rng, 2, 4096), rng.randint(1, 12)
        while m * pairs * hidden * hidden > 4096 * 12 * 768 * 768:
            m //= 2
        return {"kind": kind, "m": m, "pairs": pairs, "hidden": hidden, "inter": 4 * hidden}
    if kind == "ffn":
        return {"kind": kind, "m": _log(rng, 2, 2048), "k": 16 * _log(rng, 64, 512), "n": 4 * _log(rng, 256, 7168),
                "out": rng.choice(("u8", "f32")), "rows": rng.random() < 0.7}
    if kind == "gemv":
        return {"kind": kind, "n": _log(rng, 256, 28672), "k": _log(rng, 64, 8192), "out": rng.choice(("f32", "s32", "u8"))}
    if kind == "attention":
        heads = rng.choice((4, 8, 12, 16))
        q = kv = _log(rng, 8, 384)
        if rng.random() < 0.3:
            q = rng.choice((1, 2, 7, 32))     # decoding: few queries against a longer context
        return {"kind": kind, "batch": rng.randint(1, max(1, 384 // heads)), "heads": heads, "q": q, "kv": kv, "dim": rng.choice((32, 64, 80, 128))}
    if kind == "resnet":
        image, width = rng.randint(96, 256), rng.choice((32, 48, 64))
        batch = _log(rng, 1, 64)
        while batch * image * image * width * width > 64 * 224 * 224 * 64 * 64:
            batch //= 2
        return {"kind": kind, "batch": batch, "image": image, "width": width, "out": rng.choice(("u8", "f32", "dynamic"))}
    if kind == "bnn":
        hw, ic, oc = rng.randint(5, 56), 8 * rng.randint(4, 64), 8 * rng.randint(4, 64)
        batch = _log(rng, 1, 128)
        while batch * hw * hw * ic * oc > 128 * 28 * 28 * 256 * 256:
            batch //= 2
        return {"kind": kind, "batch": max(1, batch), "ic": ic, "oc": oc, "hw": hw, "kernel": rng.choice((1, 3, 3)),
                "stride": rng.choice((1, 1, 2)), "xnor": rng.random() < 0.6}
    return {"kind": kind, "n": _log(rng, 1000, 16384 * 3072), "to": rng.choice(("u8", "i8"))}


def _p(t, off=0):
    return C.c_void_p(t.data_ptr() + off)


def _bytes(n):
    return torch.empty(max(16, int(n)), dtype=torch.uint8, device="cuda")


def _s8(g, *shape):
    return torch.randint(-127, 128, shape, dtype=torch.int8, device="cuda", generator=g)


def _resnet_layers(case):
    """(ic, hw, oc, k, stride, pad) of the 22 layers at the case's image size and width"""
    size = {56: (case["image"] + 3) // 4}
    for hw in (28, 14, 7):
        size[hw] = (size[2 * hw] + 1) // 2
    return [(ic * case["width"] // 64, size[hw], oc * case["width"] // 64, k, s, p) for ic, hw, oc, k, s, p in RESNET50_LAYERS]


def _out_hw(hw, k, s, p):
    return (hw + 2 * p - k) // s + 1


# ---- what a program has in hand before the call ------------------------------------------------------------------
def _prepare_linear(c, g):
    m, k, n = c["m"], c["k"], c["n"]
    dt, tdt = OUT_DT[c["out"]]
    x = torch.randn((k, m) if c["a_t"] else (m, k), device="cuda", generator=g)
    w = _s8(g, k, n)
    rows, cols = (k, m) if c["a_t"] else (m, k)
    s = {"x": x, "x_desc": B.tensor2df(B.DT_F32, B.DF_NORMAL, rows, cols), "q": _bytes(m * k), "w_scale": 127.0 / 0.09,
         "q_desc": B.tensor2df(B.DT_U8_Q, B.DF_TRANSPOSE if c["a_t"] else B.DF_NORMAL, rows, cols),
         "w": w, "w_desc": B.tensor2df(B.DT_I8, B.DF_NORMAL, k, n), "out": c["out"],
         "c": torch.zeros((m, n), dtype=tdt, device="cuda"), "c_desc": B.tensor2df(dt, B.DF_NORMAL, m, n)}
    off = None
    if c["packed"]:
        nbytes, rhs = B.matrix_matrix_multiply_transform_rhs_bytes(s["w_desc"])
        packed = _bytes(nbytes)
        s["w_desc"] = B.matrix_matrix_multiply_transform_rhs(s["w_desc"], _p(w), _p(packed))
        s["w"], off = packed, packed[rhs: rhs + 4 * n]
    s["tmp_bytes"] = B.matrix_matrix_multiply_tmp_bytes(s["q_desc"], s["w_desc"])
    s["tmp"] = _bytes(s["tmp_bytes"])
    if off is not None:
        s["tmp"][: 4 * n] = off               # the offsets of a pre-packed weight travel in tmp
    # calibrated: the real-valued results are about N(0, k * 0.03^2), four sigma fill the u8 range
    s["out_scale"] = 127.0 / (4 * 0.05 * math.sqrt(k))
    return s


def _run_linear(s):
    scale = [-1.0]
    B.quantize(s["x_desc"], _p(s["x"]), s["q_desc"], _p(s["q"]), scale)
    so = scale[0] * s["w_scale"]
    if s["out"] == "u8":
        sc = [-1.0, s["out_scale"] / so]
    else:
        s["c"].zero_()                        # the product accumulates on top of C
        sc = [so] if s["out"] == "f32" else None
    B.matrix_matrix_multiply(s["q_desc"], _p(s["q"]), s["w_desc"], _p(s["w"]), s["tmp_bytes"], _p(s["tmp"]), s["c_desc"], _p(s["c"]), sc)
    return {"scale": scale[0], "c": s["c"]}


def _prepare_stack(c, g):
    layers = []
    for _ in range(c["pairs"]):
        for k, n in ((c["hidden"], c["inter"]), (c["inter"], c["hidden"])):
            w = torch.randn(k, n, device="cuda", generator=g) * 0.02
            ws = 127.0 / w.abs().amax(dim=0)
            q = torch.clamp(torch.round(w * ws), -127, 127).to(torch.int8)
            layers.append(Linear(q.cpu().numpy(), ws.cpu().numpy()))
    st = LinearStack(layers, c["m"])
    st.x_dev.copy_(torch.randn(c["m"] * c["hidden"], device="cuda", generator=g))
    st.calibrate()
    return {"stack": st}


def _run_stack(s):
    s["stack"].step()
    return s["stack"].out_dev


def _prepare_ffn(c, g):
    m, k, n = c["m"], c["k"], c["n"]
    dt, tdt = OUT_DT[c["out"]]
    w = _s8(g, k, n)
    desc = B.tensor2df(B.DT_I8, B.DF_NORMAL, k, n)
    nbytes, rhs = B.matrix_matrix_multiply_transform_rhs_bytes(desc)
    packed = _bytes(nbytes)
    B.matrix_matrix_multiply_transform_rhs(desc, _p(w), _p(packed))
    s = {"m": m, "k": k, "n": n, "packed": packed, "rhs": rhs, "c": torch.empty((m, n), dtype=tdt, device="cuda"),
         # post-normalisation activations: bell shaped around the zero point
         "a": torch.clamp(torch.round(torch.randn((m, k), device="cuda", generator=g) * 32) + 128, 1, 255).to(torch.uint8),
         "row": (torch.rand(m, device="cuda", generator=g) * 20 + 30).float(),
         "col": (127.0 / (0.05 + 0.02 * torch.rand(n, device="cuda", generator=g))).float()}
    ep = B.GemmEpilogue()
    ep.out_dt, ep.accumulate, ep.out_scale, ep.sA, ep.sB = dt, 0, 1.0, 40.0, 1.0
    if c["out"] == "u8":
        ep.out_scale = 127.0 / (4 * 32 * 73 * math.sqrt(k)) * 40 * 2100
    ep.row_scale = _p(s["row"]) if c["rows"] else None
    ep.col_scale = _p(s["col"])
    s["ep"] = ep
    return s


def _run_ffn(s):
    B.CHECK_STATUS(B.lib().bolt_b200_gemm_u8s8_ex(s["n"], s["m"], s["k"], _p(s["a"]), _p(s["packed"]), _p(s["packed"], s["rhs"]), _p(s["c"]),
                                                  C.byref(s["ep"])), "gemm")
    return s["c"]


def _prepare_gemv(c, g):
    n, k = c["n"], c["k"]
    dt, tdt = OUT_DT[c["out"]]
    w = _s8(g, n, k)
    desc = B.tensor2df(B.DT_I8, B.DF_NORMAL, n, k)
    packed = _bytes(B.matrix_vector_multiply_transform_weight_bytes(desc))
    s = {"desc": B.matrix_vector_multiply_transform_weight(desc, _p(w), _p(packed)), "packed": packed, "out": c["out"],
         "x": torch.clamp(torch.round(torch.randn(k, device="cuda", generator=g) * 32) + 128, 1, 255).to(torch.uint8),
         "x_desc": B.tensor1d(B.DT_U8_Q, k), "y": torch.zeros(n, dtype=tdt, device="cuda"), "y_desc": B.tensor1d(dt, n)}
    off = (n + 15) // 16 * 16 * ((k + 7) // 8 * 8)
    s["tmp_bytes"] = B.matrix_vector_multiply_tmp_bytes(s["desc"], s["x_desc"])
    s["tmp"] = _bytes(s["tmp_bytes"])
    s["tmp"][: 4 * n] = packed[off: off + 4 * n]
    s["scale"] = {"f32": [40.0 * 1400.0], "s32": None, "u8": [-1.0, 127.0 / (4 * 32 * 73 * math.sqrt(k))]}[c["out"]]
    return s


def _run_gemv(s):
    if s["out"] != "u8":
        s["y"].zero_()                        # the product accumulates on top of y
    B.matrix_vector_multiply(s["desc"], _p(s["packed"]), s["x_desc"], _p(s["x"]), s["tmp_bytes"], _p(s["tmp"]), s["y_desc"], _p(s["y"]), s["scale"])
    return s["y"]


def _matmul_call(a, b, tb):
    """both operands fp32, quantized inside the call; fp32 result"""
    ad, bd = B.tensor_nd(B.DT_F32, tuple(a.shape)), B.tensor_nd(B.DT_F32, tuple(b.shape))
    cd = B.matmul_infer_output_size(ad, 0, bd, tb)
    cd.dt = B.DT_F32
    out = torch.empty(tuple(reversed(list(cd.dims[: cd.nDims]))), dtype=torch.float32, device="cuda")
    nb = B.matmul_infer_forward_tmp_bytes(ad, 0, bd, tb, cd, -1.0)
    return {"ad": ad, "a": a, "bd": bd, "b": b, "tb": tb, "cd": cd, "c": out, "nb": nb, "tmp": _bytes(nb)}


def _prepare_attention(c, g):
    shape = (c["batch"], c["heads"])
    q = torch.randn(shape + (c["q"], c["dim"]), device="cuda", generator=g)
    k = torch.randn(shape + (c["kv"], c["dim"]), device="cuda", generator=g)
    v = torch.randn(shape + (c["kv"], c["dim"]), device="cuda", generator=g)
    prob = torch.softmax(torch.randn(shape + (c["q"], c["kv"]), device="cuda", generator=g), dim=-1)
    return {"calls": [_matmul_call(q, k, 1), _matmul_call(prob, v, 0)]}


def _run_attention(s):
    for m in s["calls"]:
        B.matmul(m["ad"], 0, _p(m["a"]), -1.0, m["bd"], m["tb"], _p(m["b"]), -1.0, None, None, m["nb"], _p(m["tmp"]), m["cd"], _p(m["c"]), -1.0)
    return [m["c"] for m in s["calls"]]


def _prepare_resnet(c, g):
    n, target = c["batch"], B.DT_F32 if c["out"] == "f32" else B.DT_U8_Q
    convs = []
    for ic, hw, oc, k, st, pad in _resnet_layers(c):
        p = B.conv_param(oc, k, k, st, pad, 1, True)
        in_desc, f_desc = B.tensor4df(B.DT_U8_Q, B.DF_NCHWC16, n, ic, hw, hw), B.tensor4df(B.DT_I8, B.DF_NCHW, oc, ic, k, k)
        out_desc = B.convolution_infer_output_size(in_desc, f_desc, p, target)
        alg = B.convolution_infer_forward_algorithm(in_desc, f_desc, out_desc, p, target)
        w = torch.clamp(torch.round(torch.randn(oc * ic * k * k, device="cuda", generator=g) * 32), -127, 127).to(torch.int8)
        ftm = _bytes(B.convolution_transform_filter_bytes(f_desc, p, alg))
        ftm_desc = B.convolution_transform_filter(f_desc, _p(w), p, alg, _p(ftm))
        tb = B.convolution_infer_forward_tmp_bytes(in_desc, ftm_desc, out_desc, p, alg)
        oh = _out_hw(hw, k, st, pad)
        # ReLU-distributed activations with zero point 128, four sigma at 255
        x = torch.clamp(torch.round(torch.relu(torch.randn(n * ic * hw * hw, device="cuda", generator=g)) * 31.75) + 128, 1, 255).to(torch.uint8)
        s_in, s_w = 31.75, 32 / 0.05
        convs.append({"in_desc": in_desc, "x": x, "ftm_desc": ftm_desc, "ftm": ftm, "p": p, "alg": alg, "tb": tb, "tmp": _bytes(tb),
                      "scale": [s_in, -1.0, s_w], "bias": torch.randn(oc, device="cuda", generator=g) * 0.1, "out_desc": out_desc,
                      "out": torch.empty(n * oc * oh * oh, dtype=torch.float32 if c["out"] == "f32" else torch.uint8, device="cuda"),
                      # results are about N(0, ic k^2 / 2 * 0.05^2)
                      "out_scale": 127.0 / (4 * 0.05 * math.sqrt(ic * k * k / 2)) if c["out"] == "u8" else None})
    ch, hw = c["width"], 2 * _resnet_layers(c)[0][1]
    oh = _out_hw(hw, 3, 2, 1)
    pool = {"x": torch.clamp(torch.round(torch.relu(torch.randn(n * ch * hw * hw, device="cuda", generator=g)) * 31.75) + 128, 1, 255).to(torch.uint8),
            "in_desc": B.tensor4df(B.DT_U8_Q, B.DF_NCHWC16, n, ch, hw, hw), "out_desc": B.tensor4df(B.DT_U8_Q, B.DF_NCHWC16, n, ch, oh, oh),
            "out": _bytes(n * ch * oh * oh), "p": B.pooling_param(3, 2, 1)}
    return {"convs": convs, "pool": pool}


def _run_resnet(s):
    p = s["pool"]
    B.pooling(p["in_desc"], _p(p["x"]), p["p"], [31.75, 0.0], p["out_desc"], _p(p["out"]))
    scales = []
    for v in s["convs"]:
        scale = list(v["scale"])
        B.convolution(v["in_desc"], _p(v["x"]), v["ftm_desc"], _p(v["ftm"]), v["p"], v["alg"], scale, _p(v["bias"]), v["tb"], _p(v["tmp"]),
                      v["out_desc"], _p(v["out"]), True, None, v["out_scale"])
        scales.append(scale[1])
    return {"pool": p["out"], "out": [v["out"] for v in s["convs"]], "scales": scales}


def _prepare_bnn(c, g):
    n, ic, oc, hw, k, st = c["batch"], c["ic"], c["oc"], c["hw"], c["kernel"], c["stride"]
    pad = k // 2
    oh = _out_hw(hw, k, st, pad)
    p = B.conv_param(oc, k, k, st, pad)
    in_desc, out_desc = B.tensor4df(B.DT_F16, B.DF_NCHWC8, n, ic, hw, hw), B.tensor4df(B.DT_F16, B.DF_NCHWC8, n, oc, oh, oh)
    f_desc = B.tensor4df(B.DT_BIN11 if c["xnor"] else B.DT_BIN01, B.DF_NCHW, oc, ic, k, k)
    alg = B.convolution_infer_forward_algorithm(in_desc, f_desc, out_desc, p, B.DT_F16)
    bits = torch.randint(0, 256, (oc * ic * k * k // 8,), dtype=torch.uint8, device="cuda", generator=g)
    ftm = torch.zeros(B.convolution_transform_filter_bytes(f_desc, p, alg), dtype=torch.uint8, device="cuda")
    ftm_desc = B.convolution_transform_filter(f_desc, _p(bits), p, alg, _p(ftm))
    tb = B.convolution_infer_forward_tmp_bytes(in_desc, ftm_desc, out_desc, p, alg)
    x = torch.randn(n * ic * hw * hw, device="cuda", generator=g)
    return {"x": (x if c["xnor"] else x * 0.5 + 0.5).half(), "in_desc": in_desc, "ftm": ftm, "ftm_desc": ftm_desc, "p": p, "alg": alg, "tb": tb,
            "tmp": _bytes(tb), "alpha": (torch.rand(oc, device="cuda", generator=g) * 0.1 + 0.01).half(),
            "beta": (torch.randn(oc, device="cuda", generator=g) * 0.1).half(), "out_desc": out_desc,
            "out": torch.empty(n * oc * oh * oh, dtype=torch.float16, device="cuda")}


def _run_bnn(s):
    B.convolution(s["in_desc"], _p(s["x"]), s["ftm_desc"], _p(s["ftm"]), s["p"], s["alg"], _p(s["alpha"]), _p(s["beta"]), s["tb"], _p(s["tmp"]),
                  s["out_desc"], _p(s["out"]))
    return s["out"]


def _prepare_quantize(c, g):
    n = c["n"]
    return {"x": torch.randn(n, device="cuda", generator=g), "acc": torch.round(torch.randn(n, device="cuda", generator=g) * 20000).to(torch.int32),
            "q": _bytes(n), "r": _bytes(n), "f": torch.empty(n, device="cuda"), "f_desc": B.tensor1d(B.DT_F32, n), "i_desc": B.tensor1d(B.DT_I32, n),
            "q_desc": B.tensor1d(B.DT_U8_Q if c["to"] == "u8" else B.DT_I8, n)}


def _run_quantize(s):
    """fp32 activations to 8 bits with the scale found, int32 accumulators to 8 bits with the scale found, and to fp32"""
    sq, sr = [-1.0], [-1.0, 40.0]
    B.quantize(s["f_desc"], _p(s["x"]), s["q_desc"], _p(s["q"]), sq)
    B.quantize(s["i_desc"], _p(s["acc"]), s["q_desc"], _p(s["r"]), sr)
    B.dequantize(s["i_desc"], _p(s["acc"]), 40.0, s["f_desc"], _p(s["f"]))
    return {"q": s["q"], "r": s["r"], "f": s["f"], "scales": [sq[0], sr[0]]}


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    s = globals()["_prepare_" + case["kind"]](case, g)
    s["kind"] = case["kind"]
    return s


def run(state):
    return globals()["_run_" + state["kind"]](state)


def work(case):
    c, kind = case, case["kind"]
    size = {"f32": 4, "s32": 4, "u8": 1, "dynamic": 1}
    if kind == "linear":
        m, k, n = c["m"], c["k"], c["n"]
        return {"bytes": 4 * m * k + k * n + 4 * n + m * n * size[c["out"]], "flops": 2 * m * k * n}
    if kind == "stack":
        m, h, i, pairs = c["m"], c["hidden"], c["inter"], c["pairs"]
        # fp32 in and out; between layers the u8 activations are an output of one layer and an input of the next
        return {"bytes": 8 * m * h + pairs * (2 * h * i + 8 * (h + i) + 2 * m * i) + (pairs - 1) * 2 * m * h, "flops": pairs * 4 * m * h * i}
    if kind == "ffn":
        m, k, n = c["m"], c["k"], c["n"]
        return {"bytes": m * k + k * n + 8 * n + 4 * m + m * n * size[c["out"]], "flops": 2 * m * k * n}
    if kind == "gemv":
        return {"bytes": c["n"] * c["k"] + c["k"] + c["n"] * (4 + size[c["out"]]), "flops": 2 * c["n"] * c["k"]}
    if kind == "attention":
        b, q, kv, d = c["batch"] * c["heads"], c["q"], c["kv"], c["dim"]
        return {"bytes": 4 * b * (q * d + kv * d + q * kv) * 2, "flops": 4 * b * q * kv * d}
    if kind == "resnet":
        n, layers = c["batch"], _resnet_layers(c)
        hw = 2 * layers[0][1]
        nbytes, flops = n * c["width"] * (hw * hw + _out_hw(hw, 3, 2, 1) ** 2), 0
        for ic, hw, oc, k, st, pad in layers:
            oh = _out_hw(hw, k, st, pad)
            nbytes += n * ic * hw * hw + oc * ic * k * k + 8 * oc + n * oc * oh * oh * size[c["out"]]
            flops += 2 * n * oc * oh * oh * ic * k * k
        return {"bytes": nbytes, "flops": flops}
    if kind == "bnn":
        n, ic, oc, hw, k = c["batch"], c["ic"], c["oc"], c["hw"], c["kernel"]
        oh = _out_hw(hw, k, c["stride"], k // 2)
        return {"bytes": 2 * n * ic * hw * hw + oc * ic * k * k // 8 + 4 * oc + 2 * n * oc * oh * oh, "flops": 2 * n * oc * oh * oh * ic * k * k}
    return {"bytes": (4 + 1 + 4 + 1 + 4) * c["n"], "flops": 0}


def tolerance(case):
    return "exact"
