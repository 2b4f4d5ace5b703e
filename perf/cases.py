"""What this framework's speed is judged by: the quantized projections of RWKV-7 layers, as an engine calls them.

One pass walks the projections of `layers` layers of width C (feed-forward width 4 C):

    r, k, v       [C, C] each      one call where the scheme has a fused one (FP8, INT8 W8A8), else three
    output        [C, C]
    FFN           [4C, C] then [C, 4C]; relu^2 between them (FP8, INT8: one call for the pair; the other schemes: two
                  calls, the value projection on activations that were rectified and squared before)

`scheme`  fp8 (W8A8, e4m3, one scale per call), int8 (W8A8, one scale per row), int4 (weight only, groups of 128),
          nvfp4 (W4A4, blocks of 16), w8a16 (INT8 weight only, one scale)
`rows`    tokens in the call: 1 = one sequence being decoded, a few to some dozens = several sequences decoded
          together, more = a prompt
`mode`    how the program calls: "calls" = the operators from Python, one after another; "graph" = the same operators
          captured once in a CUDA graph and replayed (a decode loop); "layer" = rwkvq_layer.DecodeLayer, which binds
          weights and outputs once (decode, up to 8 rows)
`x`       type of the activations

Weights are N(0, 1/K), quantized as the scheme defines; activations are N(0, 1) with a few channels 20 times larger.
"""
import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rwkv7-quantization_b200"))

NAMES = ("r", "k", "v", "o", "ffn_k", "ffn_v")


def listed():
    c = lambda name, scheme, width, rows, layers, mode, x="f16": dict(  # noqa: E731
        name=name, scheme=scheme, width=width, rows=rows, layers=layers, mode=mode, x=x)
    return [
        # one sequence decoded, mid-sized model, eager: the smallest calls, where host work and launches weigh most
        c("fp8_token_layer", "fp8", 2560, 1, 1, "layer", "bf16"),
        # one sequence decoded, large model, decode loop in a graph
        c("fp8_token_graph", "fp8", 4096, 1, 2, "graph"),
        # a dozen sequences decoded together
        c("fp8_batch_13", "fp8", 4096, 13, 1, "graph"),
        # a short prompt of odd length
        c("fp8_prompt_201", "fp8", 2560, 201, 2, "calls", "bf16"),
        # a long prompt: the largest W8A8 work
        c("fp8_prompt_2048", "fp8", 4096, 2048, 1, "calls"),
        # a few sequences decoded together, INT8
        c("int8_batch_5", "int8", 4096, 5, 1, "layer"),
        # a prompt of odd length, INT8
        c("int8_prompt_717", "int8", 4096, 717, 1, "calls"),
        # one sequence decoded, INT4 weights
        c("int4_token", "int4", 4096, 1, 2, "graph"),
        # a prompt through INT4 weights
        c("int4_prompt_1000", "int4", 4096, 1000, 1, "calls"),
        # some sequences decoded together, NVFP4
        c("nvfp4_batch_7", "nvfp4", 4096, 7, 2, "graph", "bf16"),
        # a long prompt, NVFP4
        c("nvfp4_prompt_2048", "nvfp4", 4096, 2048, 1, "calls", "bf16"),
        # a few sequences decoded together, INT8 weights with 16-bit activations
        c("w8a16_batch_3", "w8a16", 2560, 3, 2, "graph"),
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """Widths are multiples of 256 (every scheme's blocks and groups divide them), prompts of up to 2048 tokens (weight-only
    schemes: 1000)."""
    scheme = rng.choice(("fp8", "fp8", "fp8", "int8", "int8", "int4", "int4", "nvfp4", "nvfp4", "w8a16"))
    width = 256 * _spread(rng, 3, 16)
    rows = {"int4": 1000, "w8a16": 1000}.get(scheme, 2048)
    rows = 1 if rng.random() < 0.15 else rng.randint(2, 8) if rng.random() < 0.2 else _spread(rng, 1, rows)
    modes = ["calls"]
    if rows <= 64:
        modes += ["graph", "graph"]
    if rows <= 8 and scheme in ("fp8", "int8") and rows * (8 * width) * (2 if scheme == "fp8" else 1) <= 128 * 1024:
        modes += ["layer"]
    return dict(scheme=scheme, width=width, rows=rows, layers=rng.randint(1, 2) if width > 1536 else rng.randint(1, 4) if rows <= 512 else 1,
                mode=rng.choice(modes), x=rng.choice(("f16", "bf16")))


def _shape(case, name):
    """(N, K) of a projection."""
    c = case["width"]
    return {"ffn_k": (4 * c, c), "ffn_v": (c, 4 * c)}.get(name, (c, c))


# ----------------------------------------------------------------------------------------------- inputs
def _e2m1_index(a):
    """Index of the e2m1 value (0, .5, 1, 1.5, 2, 3, 4, 6) nearest to a >= 0, ties to the even index."""
    a = a.clamp(max=6.0)
    low, mid, high = torch.round(a * 2), torch.round(a) + 2, torch.round(a / 2) + 4
    return torch.where(a < 2, low, torch.where(a < 4, mid, high)).to(torch.uint8)


def _nvfp4_quantize(v):
    """fp32 [rows, K] -> (signed e2m1 values, block scales as fp32, codes, block scales as e4m3, tensor scale)."""
    amax = v.abs().max().clamp(min=1e-12)
    pts = amax / 2688.0
    blk = v.reshape(v.shape[0], -1, 16)
    bs = (blk.abs().amax(dim=2) * (448.0 / amax)).clamp(2.0 ** -6, 448.0).to(torch.float8_e4m3fn)
    scaled = (blk * (1.0 / pts) / bs.float().unsqueeze(2)).reshape(v.shape)
    idx = _e2m1_index(scaled.abs())
    grid = torch.tensor((0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0), device=v.device)
    return torch.copysign(grid[idx.long()], scaled), bs, idx | (torch.signbit(scaled).to(torch.uint8) << 3), pts


def _weight(scheme, n, k, gen):
    w = torch.randn((n, k), generator=gen, device="cuda") * (1.0 / k) ** 0.5
    if scheme == "fp8":
        s = w.abs().max() / 448.0
        return {"weight": (w / s).clamp(-448.0, 448.0).round().to(torch.float8_e4m3fn), "tensor_scale": s, "qtype": "fp8"}
    if scheme in ("int8", "w8a16"):
        s = w.abs().max() / 127.0
        return {"weight": (w / s).round().clamp(-128, 127).to(torch.int8), "tensor_scale": s,
                "qtype": "int8" if scheme == "int8" else "int8_per_tensor"}
    if scheme == "int4":
        g = w.reshape(n, k // 128, 128)
        lo = g.amin(dim=2, keepdim=True)
        s = ((g.amax(dim=2, keepdim=True) - lo) / 15.0).clamp(min=1e-12)
        q = ((g - lo) / s).round().clamp(0, 15).to(torch.uint8).reshape(n, k)
        return {"packed": q[:, 0::2] | (q[:, 1::2] << 4), "scales": s.squeeze(2).contiguous(), "zeros": lo.squeeze(2).contiguous(),
                "group_size": 128, "qtype": "int4_groupwise"}
    _, bs, codes, pts = _nvfp4_quantize(w)
    return {"weight": (codes[:, 0::2] | (codes[:, 1::2] << 4)).contiguous(), "block_scale": bs.contiguous(), "tensor_scale": pts,
            "qtype": "nvfp4"}


def _inputs(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    dt = torch.float16 if case["x"] == "f16" else torch.bfloat16
    pair = case["scheme"] in ("fp8", "int8")
    ws, xs = [], []
    for _ in range(case["layers"]):
        ws.append({p: _weight(case["scheme"], *_shape(case, p), gen) for p in NAMES})
        x = {}
        for p in NAMES[:5] if pair else NAMES:
            k = _shape(case, p)[1]
            v = torch.randn((case["rows"], k), generator=gen, device="cuda")
            v[:, torch.randint(0, k, (max(1, k // 1000),), generator=gen, device="cuda")] *= 20.0
            x[p] = (v.clamp(min=0).square() if p == "ffn_v" else v).to(dt)
        xs.append(x)
    return ws, xs


# ----------------------------------------------------------------------------------------------- the calls
def _calls(scheme, rows, ws, xs):
    import fused_fp8_gemm as f
    from int8.int8_ops import linear_int8
    outs = []
    for w, x in zip(ws, xs):
        if scheme == "w8a16":
            outs.append([linear_int8(x[p], w[p]) for p in NAMES])
        elif scheme in ("int4", "nvfp4"):
            outs.append([f.linear_quantized_fused(x[p], w[p]) for p in NAMES])
        else:
            rkv = f.linear_rkv_int8_fused if scheme == "int8" else f.linear_rkv_fused
            ffn = f.ffn_relu2_int8 if scheme == "int8" else f.ffn_relu2_fp8
            if rows <= f.FUSED_M_MAX:                # the engine's rule: longer prompts take three calls
                o = list(rkv(x["r"], x["k"], x["v"], w["r"], w["k"], w["v"]))
            else:
                o = [f.linear_quantized_fused(x[p], w[p]) for p in "rkv"]
            outs.append(o + [f.linear_quantized_fused(x["o"], w["o"]), ffn(x["ffn_k"], w["ffn_k"], w["ffn_v"])])
    return outs


_side = []


def prepare(case, seed):
    ws, xs = _inputs(case, seed)
    state = {"case": case, "w": ws, "x": xs}
    if case["mode"] == "layer":
        from rwkvq_layer import DecodeLayer
        state["layers"] = [DecodeLayer(*(w[p] for p in NAMES), rows=case["rows"], x_dtype=xs[0]["r"].dtype, compat_shared_scale=True)
                           for w in ws]
    elif case["mode"] == "graph":
        if not _side:
            _side.append(torch.cuda.Stream())
        _side[0].wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(_side[0]):
            _calls(case["scheme"], case["rows"], ws, xs)        # buffers that the library keeps are made outside the capture
            _side[0].synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=_side[0]):
                state["outs"] = _calls(case["scheme"], case["rows"], ws, xs)
        state["graph"] = graph
    return state


def run(state):
    case = state["case"]
    if case["mode"] == "graph":
        state["graph"].replay()
        return state["outs"]
    if case["mode"] == "calls":
        return _calls(case["scheme"], case["rows"], state["w"], state["x"])
    outs = []
    for layer, x in zip(state["layers"], state["x"]):
        rkv = layer.rkv(x["r"], x["k"], x["v"])
        o = layer.att_out(x["o"])
        outs.append([*rkv, o, layer.ffn(x["ffn_k"])[0]])
    return outs


# ----------------------------------------------------------------------------------------------- what a pass has to do
def work(case):
    """Weights with their scales once, each call's activations and fp16 results once."""
    per_weight = {"fp8": 1.0, "int8": 1.0, "w8a16": 1.0, "int4": 0.5 + 8 / 128, "nvfp4": 0.5 + 1 / 16}[case["scheme"]]
    pair = case["scheme"] in ("fp8", "int8")
    m, nbytes, flops = case["rows"], 0, 0
    for p in NAMES:
        n, k = _shape(case, p)
        nbytes += per_weight * n * k
        nbytes += 0 if pair and p == "ffn_v" else 2 * m * k
        nbytes += 0 if pair and p == "ffn_k" else 2 * m * n
        flops += 2 * m * n * k
    return {"bytes": case["layers"] * nbytes, "flops": case["layers"] * flops}


def tolerance(case):
    """fp16 results of 32-bit sums (against 64 bits: 2.1e-4 where no activation code differs).  The FFN pair quantizes its
    hidden activations again, where a last bit moves some codes to the neighbour."""
    return {"rel": 1e-3}


# ----------------------------------------------------------------------------------------------- the same in 64 bits
def _fp8_codes(x, bf16_first):
    """Activation codes as fp64 and their scale: one maximum per call, quantized from the bf16 value."""
    xb = x.to(torch.bfloat16).float()
    amax = (xb if bf16_first else x.float()).abs().max().clamp(min=1e-12)
    return (xb * (448.0 / amax)).clamp(-448.0, 448.0).to(torch.float8_e4m3fn).double(), amax.double() / 448.0


def _int8_codes(x):
    xf = x.float()
    amax = xf.abs().amax(dim=1, keepdim=True).clamp(min=1e-12)
    return (xf * (torch.full_like(amax, 127.0) / amax)).clamp(-128.0, 127.0).trunc().double(), amax.double() / 127.0


def _exact_linear(scheme, x, w, w_scale=None, bf16_first=False, via_bf16=False):
    if scheme == "fp8":
        a, s = _fp8_codes(x, bf16_first)
        y = (a @ w["weight"].double().t()) * (s * w["tensor_scale"].double())
        return y.to(torch.bfloat16).double() if via_bf16 else y
    if scheme == "int8":
        a, s = _int8_codes(x)
        return (a @ w["weight"].double().t()) * (s * (w["tensor_scale"] if w_scale is None else w_scale).double())
    if scheme == "w8a16":
        return (x.to(torch.float16).double() @ w["weight"].double().t()) * w["tensor_scale"].double()
    if scheme == "int4":
        p = w["packed"]
        u = torch.stack((p & 15, p >> 4), dim=2).reshape(p.shape[0], -1, 128).double()
        d = u * w["scales"].double().unsqueeze(2) + w["zeros"].double().unsqueeze(2)
        return x.to(torch.float16).double() @ d.reshape(p.shape[0], -1).t()
    a, bs, _, pts = _nvfp4_quantize(x.float())
    p = w["weight"]
    c = torch.stack((p & 15, p >> 4), dim=2).reshape(p.shape[0], -1).long()
    grid = torch.tensor((0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0), device=p.device, dtype=torch.float64)
    d = torch.where(c >= 8, -grid[c & 7], grid[c & 7]) * w["block_scale"].double().repeat_interleave(16, dim=1)
    return ((a.double() * bs.double().repeat_interleave(16, dim=1)) @ d.t()) * (pts.double() * w["tensor_scale"].double())


def exact(case, seed):
    """The quantized values are the scheme's own (they are what the path computes on); sums and scales in 64 bits.  The hidden
    activations of the FFN pair are fp16 values, as they are between its two projections."""
    ws, xs = _inputs(case, seed)
    scheme, m = case["scheme"], case["rows"]
    outs = []
    for w, x in zip(ws, xs):
        if scheme not in ("fp8", "int8"):
            outs.append([_exact_linear(scheme, x[p], w[p]) for p in NAMES])
            continue
        single = dict(bf16_first=m == 1 or m > 512, via_bf16=m > 512) if scheme == "fp8" else {}
        fused = {} if scheme == "int8" or m <= 512 else single
        shared = {"w_scale": w["r"]["tensor_scale"]} if scheme == "int8" and m <= 512 else {}   # r's scale serves r, k and v
        o = [_exact_linear(scheme, x[p], w[p], **fused, **shared) for p in "rkv"]
        o.append(_exact_linear(scheme, x["o"], w["o"], **single))
        y = _exact_linear(scheme, x["ffn_k"], w["ffn_k"], **single).to(torch.float16).float()
        hid = y.clamp(min=0.0).square().to(torch.float16)
        outs.append(o + [_exact_linear(scheme, hid, w["ffn_v"], **single)])
    return outs
