"""The work that a user of this library has it do, as timed cases: single W8A8 linears (quantize + GEMM + dequantize
[+ re-quantize]) from one token to the largest prefill, the whole quantized path of one transformer layer (norm +
quantize, fused QKV, output projection, gate + up with SwiGLU, down projection), and the linear on host buffers.

`listed()` are fixed cases, `draw(rng)` gives more of the same ranges.  A case is run with `run(prepare(case, seed))`.
"""
import os
import sys

import torch

_PKG = os.path.join(os.getcwd(), "ppl.llm.kernel.cuda_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import pplb200  # noqa: E402

HIDDEN_UP = 8192.0  # column scales are stored as s_n * 8192 in fp16


def listed():
    return [
        # one token through a 4096-wide output projection: a single conversation being decoded
        dict(name="linear m1", kind="linear", m=1, k=4096, n=4096, bias=True, requant=False, x="normal"),
        # decode with sixteen conversations (the benchmark's smallest configuration)
        dict(name="linear m16", kind="linear", m=16, k=4096, n=4096, bias=True, requant=False, x="normal"),
        # decode, an odd batch, down projection of an 11008-wide MLP
        dict(name="linear m37 k11008", kind="linear", m=37, k=11008, n=4096, bias=True, requant=False, x="normal"),
        # batched decode, fused QKV, the result re-quantized for the next operator (benchmark configuration)
        dict(name="linear m128 requant", kind="linear", m=128, k=4096, n=12288, bias=True, requant=True, x="normal"),
        # one scheduler step that mixes decoding tokens and a piece of a prompt
        dict(name="linear m333", kind="linear", m=333, k=4096, n=4096, bias=True, requant=False, x="normal"),
        # prefill of a 4096-token prompt, gate + up projection, outlier channels (benchmark configuration)
        dict(name="linear m4096", kind="linear", m=4096, k=4096, n=22016, bias=False, requant=False, x="outlier"),
        # prefill, down projection with a long K (benchmark configuration)
        dict(name="linear m2048 k28672", kind="linear", m=2048, k=28672, n=8192, bias=True, requant=False, x="normal"),
        # the largest prefill, up projection, heavy-tailed activations (benchmark configuration)
        dict(name="linear m8192", kind="linear", m=8192, k=8192, n=28672, bias=False, requant=False, x="student"),
        # one layer of a 4096-wide model, eight conversations being decoded; replayed from a CUDA graph, as decoding is
        dict(name="layer m8", kind="layer", m=8, hidden=4096, q=4096, kv=4096, inter=11008),
        # one rank's eighth of a layer of an 8192-wide model with grouped KV heads, 96 conversations
        dict(name="layer m96 shard", kind="layer", m=96, hidden=8192, q=1024, kv=128, inter=3584),
        # one layer of a 4096-wide model, prefill of an odd number of tokens, called eagerly
        dict(name="layer m1999", kind="layer", m=1999, hidden=4096, q=4096, kv=4096, inter=11008),
        # activations come from and results go to pinned host memory
        dict(name="host m1024", kind="host", m=1024, k=4096, n=4096, bias=True, requant=False, x="normal"),
    ]


def _log_int(rng, lo, hi, step=1):
    """An integer multiple of `step` in [lo, hi], spread over the logarithm."""
    v = lo * (hi / lo) ** rng.random()
    return int(min(hi, max(lo, round(v / step) * step)))


def draw(rng):
    kind = rng.choice(["linear", "linear", "linear", "layer", "layer", "host"])
    if kind == "layer":
        # widths of 4096- and 8192-wide layers, whole or cut over 2, 4 or 8 ranks, and widths in between
        hidden = rng.choice([2048, 4096, 5120, 8192])
        ranks = rng.choice([1, 2, 4, 8])
        q = hidden // ranks
        kv = max(128, q // rng.choice([1, 1, 4, 8]))
        inter = max(512, _log_int(rng, 2 * hidden, 3.5 * hidden, 16 * ranks) // ranks)
        weights = hidden * (q + 2 * kv) + q * hidden + 3 * hidden * inter
        m = _log_int(rng, 1, min(4096, max(1, int(2e12 / (2 * weights)))))
        return dict(kind="layer", m=m, hidden=hidden, q=q, kv=kv, inter=inter)
    requant = rng.random() < 0.3
    bias = rng.random() < 0.6
    x = rng.choice(["normal", "outlier", "student"])
    k = _log_int(rng, 1024, 28672, 16)
    n = _log_int(rng, 1024, 28672, 16 if requant else 8)
    if kind == "host":
        m = _log_int(rng, 16, max(16, min(4096, (24 << 20) // (2 * max(n, k)))))
    else:
        m = _log_int(rng, 1, min(8192, int(3.8e12 / (2 * k * n))))
    return dict(kind=kind, m=m, k=k, n=n, bias=bias, requant=requant, x=x)


# ---- inputs ------------------------------------------------------------------------------------------------------

def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(0xB2000000 + int(seed))
    return g


def _activations(g, m, k, how):
    """fp16 [m, k]: N(0, 1); N(0, 1) with 1 % of the channels x 50; or Student-t(3) clipped to +-200."""
    x = torch.randn((m, k), generator=g, device="cuda")
    if how == "outlier":
        x[:, torch.randperm(k, generator=g, device="cuda")[:k // 100]] *= 50.0
    elif how == "student":
        d = torch.zeros_like(x)
        for _ in range(3):
            d += torch.randn((m, k), generator=g, device="cuda").square_()
        x = (x / (d / 3.0).sqrt_()).clamp_(-200.0, 200.0)
    return x.to(torch.float16)


def _weights(g, n, k):
    """int8 [n, k] uniform on [-127, 127]."""
    return torch.randint(-127, 128, (n, k), generator=g, device="cuda", dtype=torch.int8)


def _column_scales(g, n, lo, hi):
    s = torch.rand((n,), generator=g, device="cuda") * (hi - lo) + lo
    return (s * HIDDEN_UP).to(torch.float16)


def _bias(g, n):
    return (torch.randn((n,), generator=g, device="cuda") * 0.02).to(torch.float16)


def _weight_range(k):
    """Column scales that keep the outputs of a layer's linears of order one (weights of variance 1 / k)."""
    s = (1.0 / k) ** 0.5 / 73.0  # 73: root mean square of the uniform int8 weights
    return 0.7 * s, 1.3 * s


def prepare(case, seed):
    g = _generator(seed)
    if case["kind"] == "layer":
        return _prepare_layer(case, g)
    m, k, n = case["m"], case["k"], case["n"]
    w = _weights(g, n, k)
    scale_n = _column_scales(g, n, 0.001, 0.01) if k <= 8192 else _column_scales(g, n, 0.0005, 0.005)
    bias = _bias(g, n) if case["bias"] else None
    x = _activations(g, m, k, case["x"])
    if case["kind"] == "host":
        s = dict(kind="host", linear=pplb200.W8A8LinearHost(w, scale_n, bias, max_tokens=m, requant=case["requant"]))
        s["x"] = x.cpu().pin_memory()
        s["y"] = torch.empty((m, n), dtype=torch.float16).pin_memory()
        s["yq"] = torch.empty((m, n), dtype=torch.int8).pin_memory() if case["requant"] else None
        s["ys"] = torch.empty((m,), dtype=torch.float16).pin_memory() if case["requant"] else None
        return s
    return dict(kind="linear", x=x, linear=pplb200.W8A8Linear(w, scale_n, bias, max_tokens=m, requant=case["requant"]))


def _prepare_layer(case, g):
    m, hidden, q, kv, inter = (case[v] for v in ("m", "hidden", "q", "kv", "inter"))
    qkv = q + 2 * kv
    s = dict(case, qkv=qkv)
    s["x"] = _activations(g, m, hidden, "normal")            # output of the previous layer's MLP
    s["residual"] = _activations(g, m, hidden, "outlier")    # the residual stream carries the outlier channels
    s["attn"] = _activations(g, m, q, "normal")              # what attention, which is not this library's, returned
    for name, n, k in (("qkv", qkv, hidden), ("o", hidden, q), ("gate_up", 2 * inter, hidden), ("down", hidden, inter)):
        s["w_" + name] = _weights(g, n, k)
        s["sn_" + name] = _column_scales(g, n, *_weight_range(k))
    s["bias_qkv"] = _bias(g, qkv)
    for name in ("norm_in", "norm_post"):
        s[name] = (torch.rand((hidden,), generator=g, device="cuda") + 0.5).to(torch.float16)
    # workspaces and output buffers that a program keeps from call to call
    s["acc"] = torch.empty((m, qkv), dtype=torch.int32, device="cuda")
    s["act"] = (torch.empty((m, inter), dtype=torch.float16, device="cuda"),
                torch.empty((m, inter), dtype=torch.int8, device="cuda"), torch.empty((m,), dtype=torch.float16, device="cuda"))
    s["o"] = torch.empty((m, hidden), dtype=torch.float16, device="cuda")
    s["y"] = torch.empty((m, hidden), dtype=torch.float16, device="cuda")
    need = pplb200.gemm_workspace_bytes(m, max(qkv, hidden), max(hidden, q, inter), pplb200.EPI_DEQUANT_F16)
    s["ws"] = torch.empty((max(need, 256),), dtype=torch.uint8, device="cuda")
    need = pplb200.lib.pplb200_i8i8_gate_up_swiglu_workspace_bytes(m, inter, hidden)
    s["ws_gate_up"] = torch.empty((need,), dtype=torch.uint8, device="cuda")
    # Decoding replays a captured graph, step after step; a prefill, whose length differs from call to call, does not.
    if m <= 256:
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            _layer(s)
        torch.cuda.current_stream().wait_stream(side)
        s["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(s["graph"]):
            s["out"] = _layer(s)
    return s


def _layer(s):
    """Everything of one transformer layer that the library computes, before and after attention."""
    hidden, q, kv, qkv, inter = (s[v] for v in ("hidden", "q", "kv", "qkv", "inter"))
    residual, xq, xs = pplb200.skip_rmsnorm_minmax_quantize_fp16(s["x"], s["norm_in"], skip=s["residual"])
    acc = pplb200.column_parallel_linear(xq, s["w_qkv"], xs, s["sn_qkv"], None, hidden, qkv, gather_output=False,
                                         out=s["acc"], ws=s["ws"])
    heads = pplb200.minmax_dequantize_split3_fp16(acc, xs, s["sn_qkv"], (q, kv, kv), bias=s["bias_qkv"])
    aq, as_ = pplb200.minmax_quantize_fp16(s["attn"])
    o = pplb200.row_parallel_linear(aq, s["w_o"], as_, s["sn_o"], None, q, hidden, out=s["o"], ws=s["ws"])
    residual, hq, hs = pplb200.skip_rmsnorm_minmax_quantize_fp16(o, s["norm_post"], skip=residual)
    _, gq, gs = pplb200.gate_up_swiglu_requant(hq, s["w_gate_up"], hs, s["sn_gate_up"], ws=s["ws_gate_up"], out=s["act"])
    y = pplb200.row_parallel_linear(gq, s["w_down"], gs, s["sn_down"], None, inter, hidden, out=s["y"], ws=s["ws"])
    return dict(q=heads[0], k=heads[1], v=heads[2], residual=residual, y=y)


def run(state):
    if state["kind"] == "linear":
        return state["linear"](state["x"])
    if state["kind"] == "host":
        state["linear"](state["x"], state["y"], state["yq"], state["ys"])
        return [t for t in (state["y"], state["yq"], state["ys"]) if t is not None]
    if "graph" in state:
        state["graph"].replay()
        return state["out"]
    return _layer(state)


def work(case):
    """Activations and results once each, weights, scales and bias once; two operations per multiply-add."""
    m = case["m"]
    if case["kind"] == "layer":
        hidden, q, kv, inter = (case[v] for v in ("hidden", "q", "kv", "inter"))
        weights = hidden * (q + 2 * kv) + q * hidden + 3 * hidden * inter
        scales = 2 * (2 * (q + 2 * kv) + hidden + 2 * inter + hidden + 2 * hidden)
        # in: x, residual, attention output; out: q, k, v, residual, y
        return {"bytes": weights + scales + 2 * m * (2 * hidden + q) + 2 * m * (q + 2 * kv + 2 * hidden), "flops": 2 * m * weights}
    k, n = case["k"], case["n"]
    moved = 2 * m * k + n * k + 2 * n + 2 * m * n
    if case["bias"]:
        moved += 2 * n
    if case["requant"]:
        moved += m * n + 2 * m
    return {"bytes": moved, "flops": 2 * m * n * k}


def tolerance(case):
    # Quantizer, integer GEMM and dequantizer are defined to the bit.
    if case["kind"] != "layer":
        return "exact"
    # The layer contains sums of squares, reciprocal square roots and exponentials.  Where another order or width of those
    # moves a value over a rounding boundary, an int8 activation changes by one step or a token's fp16 scale by one
    # ulp, and all outputs of that token move with it.  Measured over a dozen shapes against the same path with these parts
    # in 64 bits: relative error of y 0 to 0.007 (0.0045 typically), largest difference 0.15 of y's rms; of q, k, v and the
    # residual 1.5e-4 and 0.01.
    return {"rel": 2e-2, "max": 0.6}
