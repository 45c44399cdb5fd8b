"""The calls a user of this package makes, as cases that can be timed and compared.

Each case is one pass through the public modules (``mindpipe_b200.modules``) on seeded synthetic tensors of the
shapes and distributions the package's benchmark uses (``mindpipe_b200/synth.py``): weights N(0, 0.02), activations
N(0, 1), and for the int8 paths 1 % of the activation channels scaled x20.

``op`` says which path a case takes:

``w4_linear``     one W4A16 linear: ``VllmPackedInt4Linear.forward``
``w4_layer``      the four W4A16 linears of a decoder layer, held row-concatenated as serving runtimes hold them
                  (qkv, o, gate|up, down); ``graph`` replays the same forwards from a captured CUDA graph
``w4_host``       the same four on pinned host activations: ``forward_host_many``
``w8_layer``      the four linears in W8A8: ``SmoothQuantLinear.forward`` (per-token int8 activations)
``affine_layer``  the four linears in asymmetric W8A8: ``QuantLinear.forward``
``moe``           router + top-k experts in W8A8: ``moe_router_topk`` and ``SmoothQuantPackedMoeExperts.forward``
``w4_quantize``   loading: the layer's fp16 weights quantised, packed and expanded again
"""
from __future__ import annotations

import math

import torch

from mindpipe_b200 import _lib, ops, synth
from mindpipe_b200.modules import (QuantLinear, SmoothQuantLinear, SmoothQuantPackedMoeExperts, VllmPackedInt4Linear,
                                   forward_host_many)

SMALL = {"hidden": 4096, "kv": 4096, "inter": 11008}       # LLAMA2_7B_LINEARS
MEDIUM = {"hidden": 4096, "kv": 1024, "inter": 14336}      # LLAMA3_8B_LINEARS
LARGE = {"hidden": 8192, "kv": 1024, "inter": 28672}       # LLAMA2_70B_LINEARS
MOE = {"hidden": synth.MIXTRAL_8X7B.hidden, "ffn": synth.MIXTRAL_8X7B.ffn, "experts": synth.MIXTRAL_8X7B.num_experts,
       "top_k": synth.MIXTRAL_8X7B.top_k}


def listed():
    return [
        # One token through one linear: the smallest call there is, where the host side and the launch count.
        {"name": "w4_linear_m1", "op": "w4_linear", "rows": 1, "n": 4096, "k": 4096, "group": 128, "bias": False,
         "graph": False},
        # A decode step at batch 16 as serving runs it: captured once, replayed per step.
        {"name": "w4_layer_7b_m16_graph", "op": "w4_layer", "rows": 16, "group": 128, "bias": False, "graph": True,
         **SMALL},
        # The same step for a host that keeps its activations in pinned host memory.
        {"name": "w4_host_7b_m16", "op": "w4_host", "rows": 16, "group": 128, "bias": False, **SMALL},
        # A small decode batch on the largest dense layers, launched eagerly.
        {"name": "w4_layer_70b_m8", "op": "w4_layer", "rows": 8, "group": 128, "bias": False, "graph": False, **LARGE},
        # Between decode and prefill: a ragged batch (a short prompt, or many streams), linears with biases.
        {"name": "w4_layer_7b_m77", "op": "w4_layer", "rows": 77, "group": 128, "bias": True, "graph": False, **SMALL},
        # Prefill of a 2048-token prompt.
        {"name": "w4_layer_7b_m2048", "op": "w4_layer", "rows": 2048, "group": 128, "bias": False, "graph": False,
         **SMALL},
        # W8A8: a decode step at a small batch, launched eagerly.
        {"name": "w8_layer_8b_m4", "op": "w8_layer", "rows": 4, "bias": False, "graph": False, **MEDIUM},
        # W8A8: prefill of 4096 tokens.
        {"name": "w8_layer_8b_m4096", "op": "w8_layer", "rows": 4096, "bias": False, "graph": False, **MEDIUM},
        # Asymmetric W8A8: a prompt of odd length, with biases.
        {"name": "affine_layer_7b_m333", "op": "affine_layer", "rows": 333, "bias": True, "graph": False, **SMALL},
        # Mixture of experts: a decode step (every expert's weights are read for a handful of rows), captured.
        {"name": "moe_t32_graph", "op": "moe", "tokens": 32, "graph": True, **MOE},
        # Mixture of experts: a prefill batch, the largest piece of work.
        {"name": "moe_t8192", "op": "moe", "tokens": 8192, "graph": False, **MOE},
        # Loading a layer: fp16 weights to packed int4 and back (the export check's round trip).
        {"name": "w4_quantize_7b", "op": "w4_quantize", "group": 128, **SMALL},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _multiple(rng, lo, hi, of):
    return max(1, _log_int(rng, lo, hi) // of) * of


def draw(rng):
    """A case of the listed ones' ranges: widths of 2048..8192 (hidden) and 2..4 times that (intermediate), 1..4096
    rows (1..16 on the host path, 1..8192 tokens for the experts), never more work than the largest listed cases."""
    op = rng.choice(["w4_linear", "w4_layer", "w4_layer", "w4_layer", "w4_host", "w8_layer", "w8_layer",
                     "affine_layer", "moe", "moe", "w4_quantize"])
    group = rng.choice([128, 128, 128, 64])
    bias = rng.random() < 0.3
    if op == "w4_linear":
        case = {"op": op, "rows": _log_int(rng, 1, 2048), "n": _multiple(rng, 1024, 28672, 8),
                "k": _multiple(rng, 2048, 28672, 128), "group": group, "bias": bias}
    elif op == "moe":
        hidden = _multiple(rng, 1024, 4096, 128)
        case = {"op": op, "tokens": _log_int(rng, 1, 8192), "hidden": hidden,
                "ffn": _multiple(rng, 1024, 14336, 128), "experts": rng.choice([4, 8, 8, 16]), "top_k": 2}
        while case["experts"] * hidden * case["ffn"] > 8 * 4096 * 14336:
            case["experts"] //= 2
    else:
        hidden = _multiple(rng, 2048, 8192, 128)
        case = {"op": op, "hidden": hidden, "kv": max(128, hidden // rng.choice([1, 4, 8]) // 128 * 128),
                "inter": _multiple(rng, 2 * hidden, 4 * hidden if hidden < 7168 else 28672, 128)}
        if op != "w4_quantize":
            case["rows"] = _log_int(rng, 1, 16 if op == "w4_host" else 4096)
            case["bias"] = bias
        if op in ("w4_layer", "w4_host", "w4_quantize"):
            case["group"] = group
    if op not in ("w4_host", "w4_quantize"):
        case["graph"] = case.get("rows", case.get("tokens")) <= 64 and rng.random() < 0.5
    size = "tokens" if op == "moe" else "rows"
    while size in case and work(case)["flops"] > (5.8e12 if op == "moe" else 1.8e12):
        case[size] = case[size] * 3 // 4
    return case


# ------------------------------------------------------------------------------------------------ the layer's linears
def _linears(case):
    """(out_features, in_features) of the case's linears."""
    if case["op"] == "w4_linear":
        return [(case["n"], case["k"])]
    h, kv, i = case["hidden"], case["kv"], case["inter"]
    return [(h + 2 * kv, h), (h, h), (2 * i, h), (h, i)]


def _normal(gen, *shape, std=1.0):
    return torch.randn(shape, generator=gen, device="cuda", dtype=torch.float16).mul_(std)


def _with_outliers(gen, x):
    """1 % of the channels scaled x20, as activations in front of int8 linears have them."""
    k = x.shape[-1]
    hot = torch.randperm(k, generator=gen, device="cuda")[:max(1, k // 100)]
    x[..., hot] *= 20
    return x


def _float_linear(gen, n, k, bias):
    lin = torch.nn.Linear(k, n, bias=bias, device="meta", dtype=torch.float16)
    lin.weight = torch.nn.Parameter(_normal(gen, n, k, std=0.02), requires_grad=False)
    if bias:
        lin.bias = torch.nn.Parameter(_normal(gen, n, std=0.1), requires_grad=False)
    return lin


def _quantised(case, lin):
    if case["op"] == "w8_layer":
        m = SmoothQuantLinear.from_float(lin)
    elif case["op"] == "affine_layer":
        return QuantLinear(lin)
    else:
        m = VllmPackedInt4Linear.from_float(lin, group_size=case["group"])
    m.process_weights_after_loading()
    return m


_capture_stream = None


def _captured(forward):
    """``forward`` captured in a CUDA graph with chained launches, the way a serving runtime prepares a decode step."""
    global _capture_stream
    if _capture_stream is None:
        _capture_stream = torch.cuda.Stream()
    before = _lib.load().mp_set_programmatic_launch(1)
    try:
        _capture_stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(_capture_stream):
            forward()                                   # scratch buffers of this stream exist before the capture
        _capture_stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=_capture_stream):
            out = forward()
    finally:
        _lib.load().mp_set_programmatic_launch(before)
    return graph, out


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    op = case["op"]
    state = {"op": op}
    if op == "moe":
        e, h, f = case["experts"], case["hidden"], case["ffn"]
        experts = SmoothQuantPackedMoeExperts(_normal(gen, e, 2 * f, h, std=0.02), _normal(gen, e, h, f, std=0.02))
        x = _with_outliers(gen, _normal(gen, case["tokens"], h))
        logits = torch.randn((case["tokens"], e), generator=gen, device="cuda")

        def forward():
            index, weights = ops.moe_router_topk(logits, case["top_k"])
            return experts(x, index, weights)
    elif op == "w4_quantize":
        state["linears"] = [_float_linear(gen, n, k, False) for n, k in _linears(case)]
        state["group"] = case["group"]
        return state
    else:
        modules = [_quantised(case, _float_linear(gen, n, k, case["bias"])) for n, k in _linears(case)]
        xs = [_normal(gen, case["rows"], k) for _, k in _linears(case)]
        if op in ("w8_layer", "affine_layer"):
            xs = [_with_outliers(gen, x) for x in xs]
        if op == "w4_host":
            state["modules"] = modules
            state["x"] = [x.cpu().pin_memory() for x in xs]
            state["y"] = [torch.empty((case["rows"], n), dtype=torch.float16).pin_memory() for n, _ in _linears(case)]
            return state

        def forward():
            return [m(x) for m, x in zip(modules, xs)]
    state["forward"] = forward
    if case["graph"]:
        state["graph"], state["out"] = _captured(forward)
    return state


def run(state):
    if "graph" in state:
        state["graph"].replay()
        return state["out"]
    if state["op"] == "w4_host":
        return forward_host_many(state["modules"], state["x"], state["y"])
    if state["op"] == "w4_quantize":
        out = []
        for lin in state["linears"]:
            m = VllmPackedInt4Linear.from_float(lin, group_size=state["group"])
            out.append((m.weight_packed, m.weight_scale, m.weight_zero_point, m.dequantize()))
        return out
    return state["forward"]()


# ------------------------------------------------------------------------------------------------- sizes and accuracy
def work(case):
    op = case["op"]
    if op == "moe":
        t, k, e, h, f = case["tokens"], case["top_k"], case["experts"], case["hidden"], case["ffn"]
        used = e * (1.0 - (1.0 - k / e) ** t)            # experts that at least one token is routed to, on average
        return {"bytes": used * (3 * h * f + 4 * (2 * f + h)) + 4 * t * h + 4 * t * e, "flops": 6.0 * t * k * h * f}
    n_bytes = flops = 0
    for n, k in _linears(case):
        if op == "w4_quantize":
            groups = k // case["group"]
            n_bytes += 2 * n * k + n * k // 2 + 2 * n * groups + 4 * n * ((groups + 7) // 8) + 2 * n * k
            flops += 4 * n * k
            continue
        m = case["rows"]
        if op in ("w4_linear", "w4_layer", "w4_host"):
            weight = n * k // 2 + 2 * n * (k // case["group"]) + n * (k // case["group"]) // 2
        else:
            weight = n * k + (4 * n if op == "w8_layer" else 12 * n)
        n_bytes += weight + 2 * m * k + 2 * m * n + (2 * n if case["bias"] else 0)
        flops += 2 * m * n * k
    return {"bytes": n_bytes, "flops": flops}


def tolerance(case):
    if case["op"] == "w4_quantize":
        return "exact"                                   # codes, scales, zero points and Wdq are defined bit for bit
    if case["op"] == "moe":
        return {"rel": 5e-3}                             # fp16 roundings in SwiGLU decide ties of the second quantisation
    if case["op"] in ("w8_layer", "affine_layer"):
        return {"rel": 1e-3}                             # integer sums are exact; fp16 results
    return {"rel": 2e-3}                                 # fp16 weights and results, 32-bit sums
