"""The work that a user of this package has it do, as cases to be timed and compared.

Kinds of case (the `kind` of a case dict):

  linear    one quantised linear on an activation: QLinearLayer.forward or, with api "op", the fused op
            that the serving plugin calls.  quant "SHARQ" or "NVFP4"; fused=False is the reference's
            call pattern (sparse GEMM, dense GEMM with beta = 1, separate bias add).
  path      the four quantised linears of a dense decoder layer as a serving engine drives them: RMSNorm
            prepare -> qkv, attention output -> o_proj, residual add + RMSNorm prepare -> gate_up, SwiGLU
            prepare -> down.  graph=True replays the captured path, as engines do for decode steps.
            tp > 1: one rank's column- / row-parallel shards (the collectives belong to other code).
  layer     one whole decoder layer (attention included), dense or mixture of experts.
  weight    quantisation of a bf16 weight (checkpoint conversion, model load).

Sizes: Llama-3-8B, Qwen2.5-7B and Mixtral-8x7B shapes (the package's own configurations), token counts
from 1 to 16384, and generic widths.  Activations are N(0, 1) with 1 % of the channels 20 times larger,
weights N(0, 0.02), norm weights 1 + N(0, 0.1).
"""
import math

import torch

from sharq_b200 import ops
from sharq_b200.decoder import DecoderConfig, SharqDecoderLayer, rope_tables
from sharq_b200.qlinear import QLinearLayer
from sharq_b200.quantize import quantize_weight_nvfp4, quantize_weight_shared_nvfp4

DEV = "cuda"
EPS = 1e-6
CONFIGS = {"llama": DecoderConfig.llama3_8b, "qwen": DecoderConfig.qwen25_7b, "mixtral": DecoderConfig.mixtral_8x7b}


def listed():
    return [
        # one token through one projection of a served model: latency and launches
        {"name": "decode 1 o_proj", "kind": "linear", "m": 1, "n": 4096, "k": 4096, "quant": "SHARQ", "fused": True,
         "bias": False, "api": "op"},
        # a decode batch through a long-K projection, eager
        {"name": "decode 16 down", "kind": "linear", "m": 16, "n": 4096, "k": 14336, "quant": "SHARQ", "fused": True,
         "bias": False, "api": "module"},
        # a decode batch through the linears of a layer, captured in a CUDA graph
        {"name": "decode 32 llama path", "kind": "path", "model": "llama", "m": 32, "tp": 1, "graph": True},
        # an odd chunk of prompt and decode tokens through the linears of a model with qkv bias
        {"name": "chunk 211 qwen path", "kind": "path", "model": "qwen", "m": 211, "tp": 1, "graph": False},
        # the reference's call pattern on a ragged prompt
        {"name": "two-call 777 qkv", "kind": "linear", "m": 777, "n": 4608, "k": 3584, "quant": "SHARQ", "fused": False,
         "bias": True, "api": "module"},
        # the dense NVFP4 mode
        {"name": "nvfp4 1000 down", "kind": "linear", "m": 1000, "n": 4096, "k": 14336, "quant": "NVFP4", "fused": True,
         "bias": False, "api": "module"},
        # a short prompt through a layer
        {"name": "prompt 173 llama layer", "kind": "layer", "model": "llama", "batch": 1, "seq": 173},
        # a 2048-token prefill: the linears, and the layer with its attention
        {"name": "prefill 2048 llama path", "kind": "path", "model": "llama", "m": 2048, "tp": 1, "graph": True},
        {"name": "prefill 2048 llama layer", "kind": "layer", "model": "llama", "batch": 1, "seq": 2048},
        # batched prefills
        {"name": "prefill 8x2048 qwen layer", "kind": "layer", "model": "qwen", "batch": 8, "seq": 2048},
        {"name": "prefill 4x4096 moe layer", "kind": "layer", "model": "mixtral", "batch": 4, "seq": 4096},
        # a projection of a model being converted
        {"name": "weight gate_up", "kind": "weight", "n": 28672, "k": 4096, "quant": "SHARQ"},
    ]


def _spread(rng, low, high):
    """A whole number from low to high, spread over its logarithm."""
    return min(high, max(low, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    kind = rng.choice(["linear", "linear", "linear", "path", "path", "path", "layer", "layer", "weight"])
    if kind == "linear":
        quant = rng.choice(["SHARQ", "SHARQ", "NVFP4"])
        fused = quant == "NVFP4" or rng.random() < 0.7
        bias = rng.random() < 0.3
        api = "op" if quant == "SHARQ" and fused and not bias and rng.random() < 0.5 else "module"
        return {"kind": "linear", "m": _spread(rng, 1, 8192), "n": 8 * _spread(rng, 64, 3584), "k": 128 * _spread(rng, 4, 148),
                "quant": quant, "fused": fused, "bias": bias, "api": api}
    if kind == "path":
        return {"kind": "path", "model": rng.choice(["llama", "qwen"]), "m": _spread(rng, 1, 8192),
                "tp": rng.choice([1, 1, 2, 4]), "graph": rng.random() < 0.5}
    if kind == "layer":
        batch = rng.choice([1, 2, 4, 8])
        return {"kind": "layer", "model": rng.choice(["llama", "qwen", "mixtral"]), "batch": batch,
                "seq": _spread(rng, 16, 8192 // batch)}
    quant = rng.choice(["SHARQ", "NVFP4"])
    n = 8 * _spread(rng, 64, 3584)
    return {"kind": "weight", "n": n if quant == "SHARQ" else -(-n // 128) * 128, "k": 128 * _spread(rng, 4, 148), "quant": quant}


# ------------------------------------------------------------------------------------------ inputs

def _activation(gen, m, k):
    x = torch.randn(m, k, generator=gen, device=DEV)
    x[:, torch.randperm(k, generator=gen, device=DEV)[: max(1, k // 100)]] *= 20.0
    return x.to(torch.bfloat16)


def _weight(gen, n, k):
    return (0.02 * torch.randn(n, k, generator=gen, device=DEV)).to(torch.bfloat16)


def _norm(gen, k):
    return (1 + 0.1 * torch.randn(k, generator=gen, device=DEV)).to(torch.bfloat16)


def _linear(gen, n, k, quant="SHARQ", bias=False, fused=True):
    lin = torch.nn.utils.skip_init(torch.nn.Linear, k, n, bias=bias, device=DEV, dtype=torch.bfloat16)
    lin.weight.data.copy_(_weight(gen, n, k))
    if bias:
        lin.bias.data.copy_((0.02 * torch.randn(n, generator=gen, device=DEV)).to(torch.bfloat16))
    return QLinearLayer(lin, quant_type=quant, fused_gemm=fused)


def _path_shapes(case):
    """(n, k, bias) of this rank's qkv, o_proj, gate_up and down."""
    cfg, tp = CONFIGS[case["model"]](), case.get("tp", 1)
    heads, kv, ffn = cfg.heads // tp, cfg.kv_heads // tp, -(-cfg.ffn // (128 * tp)) * 128
    return {"qkv": ((heads + 2 * kv) * cfg.head_dim, cfg.hidden, cfg.qkv_bias), "o": (cfg.hidden, heads * cfg.head_dim, False),
            "gate_up": (2 * ffn, cfg.hidden, False), "down": (cfg.hidden, ffn, False)}


def prepare(case, seed):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    kind = case["kind"]
    if kind == "linear":
        return {"kind": kind, "api": case["api"], "x": _activation(gen, case["m"], case["k"]),
                "lin": _linear(gen, case["n"], case["k"], case["quant"], case["bias"], case["fused"])}
    if kind == "path":
        shapes = _path_shapes(case)
        st = {"kind": kind, "x": _activation(gen, case["m"], shapes["qkv"][1]),
              "attn": _activation(gen, case["m"], shapes["o"][1]), "g1": _norm(gen, shapes["qkv"][1]),
              "g2": _norm(gen, shapes["qkv"][1]), "graph": None}
        st["lins"] = {name: _linear(gen, n, k, bias=bias) for name, (n, k, bias) in shapes.items()}
        if case["graph"]:
            side = torch.cuda.Stream()
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):
                _path(st)
            torch.cuda.current_stream().wait_stream(side)
            st["graph"] = torch.cuda.CUDAGraph()
            with torch.cuda.graph(st["graph"]):
                st["out"] = _path(st)
        return st
    if kind == "layer":
        cfg = CONFIGS[case["model"]](layers=1)
        layer = SharqDecoderLayer(cfg, gen, torch.device(DEV, torch.cuda.current_device()))
        cos, sin = rope_tables(case["seq"], cfg.head_dim, cfg.rope_theta, DEV)
        x = _activation(gen, case["batch"] * case["seq"], cfg.hidden).view(case["batch"], case["seq"], cfg.hidden)
        return {"kind": kind, "layer": layer, "x": x, "cos": cos, "sin": sin}
    return {"kind": kind, "quant": case["quant"], "w": _weight(gen, case["n"], case["k"])}


# ------------------------------------------------------------------------------------------ passes

def _path(st):
    lin = st["lins"]
    qkv = lin["qkv"].apply_prepared(lin["qkv"].prepare_input_rmsnorm(st["x"], st["g1"], EPS))
    o = lin["o"].apply_prepared(lin["o"].prepare_input(st["attn"]))
    prep, x2 = lin["gate_up"].prepare_input_add_rmsnorm(st["x"], o, st["g2"], EPS)
    gate_up = lin["gate_up"].apply_prepared(prep)
    down = lin["down"].apply_prepared(lin["down"].prepare_input_swiglu(gate_up))
    return {"qkv": qkv, "residual": x2, "gate_up": gate_up, "down": down}


def run(state):
    kind = state["kind"]
    if kind == "linear":
        lin = state["lin"]
        if state["api"] == "op":
            return ops.sharq_linear_forward(state["x"], lin.weight_q, lin.scale_w_sparse, lin.scale_w_dense,
                                            lin.weight_scale_host)
        return lin(state["x"])
    if kind == "path":
        if state["graph"] is not None:
            state["graph"].replay()
            return state["out"]
        return _path(state)
    if kind == "layer":
        return state["layer"](state["x"], state["cos"], state["sin"])
    if state["quant"] == "SHARQ":
        return quantize_weight_shared_nvfp4(state["w"])
    q, sf, scale = quantize_weight_nvfp4(state["w"])
    # the spare band behind the scale factors of the N rows (a multiple of 128 here) is not part of the result
    return q, sf[: state["w"].numel() // 16], scale


# ------------------------------------------------------------------------------------------ work

def _gemm_work(m, n, k, shared=True):
    """Packed weight (payload and the scales its passes read) and output bytes, dense-equivalent flops."""
    return n * k * (0.5 + 1 / 16 + (1 / 32 if shared else 0)) + 2 * m * n, 2.0 * m * n * k


def work(case):
    kind = case["kind"]
    if kind == "linear":
        b, f = _gemm_work(case["m"], case["n"], case["k"], case["quant"] == "SHARQ")
        return {"bytes": b + 2 * case["m"] * case["k"], "flops": f}
    if kind == "weight":
        scales = 1 / 16 + (1 / 32 if case["quant"] == "SHARQ" else 0)
        return {"bytes": case["n"] * case["k"] * (2 + 0.5 + scales), "flops": 0}
    cfg = CONFIGS[case["model"]]()
    m = case["m"] if kind == "path" else case["batch"] * case["seq"]
    shapes = _path_shapes(case)
    total = flops = 0.0
    for name, (n, k, _) in shapes.items():
        if cfg.experts and name in ("gate_up", "down"):
            used = min(cfg.experts, m * cfg.top_k)
            total += used * n * k * (0.5 + 3 / 32)
            flops += 2.0 * m * cfg.top_k * n * k
        else:
            total += n * k * (0.5 + 3 / 32)
            flops += 2.0 * m * n * k
    if kind == "path":  # inputs x and attn; outputs qkv, residual, gate_up, down
        total += 2 * m * (shapes["qkv"][1] + shapes["o"][1] + sum(s[0] for s in (shapes["qkv"], shapes["gate_up"], shapes["down"]))
                          + shapes["qkv"][1])
        return {"bytes": total, "flops": flops}
    flops += 2.0 * case["batch"] * case["seq"] ** 2 * cfg.heads * cfg.head_dim  # causal attention
    return {"bytes": total + 4 * m * cfg.hidden, "flops": flops}


def tolerance(case):
    """About four times the largest distance seen, over these ranges, from the same path with every FP4 product
    replaced by the float64 product of the dequantised operands.  The sums of a linear are nearly exact in
    float32 (rel 3e-5, max one bf16 step); behind a second quantisation a different bf16 step moves FP4 codes
    (path: rel 5e-4, max 4e-2), more so behind attention and routing (layer: rel 6e-3, max 9e-2)."""
    if case["kind"] == "weight":
        return "exact"
    return {"linear": {"rel": 1.2e-4, "max": 0.04}, "path": {"rel": 2e-3, "max": 0.17},
            "layer": {"rel": 2.5e-2, "max": 0.35}}[case["kind"]]
