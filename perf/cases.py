"""Performance cases of the block-FP8 path: what an inference server has it do, layer by layer.

Two kinds of pass:

``linears``  the four block-FP8 projections of one dense decoder layer (qkv, o_proj, gate_up, down) on one
             tensor-parallel rank: activations in, 16-bit activations out, quantisation included. The four inputs are
             separate tensors because attention, norms and the activation function sit between the projections.
``moe``      one mixture-of-experts layer: routing of the router logits, then the fused experts.

Widths are the benchmark configurations of this repository (``sglang_b200.synthetic``) and their tensor-parallel
shards; row counts run from one decoded token to a full prefill chunk.
"""
import math

import torch

import sglang_b200 as sb
from sglang_b200.weight_quant import transform_scale_ue8m0

BLOCK = [128, 128]
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}
# hidden size, rows of qkv, intermediate size
DENSE = {"llama3_8b": (4096, 6144, 14336), "llama3_70b": (8192, 10240, 28672)}
# experts, experts per token, hidden size, intermediate size, expert groups, groups kept (0: plain softmax top-k)
EXPERTS = {"mixtral": (8, 2, 4096, 14336, 0, 0), "deepseek_v3": (256, 8, 7168, 2048, 8, 4)}


def _linears(name, model, tp, rows, dtype="bf16", scales="fp32"):
    return {"name": name, "op": "linears", "model": model, "tp": tp, "rows": rows, "dtype": dtype, "scales": scales}


def _moe(name, model, tp, rows, dtype="bf16"):
    return {"name": name, "op": "moe", "model": model, "tp": tp, "rows": rows, "dtype": dtype}


def listed():
    return [
        # one user decoding: weights are read once for a single row, launches and host time count
        _linears("linears_decode_1", "llama3_8b", 1, 1),
        # a small decode batch
        _linears("linears_decode_16", "llama3_8b", 1, 16),
        # a larger decode batch on one rank of four, fp16 model
        _linears("linears_decode_61_tp4_fp16", "llama3_70b", 4, 61, "fp16"),
        # a short prompt, or a decode batch mixed with a piece of one
        _linears("linears_mixed_203", "llama3_8b", 1, 203),
        # an ordinary prefill chunk on one rank of eight, ragged as prompts are
        _linears("linears_prefill_1027_tp8", "llama3_70b", 8, 1027),
        # the largest prefill chunk
        _linears("linears_prefill_8192", "llama3_8b", 1, 8192),
        # prefill of a checkpoint whose scales are powers of two, packed as exponent bytes
        _linears("linears_prefill_3000_ue8m0", "llama3_8b", 1, 3000, "bf16", "ue8m0"),
        # one user decoding through 256 experts
        _moe("moe256_decode_1", "deepseek_v3", 1, 1),
        # a few users through 8 large experts
        _moe("moe8_decode_7", "mixtral", 1, 7),
        # a decode batch that reaches nearly all of the 256 experts
        _moe("moe256_decode_128", "deepseek_v3", 1, 128),
        # a ragged prefill chunk through 8 large experts with skewed load
        _moe("moe8_prefill_3001", "mixtral", 1, 3001),
        # the largest prefill chunk through 256 experts
        _moe("moe256_prefill_16384", "deepseek_v3", 1, 16384),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    dtype = rng.choice(["bf16", "bf16", "bf16", "fp16"])
    if rng.random() < 0.6:
        model = rng.choice(sorted(DENSE))
        tp = rng.choice([1, 2, 4, 8])
        c = _linears("", model, tp, _log_int(rng, 1, 8192), dtype, rng.choice(["fp32", "fp32", "fp32", "ue8m0"]))
    else:
        model = rng.choice(sorted(EXPERTS))
        tp = rng.choice([1, 2, 4, 8])
        c = _moe("", model, tp, _log_int(rng, 1, 16384 if model == "deepseek_v3" else 8192), dtype)
    del c["name"]
    return c


def _shapes(case):
    """(N, K) of the four projections on one rank: qkv and gate_up split by output rows, the others by K."""
    hidden, qkv, inter = DENSE[case["model"]]
    tp = case["tp"]
    return [(qkv // tp, hidden), (hidden, hidden // tp), (2 * inter // tp, hidden), (hidden, inter // tp)]


def _expert_shape(case):
    experts, topk, hidden, inter, groups, kept = EXPERTS[case["model"]]
    return experts, topk, hidden, inter // case["tp"], groups, kept


def _weight(shape, gen):
    """FP8 weights as block quantisation of N(0, 0.02^2) leaves them: the largest value of a 128x128 block lies at
    448, about four standard deviations out, and the scales are nearly alike."""
    q = torch.empty(shape, dtype=torch.float8_e4m3fn, device="cuda")
    rows = q.view(-1, shape[-1])
    step = max(1, (1 << 28) // shape[-1])
    for r in range(0, rows.shape[0], step):
        part = rows[r:r + step]
        part.copy_(torch.randn(part.shape, generator=gen, device="cuda", dtype=torch.bfloat16).mul_(110).clamp_(-448, 448))
    blocks = (*shape[:-2], (shape[-2] + 127) // 128, (shape[-1] + 127) // 128)
    scale = (0.02 / 110) * (1 + 0.1 * torch.rand(blocks, generator=gen, device="cuda"))
    return q, scale


def _activation(rows, width, dtype, gen, outliers):
    """N(0, 1), with one channel in a hundred twenty times larger where asked for."""
    x = torch.randn(rows, width, generator=gen, device="cuda")
    if outliers:
        x[:, torch.randperm(width, generator=gen, device="cuda")[: math.ceil(width / 100)]] *= 20
    return x.to(DTYPES[dtype])


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rows = case["rows"]
    if case["op"] == "linears":
        layers = []
        for n, k in _shapes(case):
            w, s = _weight((n, k), gen)
            if case["scales"] == "ue8m0":
                s = transform_scale_ue8m0(torch.exp2(torch.ceil(torch.log2(s))), mn=n)
            layers.append((_activation(rows, k, case["dtype"], gen, True), w, s))
        return {"op": case["op"], "scales": case["scales"], "layers": layers}
    experts, topk, hidden, inter, groups, kept = _expert_shape(case)
    w1, w1_scale = _weight((experts, 2 * inter, hidden), gen)
    w2, w2_scale = _weight((experts, hidden, inter), gen)
    logits = torch.randn(rows, experts, generator=gen, device="cuda")
    if groups:
        # small against the scores: what is left of the load balancing correction when the experts are trained
        bias = 0.01 * torch.randn(experts, generator=gen, device="cuda")
        routing = sb.TopKConfig(top_k=topk, use_grouped_topk=True, topk_group=kept, num_expert_group=groups, renormalize=True,
                                correction_bias=bias, routed_scaling_factor=2.5, scoring_func="sigmoid")
    else:
        rank = torch.randperm(experts, generator=gen, device="cuda").float() + 1
        logits -= 1.2 * rank.log()  # load falls off as Zipf(1.2) over the experts
        routing = sb.TopKConfig(top_k=topk, renormalize=True)
    runner = sb.MoeRunnerConfig(num_experts=experts, num_local_experts=experts, hidden_size=hidden,
                                intermediate_size_per_partition=inter, top_k=topk, inplace=False,
                                routed_scaling_factor=2.5 if groups else None)
    return {"op": case["op"], "x": _activation(rows, hidden, case["dtype"], gen, False), "logits": logits, "w1": w1, "w2": w2,
            "w1_scale": w1_scale, "w2_scale": w2_scale, "routing": routing, "runner": runner}


def run(state):
    if state["op"] == "linears":
        if state["scales"] == "fp32":
            return [sb.w8a8_block_fp8_linear(x, w, BLOCK, s) for x, w, s in state["layers"]]
        out = []
        for x, w, s in state["layers"]:
            q, qs = sb.per_token_group_quant_fp8(x, 128, column_major_scales=True, scale_tma_aligned=True, scale_ue8m0=True)
            out.append(sb.w8a8_block_fp8_matmul(q, w, qs, s, BLOCK, output_dtype=x.dtype))
        return out
    topk = sb.select_experts(state["x"], state["logits"], state["routing"])
    out = sb.fused_experts(state["x"], state["w1"], state["w2"], topk, state["runner"], use_fp8_w8a8=True,
                           w1_scale=state["w1_scale"], w2_scale=state["w2_scale"], block_shape=BLOCK)
    return {"out": out, "topk_ids": topk.topk_ids, "topk_weights": topk.topk_weights}


def _reached(rows, experts, topk, skewed):
    """Mean number of experts that ``rows`` tokens are routed to: each has topk of them, evenly, or as Zipf(1.2)."""
    if not skewed or rows > 512:
        return experts * (1 - (1 - topk / experts) ** rows)
    gen = torch.Generator().manual_seed(0)
    logits = torch.randn(64, rows, experts, generator=gen) - 1.2 * (torch.arange(experts).float() + 1).log()
    ids = logits.topk(topk, dim=-1).indices.reshape(64, -1)
    return sum(len(set(row)) for row in ids.tolist()) / 64


def work(case):
    rows = case["rows"]
    if case["op"] == "linears":
        scale = 4 if case["scales"] == "fp32" else 1
        bytes_ = sum(n * k + scale * n * k / 16384 + 2 * rows * (n + k) for n, k in _shapes(case))
        return {"bytes": bytes_, "flops": sum(2 * rows * n * k for n, k in _shapes(case))}
    experts, topk, hidden, inter, _, _ = _expert_shape(case)
    reached = _reached(rows, experts, topk, skewed=case["model"] == "mixtral")
    weights = 3 * hidden * inter * (1 + 4 / 16384)
    bytes_ = reached * weights + 4 * rows * hidden + 4 * rows * experts + 8 * rows * topk
    return {"bytes": bytes_, "flops": 6 * rows * topk * hidden * inter}


def tolerance(case):
    # 16-bit results (half an ulp of bf16 is 2e-3 to 4e-3); the experts also round their intermediate to FP8, where another
    # order of the fp32 sums turns a few codes to the neighbouring one. Expert ids are the same.
    return {"rel": 1e-2}
