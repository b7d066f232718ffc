"""Performance cases of the MoE layer and its neighbours, through the package's public entry points.

``listed()`` names the cases, ``draw(rng)`` gives further ones of the same ranges. ``prepare`` makes
what a user's program has in hand before the call (weights quantised and laid out once, plan,
workspace, inputs), ``run`` is one pass, ``work`` the bytes and operations the pass cannot do without.

Five kinds of pass:

* ``layer``    the whole MoE layer in one eager call (``ops.moe_layer_execute``);
* ``block``    one decoder block's share of a serving step: residual add + RMSNorm + NVFP4 codes, then the
               MoE layer with the following residual add + norm folded in, replayed from a CUDA graph as
               the hybrid decode loop replays its step;
* ``experts``  routed experts on precomputed top-k routes (``ops.moe_execute_bf16``, the drop-in symbol);
* ``gemm``     dense bf16 projection (``GemmContext.gemm_bf16``): LM head, attention projections;
* ``quantise`` weight quantisation at load time.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from qs3_b200 import capi, ops, workload

# the shapes of BASELINE.json's configurations: hidden, experts, top-k, intermediate, shared intermediate
SHAPES = {
    "qwen3next": (2048, 512, 10, 512, 512),
    "qwen3_30b_a3b": (2048, 128, 8, 768, 0),
    "tiny": (256, 8, 2, 128, 0),
}
ZIPF = 1.1      # skewed expert load of the prefill configuration
VOCAB = 151936


def listed():
    return [
        # the smallest configuration: launches and host work decide
        dict(name="tiny_bf16_16", kind="layer", fmt="bf16", shape="tiny", tokens=16, zipf=0.0),
        # one sequence decoded at a time, as the upstream runtime does
        dict(name="nvfp4_decode_1", kind="layer", fmt="nvfp4", shape="qwen3next", tokens=1, zipf=0.0),
        # a decode batch inside the graph-replayed serving step
        dict(name="nvfp4_block_128", kind="block", fmt="nvfp4", shape="qwen3next", tokens=128, zipf=0.0),
        # a chunk of a chunked prefill (or a large decode batch): odd, about twenty rows per expert
        dict(name="nvfp4_chunk_1021", kind="layer", fmt="nvfp4", shape="qwen3next", tokens=1021, zipf=0.0),
        # the headline prefill batch with its skewed router
        dict(name="nvfp4_prefill_8192", kind="layer", fmt="nvfp4", shape="qwen3next", tokens=8192, zipf=ZIPF),
        # FP8 checkpoint: the decode batch of the configurations, and a prefill of the same weights
        dict(name="fp8_decode_64", kind="layer", fmt="fp8", shape="qwen3_30b_a3b", tokens=64, zipf=0.0),
        dict(name="fp8_prefill_4096", kind="layer", fmt="fp8", shape="qwen3_30b_a3b", tokens=4096, zipf=0.0),
        # bf16 checkpoint: an odd decode batch through the drop-in call, and a prefill with the shared expert
        dict(name="bf16_experts_33", kind="experts", fmt="bf16", shape="qwen3_30b_a3b", tokens=33, zipf=0.0),
        dict(name="bf16_prefill_2048", kind="layer", fmt="bf16", shape="qwen3next", tokens=2048, zipf=0.0),
        # LM head of a decode batch, and an attention-sized projection of a ragged prefill chunk
        dict(name="lm_head_128", kind="gemm", fmt="bf16", rows=128, k=2048, n=VOCAB),
        dict(name="projection_3001", kind="gemm", fmt="bf16", rows=3001, k=2048, n=4096),
        # a bf16 checkpoint loaded into an NVFP4 plan: 64 experts' gate_up
        dict(name="quantise_nvfp4_64", kind="quantise", fmt="nvfp4", experts=64, rows=1024, k=2048, gated=True),
    ]


def _log_int(rng, low, high):
    return min(high, max(low, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    kind = rng.choices(["layer", "block", "experts", "gemm", "quantise"], [10, 3, 2, 3, 2])[0]
    if kind == "layer":
        fmt = rng.choices(["nvfp4", "fp8", "bf16"], [4, 3, 3])[0]
        # the FP8 layer takes no shared expert, so FP8 checkpoints have the other shape
        shape = {"nvfp4": "qwen3next", "fp8": "qwen3_30b_a3b"}.get(fmt) or rng.choice(["qwen3next", "qwen3_30b_a3b"])
        tokens = _log_int(rng, 1, {"nvfp4": 8192, "fp8": 4096, "bf16": 2048}[fmt])
        return dict(kind=kind, fmt=fmt, shape=shape, tokens=tokens, zipf=rng.choice([0.0, ZIPF]))
    if kind == "block":
        return dict(kind=kind, fmt="nvfp4", shape="qwen3next", tokens=_log_int(rng, 1, 512), zipf=0.0)
    if kind == "experts":
        return dict(kind=kind, fmt="bf16", shape="qwen3_30b_a3b", tokens=_log_int(rng, 1, 512), zipf=0.0)
    if kind == "gemm":
        if rng.random() < 0.3:
            return dict(kind=kind, fmt="bf16", rows=_log_int(rng, 1, 256), k=2048, n=VOCAB)
        return dict(kind=kind, fmt="bf16", rows=_log_int(rng, 1, 4096), k=rng.choice([512, 2048, 4096]),
                    n=rng.choice([512, 2048, 4096, 8192]))
    fmt = rng.choice(["nvfp4", "fp8"])
    gated = rng.choice([True, False])
    rows, k = rng.choice([(1024, 2048), (1536, 2048)] if gated else [(2048, 512), (2048, 768)])
    return dict(kind=kind, fmt=fmt, experts=_log_int(rng, 1, 128), rows=rows, k=k, gated=gated)


# ------------------------------------------------------------------------------ inputs ---

def _normal(shape, std, gen):
    return (torch.randn(shape, generator=gen, device="cuda") * std).to(torch.bfloat16)


class _Layer:
    """Weights, plan, workspace and tokens of one MoE layer."""

    def __init__(self, case, seed, stream=None):
        h, experts, top_k, inter, shared = SHAPES[case["shape"]]
        self.tokens = case["tokens"]
        cfg = workload.LayerConfig("case", self.tokens, h, experts, top_k, inter, shared,
                                   nvfp4=case["fmt"] == "nvfp4", zipf_s=case["zipf"], fp8=case["fmt"] == "fp8")
        self.ctx = ops.Context(torch.cuda.current_device(), stream)
        self.data = workload.LayerData(cfg, self.ctx, seed=seed)
        self.plan = self.data.plan(self.ctx)
        self.workspace = torch.zeros(self.plan.layer_workspace_size(self.tokens, shared), dtype=torch.uint8,
                                     device="cuda")
        self.out = torch.empty((self.tokens, h), dtype=torch.bfloat16, device="cuda")

    def execute(self, **more):
        d = self.data
        ops.moe_layer_execute(self.plan, more.pop("hidden", d.hidden), d.router, d.gate_up, d.down, self.out,
                              self.workspace, router_bias=d.bias, shared=d.shared, **more)


class _Block:
    """The calls of one decoder block around the MoE layer, captured once and replayed per token."""

    def __init__(self, case, seed):
        self.stream = torch.cuda.Stream()
        self.stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(self.stream):
            self.layer = _Layer(case, seed, self.stream.cuda_stream)
            t, h = self.layer.data.hidden.shape
            gen = torch.Generator(device="cuda").manual_seed(seed + 5)
            # what the mixer and the residual stream hand over for this token
            self.mixed, self.residual_in = self.layer.data.hidden, _normal((t, h), 1.0, gen)
            self.norm_weight = (1.0 + torch.randn(h, generator=gen, device="cuda") * 0.1).to(torch.bfloat16)
            self.next_weight = (1.0 + torch.randn(h, generator=gen, device="cuda") * 0.1).to(torch.bfloat16)
            self.x = torch.empty_like(self.mixed)
            self.residual = torch.empty_like(self.residual_in)
            self.packed = torch.empty((t, h // 2), dtype=torch.uint8, device="cuda")
            self.tiled = torch.zeros(ops.nvfp4_tiled_scale_bytes(t, h), dtype=torch.uint8, device="cuda")
            self.step()
            self.stream.synchronize()
            self.graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(self.graph, stream=self.stream):
                self.step()
        torch.cuda.current_stream().wait_stream(self.stream)

    def step(self):
        self.x.copy_(self.mixed)
        self.residual.copy_(self.residual_in)
        ops.fused_add_rmsnorm_nvfp4(self.layer.ctx, self.x, self.residual, self.norm_weight, packed=self.packed,
                                    tiled=self.tiled)
        self.layer.execute(hidden=self.x, hidden_packed=self.packed, hidden_scale_tiled=self.tiled,
                           residual_inout=self.residual, next_norm_weight=self.next_weight)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "layer":
        return case, _Layer(case, seed)
    if kind == "block":
        return case, _Block(case, seed)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if kind == "experts":
        layer = _Layer(case, seed)
        logits = torch.randn((case["tokens"], layer.data.cfg.experts), generator=gen, device="cuda")
        weights, ids = logits.softmax(dim=1).topk(layer.data.cfg.top_k, dim=1)
        ids, weights = ids.to(torch.int32).contiguous(), (weights / weights.sum(dim=1, keepdim=True)).contiguous()
        plan = ops.MoePlan(layer.ctx, ops.MoePlanConfig(
            max_num_tokens=case["tokens"], hidden_size=layer.data.cfg.hidden,
            intermediate_size=layer.data.cfg.inter, num_experts=layer.data.cfg.experts,
            top_k=layer.data.cfg.top_k, backend=capi.MOE_BACKEND_STAGED_BF16))
        workspace = torch.zeros(plan.workspace_size(case["tokens"]), dtype=torch.uint8, device="cuda")
        return case, (layer, plan, ids, weights, workspace)
    if kind == "gemm":
        x = _normal((case["rows"], case["k"]), 1.0, gen)
        weight = _normal((case["n"], case["k"]), 0.02, gen)
        out = torch.empty((case["rows"], case["n"]), dtype=torch.bfloat16, device="cuda")
        return case, (ops.GemmContext(), x, weight, out)
    weight = _normal((case["experts"], case["rows"], case["k"]), 0.02, gen)
    return case, (ops.Context(), weight)


def run(state):
    case, s = state
    kind = case["kind"]
    if kind == "layer":
        s.execute()
        return s.out
    if kind == "block":
        s.graph.replay()
        return s.layer.out, s.residual, s.x, s.packed
    if kind == "experts":
        layer, plan, ids, weights, workspace = s
        ops.moe_execute_bf16(plan, layer.data.hidden, ids, weights, layer.data.gate_up, layer.data.down, layer.out,
                             workspace)
        return layer.out
    if kind == "gemm":
        ctx, x, weight, out = s
        ctx.gemm_bf16(x, weight, out, alpha=1.0)
        return out
    ctx, weight = s
    if case["fmt"] == "fp8":
        q = ops.fp8_quantize_weight(ctx, weight)
        return q.codes, q.scale
    q = ops.nvfp4_quantize_weight(ctx, weight, case["gated"])
    return q.packed, q.scale_linear, q.scale_tiled, q.global_scale


# -------------------------------------------------------------------------------- work ---

@functools.lru_cache(maxsize=None)
def _route_share(shape, zipf):
    """Share of the tokens that choose each expert, from a seeded sample of router logits."""
    h, experts, top_k, _, _ = SHAPES[shape]
    rng = np.random.RandomState(0)
    logits = rng.standard_normal((2048, experts)) * 0.02 * math.sqrt(h)
    if zipf:
        logits -= zipf * np.log1p(np.arange(experts))
    ids = np.argpartition(-logits, top_k - 1, axis=1)[:, :top_k]
    return np.bincount(ids.ravel(), minlength=experts) / logits.shape[0]


def work(case):
    """Every weight an expert with a route needs once, every token and result once; no intermediate."""
    kind = case["kind"]
    if kind == "gemm":
        m, k, n = case["rows"], case["k"], case["n"]
        return {"bytes": 2 * (m * k + n * k + m * n), "flops": 2 * m * k * n}
    if kind == "quantise":
        n = case["experts"] * case["rows"] * case["k"]
        # nvfp4: codes, row-major and tiled block scales; fp8: codes and one f32 per 128 x 128
        return {"bytes": int(n * (2 + 0.5 + 2 / 16) if case["fmt"] == "nvfp4" else n * (2 + 1 + 4 / 16384)), "flops": 0}
    t = case["tokens"]
    h, experts, top_k, inter, shared = SHAPES[case["shape"]]
    share = _route_share(case["shape"], case["zipf"])
    hit = float(np.sum(1.0 - (1.0 - share) ** t))
    per_weight = {"nvfp4": 9 / 16, "fp8": 1 + 4 / 16384, "bf16": 2.0}[case["fmt"]]
    bytes_ = hit * 3 * inter * h * per_weight + t * h * 2 * 2
    flops = 2 * t * top_k * 3 * inter * h
    if kind == "experts":
        bytes_ += t * top_k * 8
    else:
        bytes_ += experts * h * 2                      # router
        flops += 2 * t * experts * h
        if shared:
            bytes_ += 3 * shared * h * per_weight + h * 2
            flops += 2 * t * 3 * shared * h
    if kind == "block":
        bytes_ += t * h * 2 * 3 + t * h // 2           # residual in and out, normed tokens and their codes out
    return {"bytes": int(bytes_), "flops": int(flops)}


def tolerance(case):
    """Quantised weights are exact (codes and scales follow from the formats' arithmetic). Layer outputs are bf16
    results of bf16 / NVFP4 / FP8 chains whose f32 sums may run in another order: 1e-2 is the tolerance the
    configurations state for them; a code of a re-quantised intermediate that sits on a rounding boundary, or a
    token whose last expert is a near tie, moves single values by a good part of the rms. A projection is one f32
    sum rounded to bf16."""
    if case["kind"] == "quantise":
        return "exact"
    if case["kind"] == "gemm":
        return {"rel": 4e-3, "max": 2e-2}
    if case["kind"] == "block":
        return {"rel": 1e-2, "max": 0.5, "differ": 1e-3}
    return {"rel": 1e-2, "max": 0.5}
