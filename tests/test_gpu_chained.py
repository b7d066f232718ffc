"""Calls that follow each other on one workspace without a synchronisation: a chained kernel starts while its predecessor
still runs, so that a wait that is missing anywhere would read the tables, tokens or results of the call before. Every
call has other tokens, and the batches differ in size, so that every layout of the workspace follows every other."""
import numpy as np
import pytest
import torch

from helpers import f32, make_moe_inputs, max_abs, rel_l2, to_dev, to_np

pytestmark = pytest.mark.gpu

H, E, K, I = 512, 16, 2, 256
# one token, 32-, 64- and 128-row token tiles, back to small ones, and the same size twice
BATCHES = (1, 60, 500, 160, 8, 160, 500, 40, 300, 1)


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("fmt", ["bf16", "nvfp4", "fp8"])
def test_calls_without_synchronisation(oracle, fmt, captured):
    from qs3_b200 import capi, ops
    d = make_moe_inputs(61, 1, H, E, I)
    tokens = [make_moe_inputs(70 + n, t, H, 1, 1)["hidden"] for n, t in enumerate(BATCHES)]
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        ctx = ops.Context(torch.cuda.current_device(), stream.cuda_stream)
        gate_up, down, router = to_dev(d["gate_up"]), to_dev(d["down"]), to_dev(d["router"])
        if fmt == "nvfp4":
            gate_up, down = ops.nvfp4_quantize_weight(ctx, gate_up, True), ops.nvfp4_quantize_weight(ctx, down, False)
        elif fmt == "fp8":
            gate_up, down = ops.fp8_quantize_weight(ctx, gate_up), ops.fp8_quantize_weight(ctx, down)
        plan = ops.MoePlan(ctx, ops.MoePlanConfig(
            max_num_tokens=max(BATCHES), hidden_size=H, intermediate_size=I, num_experts=E, top_k=K,
            backend=dict(bf16=capi.MOE_BACKEND_STAGED_BF16, nvfp4=capi.MOE_BACKEND_NVFP4,
                         fp8=capi.MOE_BACKEND_FP8_BLOCKSCALE)[fmt], route_mode=capi.MOE_ROUTE_ROUTER_LOGITS))
        ws = torch.zeros(plan.layer_workspace_size(max(BATCHES), 0), dtype=torch.uint8, device="cuda")
        hidden = [to_dev(x) for x in tokens]
        out = [torch.empty_like(x) for x in hidden]
        ids = [torch.empty((t, K), dtype=torch.int32, device="cuda") for t in BATCHES]
        w = [torch.empty((t, K), dtype=torch.float32, device="cuda") for t in BATCHES]

        def calls():
            for x, o, i, v in zip(hidden, out, ids, w):
                ops.moe_layer_execute(plan, x, router, gate_up, down, o, ws, topk_ids=i, topk_weights=v)
        if captured:
            calls()
            stream.synchronize()
            for o in out:
                o.zero_()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream):
                calls()
            graph.replay()
            graph.replay()
        else:
            torch.cuda.synchronize()
            calls()
        stream.synchronize()
    assert ctx.read_device_error() == 0
    for x, o, i, v in zip(tokens, out, ids, w):
        ref_ids, ref_w = oracle.router_topk(oracle.gemm_bf16(x, d["router"], "f32"), K, 0, True, 1.0)
        assert np.mean(to_np(i) != ref_ids) <= 2e-3   # near ties of the last expert
        assert np.allclose(to_np(v), ref_w, atol=1e-3)
        if fmt == "nvfp4":
            triple = lambda q: (to_np(q.packed), to_np(q.scale_linear), to_np(q.global_scale))
            ref = oracle.moe_nvfp4(*oracle.nvfp4_quantize_act(x, 1.0), to_np(i), to_np(v), triple(gate_up), triple(down))
        elif fmt == "fp8":
            pair = lambda q: (to_np(q.codes), to_np(q.scale))
            ref = oracle.moe_fp8(*oracle.fp8_quantize_act(x), to_np(i), to_np(v), pair(gate_up), pair(down))
        else:
            ref = oracle.moe_bf16(x, to_np(i), to_np(v), d["gate_up"], d["down"])
        assert rel_l2(to_np(o), ref) <= 1e-2          # the stated output tolerance
        assert max_abs(to_np(o), ref) <= 2.0 ** -5 * np.max(np.abs(f32(ref)))


# Batches of a few tokens, one after the other and between larger ones. The first launch of the experts reads the tokens and
# writes the shared expert's activations before it waits for the launch before it, while the call before may still read its
# own. With the norm, a call of as many tokens as the one before takes its normed result, as the layers of a decoder do.
FEW = (1, 3, 2, 2, 60, 1, 1, 200, 3, 3, 3, 1)


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("norm", [False, True])
@pytest.mark.parametrize("fmt", ["bf16", "nvfp4", "fp8"])
def test_few_tokens_without_synchronisation(oracle, fmt, norm, captured):
    from helpers import bf16
    from qs3_b200 import capi, ops
    shared_inter = 0 if fmt == "fp8" else I
    d = make_moe_inputs(62, 1, H, E, I, shared_inter)
    tokens = [make_moe_inputs(80 + n, t, H, 1, 1)["hidden"] for n, t in enumerate(FEW)]
    rng = np.random.default_rng(3)
    res = [bf16(rng.standard_normal((t, H), dtype=np.float32)) for t in FEW]
    weight = bf16(1 + 0.1 * rng.standard_normal(H, dtype=np.float32))
    q = {"nvfp4": ops.nvfp4_quantize_weight, "fp8": lambda c, w, gated: ops.fp8_quantize_weight(c, w),
         "bf16": lambda c, w, gated: w}[fmt]
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        ctx = ops.Context(torch.cuda.current_device(), stream.cuda_stream)
        gate_up, down, router = q(ctx, to_dev(d["gate_up"]), True), q(ctx, to_dev(d["down"]), False), to_dev(d["router"])
        shared = None
        if shared_inter:
            sgu, sdn = q(ctx, to_dev(d["sh_gate_up"]), True), q(ctx, to_dev(d["sh_down"]), False)
            shared = ops.SharedExpert(sgu, sdn, to_dev(d["sh_gate"]), shared_inter)
        plan = ops.MoePlan(ctx, ops.MoePlanConfig(
            max_num_tokens=max(FEW), hidden_size=H, intermediate_size=I, num_experts=E, top_k=K,
            backend=dict(bf16=capi.MOE_BACKEND_STAGED_BF16, nvfp4=capi.MOE_BACKEND_NVFP4,
                         fp8=capi.MOE_BACKEND_FP8_BLOCKSCALE)[fmt], route_mode=capi.MOE_ROUTE_ROUTER_LOGITS))
        ws = torch.zeros(plan.layer_workspace_size(max(FEW), shared_inter), dtype=torch.uint8, device="cuda")
        new = lambda dt, n: [torch.empty((t, n), dtype=dt, device="cuda") for t in FEW]
        source, given, out, ids, w = [to_dev(x) for x in tokens], [to_dev(x) for x in res], new(torch.bfloat16, H), new(torch.int32, K), new(torch.float32, K)
        kept, left = [torch.empty_like(x) for x in given], to_dev(weight)
        follows = [norm and n > 0 and FEW[n] == FEW[n - 1] for n in range(len(FEW))]

        def calls():
            for r, g in zip(kept, given):
                r.copy_(g)
            for n in range(len(FEW)):
                more = dict(residual_inout=kept[n], next_norm_weight=left) if norm else {}
                ops.moe_layer_execute(plan, out[n - 1] if follows[n] else source[n], router, gate_up, down, out[n], ws,
                                      shared=shared, topk_ids=ids[n], topk_weights=w[n], **more)
        calls()
        if captured:
            stream.synchronize()
            for o in out:
                o.zero_()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream):
                calls()
            graph.replay()
            graph.replay()
        stream.synchronize()
    assert ctx.read_device_error() == 0
    triple = lambda q: (to_np(q.packed), to_np(q.scale_linear), to_np(q.global_scale))
    for n, x in enumerate(tokens):
        x = to_np(out[n - 1]) if follows[n] else x
        i, v = to_np(ids[n]), to_np(w[n])
        ref_ids, ref_w = oracle.router_topk(oracle.gemm_bf16(x, d["router"], "f32"), K, 0, True, 1.0)
        assert np.mean(i != ref_ids) <= 2e-3   # near ties of the last expert
        assert np.allclose(v, ref_w, atol=1e-3)
        if fmt == "nvfp4":
            ref = oracle.moe_nvfp4(*oracle.nvfp4_quantize_act(x, 1.0), i, v, triple(gate_up), triple(down),
                                   shared=dict(gu=triple(sgu), d=triple(sdn), gate_w=d["sh_gate"]), hidden_bf16=x)
        elif fmt == "fp8":
            pair = lambda q: (to_np(q.codes), to_np(q.scale))
            ref = oracle.moe_fp8(*oracle.fp8_quantize_act(x), i, v, pair(gate_up), pair(down))
        else:
            ref = oracle.shared_expert_bf16(x, d["sh_gate_up"], d["sh_down"], d["sh_gate"],
                                            oracle.moe_bf16(x, i, v, d["gate_up"], d["down"]))
        got = to_np(out[n])
        if norm:
            # the residual is the sum of the layer's result, within the stated tolerance of it, and the one given; the
            # norm of that sum is rounded to bf16 once, like the sum itself
            layer = f32(to_np(kept[n])).astype(np.float64) - f32(res[n])
            rounding = 2.0 ** -8 * np.abs(f32(to_np(kept[n])))
            assert np.all(np.abs(layer - f32(ref)) <= rounding + 2.0 ** -5 * np.max(np.abs(f32(ref))))
            total = f32(to_np(kept[n])).astype(np.float64)
            want = total / np.sqrt(np.mean(total ** 2, axis=1, keepdims=True) + 1e-6) * f32(weight)
            assert np.all(np.abs(f32(got) - want) <= 2.0 ** -6 * np.abs(want) + 1e-3)
        else:
            assert rel_l2(got, ref) <= 1e-2          # the stated output tolerance
            assert max_abs(got, ref) <= 2.0 ** -5 * np.max(np.abs(f32(ref)))
