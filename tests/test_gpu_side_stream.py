"""The shared expert on the context's side stream: contexts that take turns on one plan without a synchronisation, and a
context whose first call is captured."""
from types import SimpleNamespace

import pytest
import torch

from helpers import f32, make_moe_inputs, max_abs, rel_l2, to_dev, to_np

pytestmark = pytest.mark.gpu

T, H, E, K, I = 150, 512, 16, 2, 256


@pytest.mark.parametrize("fmt", ["bf16", "nvfp4"])
def test_contexts_in_turn_and_first_call_captured(oracle, fmt):
    from qs3_b200 import capi, ops
    d = make_moe_inputs(3, 1, H, E, I, I)
    made = ops.Context()
    q = (lambda w, gated: ops.nvfp4_quantize_weight(made, w, gated)) if fmt == "nvfp4" else (lambda w, gated: w)
    w = {n: q(to_dev(d[n]), "gate" in n) for n in ("gate_up", "down", "sh_gate_up", "sh_down")}
    shared = ops.SharedExpert(w["sh_gate_up"], w["sh_down"], to_dev(d["sh_gate"]), I)
    router = to_dev(d["router"])
    plan = ops.MoePlan(made, ops.MoePlanConfig(
        max_num_tokens=T, hidden_size=H, intermediate_size=I, num_experts=E, top_k=K,
        backend=capi.MOE_BACKEND_NVFP4 if fmt == "nvfp4" else capi.MOE_BACKEND_STAGED_BF16))
    calls = []
    for n in range(3):
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            p = SimpleNamespace(handle=plan.handle, desc=plan.desc, ctx=ops.Context(torch.cuda.current_device(), stream.cuda_stream))
            x = make_moe_inputs(10 + n, T, H, 1, 1)["hidden"]
            calls.append(dict(stream=stream, plan=p, x=x, hidden=to_dev(x), out=torch.zeros((T, H), dtype=torch.bfloat16, device="cuda"),
                              ws=torch.zeros(plan.layer_workspace_size(T, I), dtype=torch.uint8, device="cuda"),
                              ids=torch.empty((T, K), dtype=torch.int32, device="cuda"),
                              w=torch.empty((T, K), dtype=torch.float32, device="cuda")))
    torch.cuda.synchronize()

    def call(c):
        ops.moe_layer_execute(c["plan"], c["hidden"], router, w["gate_up"], w["down"], c["out"], c["ws"], shared=shared,
                              topk_ids=c["ids"], topk_weights=c["w"])
    for _ in range(4):
        for c in calls[:2]:
            call(c)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=calls[2]["stream"]):
        call(calls[2])
    graph.replay()
    torch.cuda.synchronize()
    assert made.read_device_error() == 0
    triple = lambda v: (to_np(v.packed), to_np(v.scale_linear), to_np(v.global_scale))
    for c in calls:
        ids, wts = to_np(c["ids"]), to_np(c["w"])
        if fmt == "nvfp4":
            ref = oracle.moe_nvfp4(*oracle.nvfp4_quantize_act(c["x"], 1.0), ids, wts, triple(w["gate_up"]), triple(w["down"]),
                                   shared=dict(gu=triple(w["sh_gate_up"]), d=triple(w["sh_down"]), gate_w=d["sh_gate"]),
                                   hidden_bf16=c["x"])
        else:
            ref = oracle.shared_expert_bf16(c["x"], d["sh_gate_up"], d["sh_down"], d["sh_gate"],
                                            oracle.moe_bf16(c["x"], ids, wts, d["gate_up"], d["down"]))
        assert rel_l2(to_np(c["out"]), ref) <= 1e-2          # the stated output tolerance
        assert max_abs(to_np(c["out"]), ref) <= 2.0 ** -5 * abs(f32(ref)).max()
