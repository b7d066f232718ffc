"""The shared expert on the context's side stream: contexts that take turns on one plan without a synchronisation, a
context whose first call is captured, several streams of one context, and side streams that outlive their context."""
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


class _Calls:
    """bf16 layer calls with a shared expert beside the router chain, each on a workspace and result of its own."""

    def __init__(self):
        from qs3_b200 import capi, ops
        self.ops = ops
        d = make_moe_inputs(4, T, H, E, I, I)
        self.w = {n: to_dev(d[n]) for n in ("gate_up", "down", "router", "hidden")}
        self.shared = ops.SharedExpert(to_dev(d["sh_gate_up"]), to_dev(d["sh_down"]), to_dev(d["sh_gate"]), I)
        self.made = ops.Context()
        self.plans = [ops.MoePlan(self.made, ops.MoePlanConfig(
            max_num_tokens=T, hidden_size=H, intermediate_size=I, num_experts=E, top_k=K,
            backend=capi.MOE_BACKEND_STAGED_BF16)) for _ in range(2)]
        self.want = self.slot(self.made)
        self(self.want)
        torch.cuda.synchronize()
        assert float(self.want["out"].float().norm()) > 0

    def slot(self, ctx, plan=0):
        plan = self.plans[plan]
        return dict(plan=SimpleNamespace(handle=plan.handle, desc=plan.desc, ctx=ctx),
                    out=torch.zeros((T, H), dtype=torch.bfloat16, device="cuda"),
                    ws=torch.zeros(plan.layer_workspace_size(T, I), dtype=torch.uint8, device="cuda"))

    def __call__(self, slot):
        w = self.w
        self.ops.moe_layer_execute(slot["plan"], w["hidden"], w["router"], w["gate_up"], w["down"], slot["out"], slot["ws"],
                                   shared=self.shared)

    def check(self, *slots):
        torch.cuda.synchronize()
        assert self.made.read_device_error() == 0
        for s in slots:
            assert torch.equal(s["out"], self.want["out"])


SLEEP = 400_000_000     # clock cycles, about 0.2 s: far longer than a layer call takes


def _asleep(stream):
    """`stream` sleeps; the event is behind that."""
    with torch.cuda.stream(stream):
        torch.cuda._sleep(SLEEP)
        return stream.record_event()


def test_streams_of_one_context_do_not_wait_for_each_other():
    calls, (a, b) = _Calls(), (torch.cuda.Stream(), torch.cuda.Stream())
    ctx = calls.ops.Context(torch.cuda.current_device(), a.cuda_stream)
    one, two = calls.slot(ctx), calls.slot(ctx, plan=1)
    for stream, slot in ((a, one), (b, two)):   # (first calls make the side streams)
        ctx.set_stream(stream.cuda_stream)
        calls(slot)
    torch.cuda.synchronize()
    awake = _asleep(a)
    ctx.set_stream(a.cuda_stream)
    calls(one)
    ctx.set_stream(b.cuda_stream)
    calls(two)
    b.synchronize()
    assert not awake.query()
    calls.check(one, two)


def test_call_beside_an_open_capture():
    """A capture that is open on one stream of a context leaves its calls on another stream alone."""
    calls, (a, b) = _Calls(), (torch.cuda.Stream(), torch.cuda.Stream())
    ctx = calls.ops.Context(torch.cuda.current_device(), a.cuda_stream)
    one, two = calls.slot(ctx), calls.slot(ctx, plan=1)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=a):
        calls(one)
        ctx.set_stream(b.cuda_stream)
        calls(two)
        ctx.set_stream(a.cuda_stream)
    graph.replay()
    calls.check(one, two)


def test_more_streams_than_a_context_keeps():
    calls = _Calls()
    ctx = calls.ops.Context(torch.cuda.current_device())
    slots = []
    for n in range(12):
        stream = torch.cuda.Stream()
        ctx.set_stream(stream.cuda_stream)
        slots.append((stream, calls.slot(ctx, n % 2)))
        torch.cuda.synchronize()
        for _ in range(3):
            calls(slots[-1][1])
    calls.check(*(s for _, s in slots))


@pytest.mark.parametrize("captured", [False, True])
def test_side_stream_of_a_destroyed_context(captured):
    """A context destroyed with work outstanding does not hold up the ones that follow."""
    calls, (a, b) = _Calls(), (torch.cuda.Stream(), torch.cuda.Stream())
    first = calls.ops.Context(torch.cuda.current_device(), a.cuda_stream)
    one, two = calls.slot(first), calls.slot(None)
    # no other side stream is free: more contexts than streams are kept hold one each
    held = [calls.slot(calls.ops.Context()) for _ in range(9)]
    for s in held:
        calls(s)
    torch.cuda.synchronize()
    calls(one)
    torch.cuda.synchronize()
    awake = _asleep(a)
    calls(one)
    first.close()
    two["plan"].ctx = calls.ops.Context(torch.cuda.current_device(), b.cuda_stream)
    with torch.cuda.stream(b):
        if captured:
            graph = torch.cuda.CUDAGraph()
            graph.capture_begin()
            calls(two)
            graph.capture_end()
            graph.replay()
        else:
            calls(two)
    b.synchronize()
    assert not awake.query()
    calls.check(one, two, *held)


def test_side_stream_is_made_under_capture():
    """The first forked call of a context is captured while no side stream is left over."""
    calls, b = _Calls(), torch.cuda.Stream()
    held = [calls.slot(calls.ops.Context()) for _ in range(9)]
    for s in held:
        calls(s)
    new = calls.slot(calls.ops.Context(torch.cuda.current_device(), b.cuda_stream))
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=b):
        calls(new)
    graph.replay()
    graph.replay()
    calls.check(new, *held)
