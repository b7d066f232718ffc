"""Layer calls of a handful of tokens, whose experts run as matrix-vector products (csrc/gemv.cu): against the CPU oracle in
every format, at the smallest and largest shapes of the kernels, with every option that they take over from the launches
they replace. Tolerances are the ones that the other layer tests state for these formats."""
import numpy as np
import pytest
import torch

from helpers import bf16, f32, make_moe_inputs, max_abs, rel_l2, to_dev, to_np

pytestmark = pytest.mark.gpu

CASES = [
    # fmt, tokens, hidden, inter, experts, top-k, shared, local experts
    ("nvfp4", 1, 256, 256, 8, 2, True, None),        # two steps of k for eight parts of it
    ("nvfp4", 3, 512, 256, 40, 10, True, None),
    ("nvfp4", 1, 2048, 512, 64, 10, False, None),
    ("nvfp4", 2, 1024, 512, 300, 16, True, (100, 150)),
    ("fp8", 1, 128, 128, 8, 2, False, None),         # one k block in both products
    ("fp8", 5, 384, 640, 8, 2, False, (2, 5)),
    ("fp8", 1, 4096, 384, 16, 4, False, None),
    ("bf16", 1, 128, 32, 4, 1, True, None),          # one block of features, fewer chunks than lanes
    ("bf16", 16, 256, 128, 8, 2, False, None),       # as many tokens as a routing block has warps
    ("bf16", 3, 640, 96, 512, 16, True, (0, 256)),
    ("bf16", 1, 4096, 96, 16, 3, True, None),
]


def _run(fmt, t, h, i, e, k, shared, local, **more):
    from qs3_b200 import capi, ops
    off, le = local or (0, e)
    d = make_moe_inputs(90 + t + k, t, h, e, i, i if shared else 0)
    d["gate_up"], d["down"] = d["gate_up"][off:off + le], d["down"][off:off + le]
    ctx = ops.Context()
    q = {"nvfp4": ops.nvfp4_quantize_weight, "fp8": lambda c, w, gated: ops.fp8_quantize_weight(c, w),
         "bf16": lambda c, w, gated: w}[fmt]
    gu, dn = q(ctx, to_dev(d["gate_up"]), True), q(ctx, to_dev(d["down"]), False)
    sh = None
    if shared:
        sgu, sdn = q(ctx, to_dev(d["sh_gate_up"]), True), q(ctx, to_dev(d["sh_down"]), False)
        sh = ops.SharedExpert(sgu, sdn, to_dev(d["sh_gate"]), i)
    plan = ops.MoePlan(ctx, ops.MoePlanConfig(
        max_num_tokens=t, hidden_size=h, intermediate_size=i, num_experts=e, top_k=k, local_expert_offset=off,
        local_num_experts=le, backend=dict(bf16=capi.MOE_BACKEND_STAGED_BF16, nvfp4=capi.MOE_BACKEND_NVFP4,
                                           fp8=capi.MOE_BACKEND_FP8_BLOCKSCALE)[fmt]))
    ws = torch.full((plan.layer_workspace_size(t, i if shared else 0),), 0xff, dtype=torch.uint8, device="cuda")
    hidden = to_dev(d["hidden"])
    out = torch.empty_like(hidden)
    ids = torch.empty((t, k), dtype=torch.int32, device="cuda")
    w = torch.empty((t, k), dtype=torch.float32, device="cuda")
    logits = torch.empty((t, e), dtype=torch.float32, device="cuda")
    if more.pop("prequantised", False):
        x, r = hidden.clone(), torch.zeros_like(hidden)
        more["hidden_packed"] = torch.empty((t, h // 2), dtype=torch.uint8, device="cuda")
        more["hidden_scale_tiled"] = torch.zeros(ops.nvfp4_tiled_scale_bytes(t, h), dtype=torch.uint8, device="cuda")
        ops.fused_add_rmsnorm_nvfp4(ctx, x, r, torch.ones(h, dtype=torch.bfloat16, device="cuda"),
                                    packed=more["hidden_packed"], tiled=more["hidden_scale_tiled"])
        hidden.copy_(x)
        d["hidden"] = to_np(x)
    bias = more.pop("bias", None)
    before = ops.launch_count()
    ops.moe_layer_execute(plan, hidden, to_dev(d["router"]), gu, dn, out, ws, router_bias=None if bias is None else to_dev(bias),
                          shared=sh, topk_ids=ids, topk_weights=w, router_logits=logits, **more)
    launches = ops.launch_count() - before
    torch.cuda.synchronize()
    assert ctx.read_device_error() == 0
    return dict(d=d, plan=plan, ws=ws, out=to_np(out), ids=to_np(ids), w=to_np(w), logits=to_np(logits), gu=gu, dn=dn,
                sh=sh, launches=launches, off=off, le=le, bias=bias, k=k)


def _reference(oracle, fmt, r, score=0):
    d = r["d"]
    ids, w = oracle.router_topk(r["logits"], r["k"], score, True, 1.0, bias=r["bias"])
    assert np.array_equal(r["ids"], ids)
    assert np.allclose(r["w"], w, rtol=1e-5, atol=1e-7)
    w = r["w"]
    triple = lambda q: (to_np(q.packed), to_np(q.scale_linear), to_np(q.global_scale))
    if fmt == "nvfp4":
        shared = None if r["sh"] is None else dict(gu=triple(r["sh"].gate_up), d=triple(r["sh"].down), gate_w=d["sh_gate"])
        return oracle.moe_nvfp4(*oracle.nvfp4_quantize_act(d["hidden"], 1.0), ids, w, triple(r["gu"]), triple(r["dn"]),
                                local_offset=r["off"], shared=shared, hidden_bf16=d["hidden"])
    if fmt == "fp8":
        pair = lambda q: (to_np(q.codes), to_np(q.scale))
        return oracle.moe_fp8(*oracle.fp8_quantize_act(d["hidden"]), ids, w, pair(r["gu"]), pair(r["dn"]), local_offset=r["off"])
    ref = oracle.moe_bf16(d["hidden"], ids, w, d["gate_up"], d["down"], r["off"])
    return ref if r["sh"] is None else oracle.shared_expert_bf16(d["hidden"], d["sh_gate_up"], d["sh_down"], d["sh_gate"], ref)


def _check(out, ref):
    assert rel_l2(out, ref) <= 1e-2
    assert max_abs(out, ref) <= 2.0 ** -5 * np.max(np.abs(f32(ref)))


@pytest.mark.parametrize("case", CASES, ids=lambda c: "-".join(map(str, c)))
def test_layer_of_few_tokens(oracle, case):
    r = _run(*case)
    assert r["launches"] == 3  # logits, gate_up, down
    _check(r["out"], _reference(oracle, case[0], r))
    # the tables are those of the sort that the other paths run
    for got, ref in zip(r["plan"].routing_tables(r["ws"], case[1]), oracle.route_sort(r["ids"], r["w"], r["off"], r["le"])):
        assert np.array_equal(to_np(got), ref)


@pytest.mark.parametrize("fmt,shared", [("nvfp4", True), ("fp8", False), ("bf16", True)])
def test_options(oracle, fmt, shared):
    """Sigmoid scores with a bias; the post-layer residual and norm, which take the slots' rows from the down launch."""
    t, h, i, e, k = 3, 512, 256, 24, 4
    bias = (np.arange(e, dtype=np.float32) % 7 - 3) * 0.25
    r = _run(fmt, t, h, i, e, k, shared, None, score=1, bias=bias)
    _check(r["out"], _reference(oracle, fmt, r, score=1))
    rng = np.random.default_rng(5)
    res, weight = bf16(rng.standard_normal((t, h), dtype=np.float32)), bf16(1 + 0.1 * rng.standard_normal(h, dtype=np.float32))
    res_t = to_dev(res)
    n = _run(fmt, t, h, i, e, k, shared, None, residual_inout=res_t, next_norm_weight=to_dev(weight))
    plain = _run(fmt, t, h, i, e, k, shared, None)
    norm, res_ref = oracle.fused_add_rmsnorm(plain["out"], res, weight)
    assert np.array_equal(to_np(res_t), bf16(res_ref))
    assert np.max(np.abs(f32(n["out"]) - norm)) <= 2.0 ** -8 * np.max(np.abs(norm)) + 1e-6  # one rounding to bf16


def test_prequantised_tokens(oracle):
    r = _run("nvfp4", 2, 512, 256, 16, 4, True, None, prequantised=True)
    _check(r["out"], _reference(oracle, "nvfp4", r))


def test_given_routes(oracle):
    """The drop-in call: ids and weights from the caller, among them one expert twice, and routes of other ranks."""
    from qs3_b200 import capi, ops
    t, h, i, e, k, off, le = 2, 256, 64, 1024, 4, 8, 1000
    d = make_moe_inputs(7, t, h, le, i)
    ids = np.array([[8, 8, 1007, 3], [1020, 500, 9, 0]], np.int32)
    w = np.array([[0.5, 0.25, 0.125, 9.0], [9.0, 0.75, 0.5, 9.0]], np.float32)
    ctx = ops.Context()
    plan = ops.MoePlan(ctx, ops.MoePlanConfig(max_num_tokens=t, hidden_size=h, intermediate_size=i, num_experts=e, top_k=k,
                                              local_expert_offset=off, local_num_experts=le,
                                              backend=capi.MOE_BACKEND_STAGED_BF16))
    ws = torch.zeros(plan.workspace_size(t), dtype=torch.uint8, device="cuda")
    out = torch.empty((t, h), dtype=torch.bfloat16, device="cuda")
    before = ops.launch_count()
    ops.moe_execute_bf16(plan, to_dev(d["hidden"]), to_dev(ids), to_dev(w), to_dev(d["gate_up"]), to_dev(d["down"]), out, ws)
    assert ops.launch_count() - before == 2
    torch.cuda.synchronize()
    _check(to_np(out), oracle.moe_bf16(d["hidden"], ids, w, d["gate_up"], d["down"], off))


def test_result_in_the_tokens_place(oracle):
    """Every token's gate is read by many blocks: not while others write the result over the tokens."""
    from qs3_b200 import capi, ops
    t, h, i, e, k = 2, 512, 128, 8, 2
    d = make_moe_inputs(11, t, h, e, i, i)
    ctx = ops.Context()
    plan = ops.MoePlan(ctx, ops.MoePlanConfig(max_num_tokens=t, hidden_size=h, intermediate_size=i, num_experts=e, top_k=k,
                                              backend=capi.MOE_BACKEND_STAGED_BF16))
    ws = torch.zeros(plan.layer_workspace_size(t, i), dtype=torch.uint8, device="cuda")
    x, ids, w = to_dev(d["hidden"]), torch.empty((t, k), dtype=torch.int32, device="cuda"), torch.empty((t, k), dtype=torch.float32, device="cuda")
    before = ops.launch_count()
    ops.moe_layer_execute(plan, x, to_dev(d["router"]), to_dev(d["gate_up"]), to_dev(d["down"]), x, ws,
                          shared=ops.SharedExpert(to_dev(d["sh_gate_up"]), to_dev(d["sh_down"]), to_dev(d["sh_gate"]), i),
                          topk_ids=ids, topk_weights=w)
    assert ops.launch_count() - before > 3
    torch.cuda.synchronize()
    ref = oracle.moe_bf16(d["hidden"], to_np(ids), to_np(w), d["gate_up"], d["down"])
    _check(to_np(x), oracle.shared_expert_bf16(d["hidden"], d["sh_gate_up"], d["sh_down"], d["sh_gate"], ref))


@pytest.mark.parametrize("h,i,refused", [(4096, 128, False), (4224, 128, True), (128, 4096, False), (128, 4224, True)])
def test_fp8_refusals_do_not_depend_on_the_batch(oracle, h, i, refused):
    from qs3_b200 import capi, ops
    case = ("fp8", 1, h, i, 2, 1, False, None)
    if not refused:
        r = _run(*case)
        return _check(r["out"], _reference(oracle, "fp8", r))
    with pytest.raises(ops.Qs3Error) as error:
        _run(*case)
    assert error.value.status == capi.STATUS_UNSUPPORTED


@pytest.mark.parametrize("fmt,shared", [("nvfp4", True), ("fp8", False), ("bf16", True), ("bf16", False)])
def test_profile_has_the_stages_apart(oracle, fmt, shared):
    """A profiled call of a handful of tokens takes the stages one by one, with the same result."""
    from qs3_b200 import ops
    ctx = ops.Context()
    case = (fmt, 2, 512, 256, 24, 4, shared, None)
    ops.profile_begin(ctx)
    r = _run(*case)
    stages = ops.profile_end(ctx)
    _check(r["out"], _reference(oracle, fmt, r))
    names = [name for name, _ in stages]
    # (a shared expert of the experts' size joins the NVFP4 GEMMs)
    want = ["router_logits_gemm", "router_topk", "route_sort", "gather_quantize", "gate_up_gemm_swiglu", "down_gemm",
            "shared_expert", "combine"]
    assert names == [n for n in want if n != "shared_expert" or (shared and fmt == "bf16")]
    # the sort is in the top-k's launch; bf16 rows of small tiles are read in place, NVFP4 tokens quantised beside the sort
    empty = {"route_sort"} | ({"gather_quantize"} if fmt != "fp8" else set())
    assert all(ms > 1e-3 for name, ms in stages if name not in empty)
    assert r["launches"] > 3


# (12, 8 and 16 tokens: 36.7, 54.9 and 34.0 us as matrix-vector products, 23.6, 37.9 and 25.7 grouped)
@pytest.mark.parametrize("case", [("fp8", 12, 256, 1024, 128, 8, False, None), ("bf16", 8, 2048, 256, 512, 10, False, (0, 64)),
                                  ("nvfp4", 16, 512, 768, 128, 4, False, None)], ids=lambda c: "-".join(map(str, c)))
def test_many_slots_stay_with_the_grouped_gemms(oracle, case):
    r = _run(*case)
    assert r["launches"] > 3
    _check(r["out"], _reference(oracle, case[0], r))
