"""GPU parity of the NVFP4 path: quantisers and scale layouts bit-exact against the
CPU oracle, routed experts and the whole layer within the stated output tolerance.
Upstream has no NVFP4 arithmetic, so these outputs are pinned to the oracle only."""
import numpy as np
import pytest
import torch

from helpers import bf16, f32, make_moe_inputs, max_abs, rel_l2, tile_height, to_dev, to_np, zipf_bias

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from qs3_b200 import ops as m
    return m


@pytest.fixture(scope="module")
def ctx(ops):
    return ops.Context()


def test_activation_quantiser_is_bit_exact(ops, ctx, oracle):
    rng = np.random.default_rng(21)
    x = rng.standard_normal((37, 256), dtype=np.float32)
    x[0, :16] = 0.0                       # all-zero block -> scale 0, codes 0
    x[1, :16] = [0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0, 6.0, -0.25, -0.75, -1.25, -1.75, -2.5, -3.5, -5.0, -6.0]
    x[2] *= 1e-4                          # tiny values: sub-normal block scales
    x[3] *= 300.0
    xb = bf16(x)
    for g in (1.0, 0.37):
        packed, scale = ops.nvfp4_quantize_act(ctx, to_dev(xb), g)
        p_ref, s_ref = oracle.nvfp4_quantize_act(xb, g)
        assert np.array_equal(to_np(scale), s_ref)
        assert np.array_equal(to_np(packed), p_ref)


@pytest.mark.parametrize("gated", [False, True])
def test_weight_quantiser_and_scale_tiling_are_bit_exact(ops, ctx, oracle, gated):
    rng = np.random.default_rng(22)
    e, rows, k = 3, 256, 512
    w = bf16(rng.standard_normal((e, rows, k), dtype=np.float32) * 0.02)
    w[1] = 0  # all-zero expert: global scale 1
    q = ops.nvfp4_quantize_weight(ctx, to_dev(w), gated)
    p_ref, s_ref, st_ref, g_ref = oracle.nvfp4_quantize_weight(w, gated)
    assert np.array_equal(to_np(q.global_scale), g_ref)
    assert np.array_equal(to_np(q.scale_linear), s_ref)
    assert np.array_equal(to_np(q.packed), p_ref)
    assert np.array_equal(to_np(q.scale_tiled), st_ref)
    # re-tiling the declared (linear) layout gives the same tiled buffer
    assert np.array_equal(to_np(ops.nvfp4_tile_scales(ctx, q.scale_linear, gated)), st_ref)


# one block, a k that is no multiple of the 512-element unit, a last row block that is not full, more experts
# than clusters run at a time; many experts so small that most blocks of a cluster have nothing to read before they
# exchange their maxima; few experts large enough for the whole grid each, a k tail and a row tail among them
@pytest.mark.parametrize("e,rows,k,gated", [(1, 128, 64, True), (2, 384, 576, True), (3, 200, 832, False),
                                            (40, 128, 1024, False), (600, 128, 64, True), (2, 2048, 1088, True),
                                            (1, 2056, 1024, False)])
def test_weight_quantiser_edges(ops, ctx, oracle, e, rows, k, gated):
    rng = np.random.default_rng(rows + k)
    w = bf16(rng.standard_normal((e, rows, k), dtype=np.float32) * 0.02)
    w[-1, -1, -1] = 3.0  # the expert's amax sits in its last element
    q = ops.nvfp4_quantize_weight(ctx, to_dev(w), gated)
    for got, ref in zip((q.packed, q.scale_linear, q.scale_tiled, q.global_scale),
                        oracle.nvfp4_quantize_weight(w, gated)):
        assert np.array_equal(to_np(got), ref)


def _check(out, ref):
    assert rel_l2(out, ref) <= 1e-2
    assert max_abs(out, ref) <= 2.0 ** -5 * np.max(np.abs(f32(ref)))


def _quantise_all(ops, ctx, d, shared):
    gu = ops.nvfp4_quantize_weight(ctx, to_dev(d["gate_up"]), True)
    dn = ops.nvfp4_quantize_weight(ctx, to_dev(d["down"]), False)
    sh = None
    if shared:
        sh = (ops.nvfp4_quantize_weight(ctx, to_dev(d["sh_gate_up"]), True),
              ops.nvfp4_quantize_weight(ctx, to_dev(d["sh_down"]), False))
    return gu, dn, sh


def _hot_bias(e):
    """Router bias that sends a route of every token to expert 3."""
    return np.where(np.arange(e) == 3, 10.0, 0.0).astype(np.float32)


def _triple(q):
    return to_np(q.packed), to_np(q.scale_linear), to_np(q.global_scale)


@pytest.mark.parametrize("cfg", [
    dict(t=64, h=256, e=8, k=2, i=256),
    dict(t=200, h=512, e=16, k=4, i=256, local=(4, 8)),
])
def test_declared_abi_execute_matches_oracle(ops, ctx, oracle, cfg):
    """qsfi_moe_execute_nvfp4 with the declared (pre-quantised, linear-scale) layout."""
    t, h, e, k, i = cfg["t"], cfg["h"], cfg["e"], cfg["k"], cfg["i"]
    off, le = cfg.get("local", (0, e))
    d = make_moe_inputs(31, t, h, e, i)
    d["gate_up"], d["down"] = d["gate_up"][off:off + le], d["down"][off:off + le]
    ids, w = oracle.router_topk(oracle.gemm_bf16(d["hidden"], d["router"], "f32"), k, 0, True, 1.0)
    # the declared ABI has no per-expert scale for the gate_up product, so its weights are
    # quantised against a global scale of 1 (weights scaled up so that block scales stay normal)
    gu_w = bf16(f32(d["gate_up"]) * 8.0)
    dn_w = bf16(f32(d["down"]) * 8.0)
    gup, gus = oracle.nvfp4_quantize_act(gu_w.reshape(-1, h), 1.0)
    dnp, dns = oracle.nvfp4_quantize_act(dn_w.reshape(-1, i), 1.0)
    gup, gus = gup.reshape(le, 2 * i, h // 2), gus.reshape(le, 2 * i, h // 16)
    dnp, dns = dnp.reshape(le, h, i // 2), dns.reshape(le, h, i // 16)
    out_scale = (0.5 + d["rng"].random(le)).astype(np.float32)
    hp, hs = ops.nvfp4_quantize_act(ctx, to_dev(d["hidden"]), 1.0)
    plan = ops.MoePlan(ctx, ops.MoePlanConfig(max_num_tokens=t, hidden_size=h, intermediate_size=i,
                                              num_experts=e, top_k=k, local_expert_offset=off,
                                              local_num_experts=le, backend=ops.capi.MOE_BACKEND_NVFP4))
    ws = torch.zeros(plan.workspace_size(t), dtype=torch.uint8, device="cuda")
    out = torch.empty((t, h), dtype=torch.bfloat16, device="cuda")
    ops.moe_execute_nvfp4(plan, hp, hs, to_dev(ids), to_dev(w), to_dev(gup), to_dev(gus), to_dev(dnp),
                          to_dev(dns), out, ws, expert_output_scale=to_dev(out_scale))
    torch.cuda.synchronize()
    assert ctx.read_device_error() == 0
    ones = np.ones(le, np.float32)
    ref = oracle.moe_nvfp4(to_np(hp), to_np(hs), ids, w, (gup, gus, ones), (dnp, dns, out_scale),
                           local_offset=off)
    _check(to_np(out), ref)


@pytest.mark.parametrize("cfg", [
    dict(t=64, h=256, e=8, k=2, i=256, s=0),
    dict(t=300, h=512, e=32, k=4, i=256, s=256, bias=True),
    dict(t=128, h=2048, e=64, k=10, i=512, s=512, bias=True),   # layer shape of the prefill workload
])
def test_whole_layer_matches_oracle(ops, ctx, oracle, cfg):
    t, h, e, k, i, s = cfg["t"], cfg["h"], cfg["e"], cfg["k"], cfg["i"], cfg["s"]
    d = make_moe_inputs(33, t, h, e, i, s)
    bias = zipf_bias(e, d["rng"]) if cfg.get("bias") else None
    gu, dn, sh = _quantise_all(ops, ctx, d, bool(s))
    plan = ops.MoePlan(ctx, ops.MoePlanConfig(max_num_tokens=t, hidden_size=h, intermediate_size=i,
                                              num_experts=e, top_k=k, backend=ops.capi.MOE_BACKEND_NVFP4))
    ws = torch.zeros(plan.layer_workspace_size(t, s), dtype=torch.uint8, device="cuda")
    out = torch.empty((t, h), dtype=torch.bfloat16, device="cuda")
    ids_t = torch.empty((t, k), dtype=torch.int32, device="cuda")
    w_t = torch.empty((t, k), dtype=torch.float32, device="cuda")
    logits_t = torch.empty((t, e), dtype=torch.float32, device="cuda")
    shared = None
    if s:
        shared = ops.SharedExpert(sh[0], sh[1], to_dev(d["sh_gate"]), s)
    ops.moe_layer_execute(plan, to_dev(d["hidden"]), to_dev(d["router"]), gu, dn, out, ws,
                          router_bias=None if bias is None else to_dev(bias), shared=shared,
                          topk_ids=ids_t, topk_weights=w_t, router_logits=logits_t)
    torch.cuda.synchronize()
    assert ctx.read_device_error() == 0
    ids_ref, w_ref = oracle.router_topk(to_np(logits_t), k, 0, True, 1.0, bias)
    assert np.array_equal(to_np(ids_t), ids_ref)
    hp, hs = oracle.nvfp4_quantize_act(d["hidden"], 1.0)
    shared_ref = None
    if s:
        shared_ref = dict(gu=_triple(sh[0]), d=_triple(sh[1]), gate_w=d["sh_gate"])
    ref = oracle.moe_nvfp4(hp, hs, ids_ref, w_ref, _triple(gu), _triple(dn), shared=shared_ref,
                           hidden_bf16=d["hidden"])
    _check(to_np(out), ref)
    # and against the unquantised bf16 chain: NVFP4 is a lossy format, so only a loose bound
    full = oracle.moe_bf16(d["hidden"], ids_ref, w_ref, d["gate_up"], d["down"])
    if s:
        full = oracle.shared_expert_bf16(d["hidden"], d["sh_gate_up"], d["sh_down"], d["sh_gate"], full)
    assert rel_l2(to_np(out), full) <= 0.25


def test_layer_call_replays_from_a_cuda_graph(ops, oracle):
    """The whole-layer call (with its internal side-stream fork for the shared expert) captured
    once in a CUDA graph and replayed on fresh inputs gives the eager result bit for bit."""
    t, h, e, k, i, s = 256, 512, 32, 4, 256, 256
    d = make_moe_inputs(35, t, h, e, i, s)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        ctx = ops.Context()          # bound to this (non-default) stream
        gu, dn, sh = _quantise_all(ops, ctx, d, True)
        shared = ops.SharedExpert(sh[0], sh[1], to_dev(d["sh_gate"]), s)
        plan = ops.MoePlan(ctx, ops.MoePlanConfig(max_num_tokens=t, hidden_size=h, intermediate_size=i,
                                                  num_experts=e, top_k=k, backend=ops.capi.MOE_BACKEND_NVFP4))
        ws = torch.zeros(plan.layer_workspace_size(t, s), dtype=torch.uint8, device="cuda")
        x = to_dev(d["hidden"])
        router = to_dev(d["router"])
        out = torch.empty((t, h), dtype=torch.bfloat16, device="cuda")
        run = lambda: ops.moe_layer_execute(plan, x, router, gu, dn, out, ws, shared=shared)
        for _ in range(2):
            run()
        stream.synchronize()
        eager_first = to_np(out)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            run()
        # new tokens in the same buffer: the graph must recompute everything from them
        x.copy_(to_dev(bf16(f32(d["hidden"])[::-1].copy())))
        graph.replay()
        stream.synchronize()
        replayed = to_np(out)
        run()
        stream.synchronize()
        assert ctx.read_device_error() == 0
        assert np.array_equal(replayed, to_np(out))
        assert not np.array_equal(replayed, eager_first)


def test_gate_and_up_rows_with_separate_global_scales(ops, ctx, oracle):
    """Checkpoints that quantise gate_proj and up_proj apart carry one global scale for each;
    the layer takes them as f32 [2 * experts] (routed) and f32 [2] (shared expert)."""
    import dataclasses
    t, h, e, k, i, s = 96, 512, 16, 4, 256, 256
    d = make_moe_inputs(37, t, h, e, i, s)
    gu, dn, sh = _quantise_all(ops, ctx, d, True)
    factor = torch.linspace(0.6, 1.7, e, device="cuda")
    gu2 = dataclasses.replace(gu, global_scale=torch.cat([gu.global_scale, gu.global_scale * factor]))
    sgu2 = dataclasses.replace(sh[0], global_scale=torch.cat([sh[0].global_scale, sh[0].global_scale * 1.3]))
    plan = ops.MoePlan(ctx, ops.MoePlanConfig(max_num_tokens=t, hidden_size=h, intermediate_size=i,
                                              num_experts=e, top_k=k, backend=ops.capi.MOE_BACKEND_NVFP4))
    ws = torch.zeros(plan.layer_workspace_size(t, s), dtype=torch.uint8, device="cuda")
    out = torch.empty((t, h), dtype=torch.bfloat16, device="cuda")
    ids_t = torch.empty((t, k), dtype=torch.int32, device="cuda")
    w_t = torch.empty((t, k), dtype=torch.float32, device="cuda")
    shared = ops.SharedExpert(sgu2, sh[1], to_dev(d["sh_gate"]), s)
    ops.moe_layer_execute(plan, to_dev(d["hidden"]), to_dev(d["router"]), gu2, dn, out, ws, shared=shared,
                          topk_ids=ids_t, topk_weights=w_t)
    torch.cuda.synchronize()
    assert ctx.read_device_error() == 0
    hp, hs = oracle.nvfp4_quantize_act(d["hidden"], 1.0)
    ref = oracle.moe_nvfp4(hp, hs, to_np(ids_t), to_np(w_t), _triple(gu2), _triple(dn),
                           shared=dict(gu=_triple(sgu2), d=_triple(sh[1]), gate_w=d["sh_gate"]),
                           hidden_bf16=d["hidden"])
    _check(to_np(out), ref)
    # the second scale is really applied: the single-scale result differs
    single = oracle.moe_nvfp4(hp, hs, to_np(ids_t), to_np(w_t), _triple(gu), _triple(dn),
                              shared=dict(gu=_triple(sh[0]), d=_triple(sh[1]), gate_w=d["sh_gate"]),
                              hidden_bf16=d["hidden"])
    assert rel_l2(to_np(out), single) > 0.05


@pytest.mark.parametrize("cfg", [
    dict(t=16, h=512, e=64, k=4, i=256, s=256, rows=32),        # a few rows per expert, most experts empty
    dict(t=100, h=2048, e=128, k=10, i=512, s=512, bias=True, rows=32),  # decode batch of the prefill layer's shape
    dict(t=128, h=2048, e=128, k=10, i=512, s=512, bias=True, rows=64),
    dict(t=40, h=256, e=16, k=2, i=256, s=0, hot=True, rows=32),         # an expert with 40 rows: two tiles
    dict(t=40, h=256, e=4, k=2, i=256, s=0, rows=64),
])
def test_decode_batches_take_the_swapped_operand_kernel(ops, ctx, oracle, cfg):
    """Up to 8 routes per expert on average the plan pads expert segments to 32 rows, up to 22 to 64, and the grouped GEMMs
    run with the weights as the M side of the MMA (a shared expert joins them with 32-row tiles); same results as the
    oracle."""
    t, h, e, k, i, s = cfg["t"], cfg["h"], cfg["e"], cfg["k"], cfg["i"], cfg["s"]
    d = make_moe_inputs(41, t, h, e, i, s)
    bias = zipf_bias(e, d["rng"]) if cfg.get("bias") else _hot_bias(e) if cfg.get("hot") else None
    gu, dn, sh = _quantise_all(ops, ctx, d, bool(s))
    plan = ops.MoePlan(ctx, ops.MoePlanConfig(max_num_tokens=t, hidden_size=h, intermediate_size=i,
                                              num_experts=e, top_k=k, backend=ops.capi.MOE_BACKEND_NVFP4))
    ws = torch.zeros(plan.layer_workspace_size(t, s), dtype=torch.uint8, device="cuda")
    out = torch.empty((t, h), dtype=torch.bfloat16, device="cuda")
    ids_t = torch.empty((t, k), dtype=torch.int32, device="cuda")
    w_t = torch.empty((t, k), dtype=torch.float32, device="cuda")
    shared = ops.SharedExpert(sh[0], sh[1], to_dev(d["sh_gate"]), s) if s else None
    ops.moe_layer_execute(plan, to_dev(d["hidden"]), to_dev(d["router"]), gu, dn, out, ws,
                          router_bias=None if bias is None else to_dev(bias), shared=shared,
                          act_global_scale=0.5, act2_global_scale=0.25, topk_ids=ids_t, topk_weights=w_t)
    torch.cuda.synchronize()
    assert ctx.read_device_error() == 0
    assert tile_height(plan, ws, t) == cfg["rows"]
    hp, hs = oracle.nvfp4_quantize_act(d["hidden"], 0.5)
    shared_ref = dict(gu=_triple(sh[0]), d=_triple(sh[1]), gate_w=d["sh_gate"]) if s else None
    ref = oracle.moe_nvfp4(hp, hs, to_np(ids_t), to_np(w_t), _triple(gu), _triple(dn), act_global=0.5,
                           act2_global=0.25, shared=shared_ref, hidden_bf16=d["hidden"])
    _check(to_np(out), ref)


# panels whose rows do not divide the loaders' vectors (three and five blocks of 256 elements), tiles of one row to all,
# rows beside multiples of four, an expert of several tiles
@pytest.mark.parametrize("t,e,k,h,i,hot,rows", [(37, 16, 2, 768, 256, False, 32), (67, 16, 2, 1280, 768, True, 64),
                                                (100, 32, 6, 1280, 256, False, 64), (5, 64, 5, 768, 256, False, 32)])
def test_small_tile_panels(ops, ctx, oracle, t, e, k, h, i, hot, rows):
    d = make_moe_inputs(71, t, h, e, i)
    gu, dn, _ = _quantise_all(ops, ctx, d, False)
    plan = ops.MoePlan(ctx, ops.MoePlanConfig(max_num_tokens=t, hidden_size=h, intermediate_size=i, num_experts=e, top_k=k,
                                              backend=ops.capi.MOE_BACKEND_NVFP4))
    ws = torch.zeros(plan.layer_workspace_size(t, 0), dtype=torch.uint8, device="cuda")
    ids = torch.empty((t, k), dtype=torch.int32, device="cuda")
    w = torch.empty((t, k), dtype=torch.float32, device="cuda")
    out = torch.empty((t, h), dtype=torch.bfloat16, device="cuda")
    ops.moe_layer_execute(plan, to_dev(d["hidden"]), to_dev(d["router"]), gu, dn, out, ws, topk_ids=ids, topk_weights=w,
                          router_bias=to_dev(_hot_bias(e)) if hot else None)
    torch.cuda.synchronize()
    assert ctx.read_device_error() == 0
    assert tile_height(plan, ws, t) == rows
    hp, hs = oracle.nvfp4_quantize_act(d["hidden"], 1.0)
    _check(to_np(out), oracle.moe_nvfp4(hp, hs, to_np(ids), to_np(w), _triple(gu), _triple(dn)))


# several feature blocks per CTA, so that both MMA issuers of the kernel work: a k of more blocks than the ring has stages
# (2048 with 64-row tiles: eight over seven), of as many, and one of a single block
@pytest.mark.parametrize("t,e,k,h,i,rows", [(100, 64, 8, 2048, 512, 64), (60, 64, 8, 2048, 512, 32),
                                            (300, 128, 6, 256, 256, 64)])
def test_swapped_operand_kernel_repeats(ops, ctx, oracle, t, e, k, h, i, rows):
    d = make_moe_inputs(59, t, h, e, i)
    gu, dn, _ = _quantise_all(ops, ctx, d, False)
    plan = ops.MoePlan(ctx, ops.MoePlanConfig(max_num_tokens=t, hidden_size=h, intermediate_size=i, num_experts=e, top_k=k,
                                              backend=ops.capi.MOE_BACKEND_NVFP4))
    hidden, router = to_dev(d["hidden"]), to_dev(d["router"])
    ws = torch.zeros(plan.layer_workspace_size(t, 0), dtype=torch.uint8, device="cuda")
    ids = torch.empty((t, k), dtype=torch.int32, device="cuda")
    w = torch.empty((t, k), dtype=torch.float32, device="cuda")
    outs = [torch.empty((t, h), dtype=torch.bfloat16, device="cuda") for _ in range(20)]
    for out in outs:
        ops.moe_layer_execute(plan, hidden, router, gu, dn, out, ws, topk_ids=ids, topk_weights=w)
    torch.cuda.synchronize()
    assert ctx.read_device_error() == 0
    assert tile_height(plan, ws, t) == rows
    hp, hs = oracle.nvfp4_quantize_act(d["hidden"], 1.0)
    _check(to_np(outs[0]), oracle.moe_nvfp4(hp, hs, to_np(ids), to_np(w), _triple(gu), _triple(dn)))
    assert all(torch.equal(out, outs[0]) for out in outs)


@pytest.mark.parametrize("cfg", [
    dict(t=60, h=512, e=8, k=2, i=256, linear=False, rows=64),
    dict(t=61, h=2048, e=8, k=2, i=512, linear=True, hot=True, rows=64),  # 61 rows: a row group that is not full
    dict(t=33, h=2048, e=4, k=2, i=256, linear=True, hot=True, rows=64),  # one row in the second 32-row half
    dict(t=70, h=256, e=8, k=2, i=256, linear=False, hot=True, rows=64),  # a second tile of six rows
    dict(t=40, h=256, e=8, k=2, i=256, linear=True, local=(3, 4), rows=64),
    dict(t=200, h=512, e=8, k=2, i=256, linear=False, rows=128),
    dict(t=61, h=2048, e=2, k=2, i=512, linear=True, rows=128),
    dict(t=33, h=2048, e=2, k=2, i=256, linear=True, rows=128),
    dict(t=90, h=256, e=8, k=2, i=256, linear=True, local=(3, 4), rows=128),
])
def test_64_row_token_tiles(ops, ctx, oracle, cfg):
    """More than a decode batch's rows per expert, still too few for 128-row tiles (which the last ones take): token rows
    read in place from tiled (layer call) and row-major (declared call) scales."""
    t, h, e, k, i = (cfg[n] for n in ("t", "h", "e", "k", "i"))
    off, le = cfg.get("local", (0, e))
    d = make_moe_inputs(43, t, h, e, i)
    d["gate_up"], d["down"] = d["gate_up"][off:off + le], d["down"][off:off + le]
    gu, dn, _ = _quantise_all(ops, ctx, d, False)
    plan = ops.MoePlan(ctx, ops.MoePlanConfig(max_num_tokens=t, hidden_size=h, intermediate_size=i, num_experts=e,
                                              top_k=k, local_expert_offset=off, local_num_experts=le,
                                              backend=ops.capi.MOE_BACKEND_NVFP4))
    bias = _hot_bias(e) if cfg.get("hot") else np.zeros(e, np.float32)
    ids, w = oracle.router_topk(oracle.gemm_bf16(d["hidden"], d["router"], "f32") + bias, k, 0, True, 1.0)
    out = torch.empty((t, h), dtype=torch.bfloat16, device="cuda")
    hp, hs = oracle.nvfp4_quantize_act(d["hidden"], 1.0)
    gu_ref, dn_ref = _triple(gu), _triple(dn)
    if cfg["linear"]:  # this call has no gate_up global scale: quantised against 1, weights scaled up
        def quantise(x):
            q = oracle.nvfp4_quantize_act(bf16(f32(x) * 8.0).reshape(-1, x.shape[2]), 1.0)
            return tuple(v.reshape(le, x.shape[1], -1) for v in q) + (np.ones(le, np.float32),)
        gu_ref, dn_ref = quantise(d["gate_up"]), quantise(d["down"])
        ws = torch.zeros(plan.workspace_size(t), dtype=torch.uint8, device="cuda")
        ops.moe_execute_nvfp4(plan, to_dev(hp), to_dev(hs), to_dev(ids), to_dev(w), *map(to_dev, gu_ref[:2]),
                              *map(to_dev, dn_ref[:2]), out, ws)
    else:
        ws = torch.zeros(plan.layer_workspace_size(t, 0), dtype=torch.uint8, device="cuda")
        ids_t = torch.empty((t, k), dtype=torch.int32, device="cuda")
        w_t = torch.empty((t, k), dtype=torch.float32, device="cuda")
        ops.moe_layer_execute(plan, to_dev(d["hidden"]), to_dev(d["router"]), gu, dn, out, ws, router_bias=to_dev(bias),
                              topk_ids=ids_t, topk_weights=w_t)
        ids, w = to_np(ids_t), to_np(w_t)
    torch.cuda.synchronize()
    assert ctx.read_device_error() == 0
    assert tile_height(plan, ws, t) == cfg["rows"]
    _check(to_np(out), oracle.moe_nvfp4(hp, hs, ids, w, gu_ref, dn_ref, local_offset=off))


def _chosen_height(ids, e):
    """The sort's choice between 64- and 128-row tiles: fewer tiles, a 64-row one counted as 5 and a 128-row one as 7."""
    counts = np.bincount(ids.ravel(), minlength=e)
    return 64 if 5 * np.sum((counts + 63) // 64) < 7 * np.sum((counts + 127) // 128) else 128


@pytest.mark.parametrize("t,hot,rows", [(641, 0.0, 64), (700, 0.0, 64), (1280, 0.0, 128), (641, 1.0, 64), (700, 1.0, 64),
                                        (1280, 1.0, 64), (641, 6.0, 128), (700, 6.0, 128), (1200, 6.0, 128)])
@pytest.mark.parametrize("s", [0, 256])
def test_tile_height_chosen_by_the_sort(ops, ctx, oracle, t, hot, rows, s):
    """40 to 80 rows per expert: 64-row tiles where they are not too many, alone and beside a shared expert (side stream)."""
    h, e, k, i = 256, 64, 4, 256
    d = make_moe_inputs(47, t, h, e, i, s)
    bias = np.where(np.arange(e) < 6, hot, 0.0).astype(np.float32)
    gu, dn, sh = _quantise_all(ops, ctx, d, bool(s))
    plan = ops.MoePlan(ctx, ops.MoePlanConfig(max_num_tokens=t, hidden_size=h, intermediate_size=i, num_experts=e, top_k=k,
                                              backend=ops.capi.MOE_BACKEND_NVFP4))
    out = torch.empty((t, h), dtype=torch.bfloat16, device="cuda")
    ws = torch.zeros(plan.layer_workspace_size(t, s), dtype=torch.uint8, device="cuda")
    ids = torch.empty((t, k), dtype=torch.int32, device="cuda")
    w = torch.empty((t, k), dtype=torch.float32, device="cuda")
    shared = ops.SharedExpert(sh[0], sh[1], to_dev(d["sh_gate"]), s) if s else None
    ops.moe_layer_execute(plan, to_dev(d["hidden"]), to_dev(d["router"]), gu, dn, out, ws, router_bias=to_dev(bias),
                          shared=shared, topk_ids=ids, topk_weights=w)
    torch.cuda.synchronize()
    assert ctx.read_device_error() == 0
    assert _chosen_height(to_np(ids), e) == rows == tile_height(plan, ws, t)
    hp, hs = oracle.nvfp4_quantize_act(d["hidden"], 1.0)
    shared_ref = dict(gu=_triple(sh[0]), d=_triple(sh[1]), gate_w=d["sh_gate"]) if s else None
    _check(to_np(out), oracle.moe_nvfp4(hp, hs, to_np(ids), to_np(w), _triple(gu), _triple(dn), shared=shared_ref,
                                        hidden_bf16=d["hidden"]))


@pytest.mark.parametrize("hot,rows", [(0.0, 64), (6.0, 128)])
def test_tile_height_chosen_in_the_declared_call(ops, ctx, oracle, hot, rows):
    t, h, e, k, i = 660, 256, 64, 4, 256
    d = make_moe_inputs(53, t, h, e, i)
    bias = np.where(np.arange(e) < 6, hot, 0.0).astype(np.float32)
    ids, w = oracle.router_topk(oracle.gemm_bf16(d["hidden"], d["router"], "f32") + bias, k, 0, True, 1.0)

    def quantise(x):  # this call has no gate_up global scale: quantised against 1, weights scaled up
        q = oracle.nvfp4_quantize_act(bf16(f32(x) * 8.0).reshape(-1, x.shape[2]), 1.0)
        return tuple(v.reshape(e, x.shape[1], -1) for v in q) + (np.ones(e, np.float32),)
    gu, dn = quantise(d["gate_up"]), quantise(d["down"])
    hp, hs = oracle.nvfp4_quantize_act(d["hidden"], 1.0)
    plan = ops.MoePlan(ctx, ops.MoePlanConfig(max_num_tokens=t, hidden_size=h, intermediate_size=i, num_experts=e, top_k=k,
                                              backend=ops.capi.MOE_BACKEND_NVFP4))
    ws = torch.zeros(plan.workspace_size(t), dtype=torch.uint8, device="cuda")
    out = torch.empty((t, h), dtype=torch.bfloat16, device="cuda")
    ops.moe_execute_nvfp4(plan, to_dev(hp), to_dev(hs), to_dev(ids), to_dev(w), *map(to_dev, gu[:2]), *map(to_dev, dn[:2]),
                          out, ws)
    torch.cuda.synchronize()
    assert ctx.read_device_error() == 0
    assert _chosen_height(ids, e) == rows == tile_height(plan, ws, t)
    _check(to_np(out), oracle.moe_nvfp4(hp, hs, ids, w, gu, dn))


# k of the down projections up to the longest resident panel: six and seven blocks of 256 leave a ring of one stage beside the
# staged output, eight none (rows stored directly); tiles with few rows and with many, a shared expert of another size
@pytest.mark.parametrize("t,e,k,h,i,s", [(130, 2, 1, 256, 1536, 0), (130, 2, 1, 256, 1792, 2048), (300, 2, 2, 512, 2048, 0),
                                         (3, 8, 1, 512, 256, 2048), (200, 4, 1, 256, 2048, 2048)])
def test_longest_down_projections(ops, ctx, oracle, t, e, k, h, i, s):
    d = make_moe_inputs(72, t, h, e, i, s)
    gu, dn, sh = _quantise_all(ops, ctx, d, bool(s))
    plan = ops.MoePlan(ctx, ops.MoePlanConfig(max_num_tokens=t, hidden_size=h, intermediate_size=i, num_experts=e, top_k=k,
                                              backend=ops.capi.MOE_BACKEND_NVFP4))
    ws = torch.zeros(plan.layer_workspace_size(t, s), dtype=torch.uint8, device="cuda")
    ids = torch.empty((t, k), dtype=torch.int32, device="cuda")
    w = torch.empty((t, k), dtype=torch.float32, device="cuda")
    out = torch.empty((t, h), dtype=torch.bfloat16, device="cuda")
    ops.moe_layer_execute(plan, to_dev(d["hidden"]), to_dev(d["router"]), gu, dn, out, ws, topk_ids=ids, topk_weights=w,
                          shared=ops.SharedExpert(sh[0], sh[1], to_dev(d["sh_gate"]), s) if s else None)
    torch.cuda.synchronize()
    assert ctx.read_device_error() == 0
    hp, hs = oracle.nvfp4_quantize_act(d["hidden"], 1.0)
    shared_ref = dict(gu=_triple(sh[0]), d=_triple(sh[1]), gate_w=d["sh_gate"]) if s else None
    _check(to_np(out), oracle.moe_nvfp4(hp, hs, to_np(ids), to_np(w), _triple(gu), _triple(dn), shared=shared_ref,
                                        hidden_bf16=d["hidden"]))
