"""GPU parity of the router, the route permutation and the element-wise helpers,
through the C ABI, against the CPU oracle and the upstream known-answer cases."""
import numpy as np
import pytest
import torch

from helpers import bf16, f32, make_moe_inputs, parse_floats, to_dev, to_np

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from qs3_b200 import ops as m
    return m


def _run_router(ops, logits_np, top_k, score, renorm, scale, as_bf16=False):
    t, e = logits_np.shape
    logits = to_dev(bf16(logits_np)) if as_bf16 else to_dev(logits_np.astype(np.float32))
    ids = torch.full((t, top_k), -7, dtype=torch.int32, device="cuda")
    w = torch.full((t, top_k), -7.0, dtype=torch.float32, device="cuda")
    ops.router_topk(logits, ids, w, score=score, renormalize=renorm, routed_scaling_factor=scale)
    torch.cuda.synchronize()
    return to_np(ids), to_np(w)


@pytest.mark.parametrize("name", ["router_softmax_ties", "router_sigmoid_bf16", "router_nonfinite"])
def test_router_known_answers(ops, oracle, golden, name):
    case = golden[name]
    logits = parse_floats(case["logits"]).reshape(case["num_tokens"], case["num_experts"])
    as_bf16 = name == "router_sigmoid_bf16"
    ids, w = _run_router(ops, logits, case["top_k"], case["score"], bool(case["renormalize"]),
                         case["scale"], as_bf16)
    assert ids.tolist() == case["expected_ids"]
    ref_logits = f32(bf16(logits)) if as_bf16 else logits
    _, w_ref = oracle.router_topk(ref_logits, case["top_k"], case["score"], bool(case["renormalize"]),
                                  case["scale"])
    assert np.all(np.isfinite(w))
    assert np.allclose(w, w_ref, atol=case["weight_tolerance"], rtol=0)
    if "expected_weights" in case:
        assert np.allclose(w, case["expected_weights"], atol=case["weight_tolerance"], rtol=0)


@pytest.mark.parametrize("shape", [(16, 8, 2), (64, 128, 8), (257, 512, 10), (33, 4096, 16), (5, 6, 3),
                                   (1, 1, 1), (1000, 256, 8)])
@pytest.mark.parametrize("score", [0, 1])
def test_router_matches_oracle(ops, oracle, shape, score):
    t, e, k = shape
    rng = np.random.default_rng(1000 * t + e + score)
    logits = rng.standard_normal((t, e), dtype=np.float32) * 1.5
    if score == 1:
        # sigmoid scores saturate and the device uses a fast exp: keep distinct logits
        # far enough apart that score ordering equals logit ordering on both sides
        logits = np.clip(np.round(logits * 4) / 4, -6, 6).astype(np.float32)
    else:
        logits[: t // 2] = np.round(logits[: t // 2] * 2) / 2  # exact ties in half of the rows
    for renorm, scale in ((True, 1.0), (False, 2.5)):
        ids, w = _run_router(ops, logits, k, score, renorm, scale)
        ids_ref, w_ref = oracle.router_topk(logits, k, score, renorm, scale)
        assert np.array_equal(ids, ids_ref)
        assert np.allclose(w, w_ref, atol=1e-5 * scale, rtol=0)
    # bf16 logits take the same path after widening
    lb = f32(bf16(logits))
    ids, w = _run_router(ops, logits, k, score, True, 1.0, as_bf16=True)
    ids_ref, w_ref = oracle.router_topk(lb, k, score, True, 1.0)
    assert np.array_equal(ids, ids_ref)
    assert np.allclose(w, w_ref, atol=1e-5, rtol=0)


def test_router_nan_rows_and_unfilled_slots(ops, oracle):
    logits = np.array([[np.nan, -np.inf, np.nan, 1.0],
                       [np.nan, np.nan, np.nan, np.nan],
                       [np.inf, 0.0, np.inf, -1.0]], np.float32)
    for score in (0, 1):
        ids, w = _run_router(ops, logits, 3, score, True, 1.0)
        ids_ref, w_ref = oracle.router_topk(logits, 3, score, True, 1.0)
        assert np.array_equal(ids, ids_ref)
        assert np.array_equal(np.isnan(w), np.isnan(w_ref))
        m = ~np.isnan(w_ref)
        assert np.allclose(w[m], w_ref[m], atol=1e-5, rtol=0)


def _route_tables(ops, ids_np, w_np, experts, local_offset, local_experts):
    """Run a tiny bf16 MoE (H = I = 8, CUDA-core GEMM) only to obtain the routing tables."""
    t, k = ids_np.shape
    h = i = 8
    ctx = ops.Context()
    plan = ops.MoePlan(ctx, ops.MoePlanConfig(max_num_tokens=t, hidden_size=h, intermediate_size=i,
                                              num_experts=experts, top_k=k,
                                              local_expert_offset=local_offset,
                                              local_num_experts=local_experts))
    ws = torch.zeros(plan.workspace_size(t), dtype=torch.uint8, device="cuda")
    hidden = torch.zeros((t, h), dtype=torch.bfloat16, device="cuda")
    gu = torch.zeros((local_experts, 2 * i, h), dtype=torch.bfloat16, device="cuda")
    dn = torch.zeros((local_experts, h, i), dtype=torch.bfloat16, device="cuda")
    out = torch.empty((t, h), dtype=torch.bfloat16, device="cuda")
    ops.moe_execute_bf16(plan, hidden, to_dev(ids_np), to_dev(w_np), gu, dn, out, ws)
    tables = [to_np(x) for x in plan.routing_tables(ws, t)]
    assert ctx.read_device_error() == 0
    return tables


@pytest.mark.parametrize("case", [
    dict(t=16, k=2, e=8), dict(t=1, k=1, e=1), dict(t=37, k=4, e=11), dict(t=513, k=10, e=512),
    dict(t=2049, k=8, e=128), dict(t=300, k=3, e=4096, skew=True), dict(t=64, k=2, e=16, one_expert=True),
    dict(t=200, k=6, e=32, local=(8, 8)), dict(t=200, k=6, e=32, local=(24, 8)),
    # the one-block sort: its most routes and experts (two experts a thread), and one route more
    dict(t=256, k=10, e=896), dict(t=2560, k=1, e=513), dict(t=2561, k=1, e=512), dict(t=100, k=3, e=897), dict(t=250, k=8, e=1024),
    dict(t=1, k=1, e=1025),
])
def test_route_permutation_is_bit_exact(ops, oracle, case):
    t, k, e = case["t"], case["k"], case["e"]
    rng = np.random.default_rng(7 * t + e)
    if case.get("one_expert"):
        ids = np.full((t, k), 5, np.int32)
    elif case.get("skew"):
        ids = np.minimum((rng.pareto(0.7, size=(t, k)) * 3).astype(np.int64), e - 1).astype(np.int32)
    else:
        ids = rng.integers(0, e, size=(t, k), dtype=np.int32)
    ids[0, :] = ids[0, 0]  # duplicate routes inside one token (upstream test.cu:1586)
    w = rng.random((t, k), dtype=np.float32)
    off, le = case.get("local", (0, e))
    got = _route_tables(ops, ids, w, e, off, le)
    want = oracle.route_sort(ids, w, off, le)
    for name, g, r in zip(("counts", "indptr", "route_rows", "row_tokens", "row_scales"), got, want):
        assert np.array_equal(g, r), name


# more routes than one block sorts: two launches for 8 to 1024 experts and up to 256 chunks of 1024 routes, three beyond. The
# ends of those ranges, whole chunks and one route more, experts held by another rank
@pytest.mark.parametrize("t,k,e,local", [(2561, 1, 7, None), (2561, 1, 8, None), (3072, 1, 9, None), (3073, 1, 512, None),
                                         (513, 5, 1023, None), (700, 6, 1024, None), (700, 6, 1025, None),
                                         (900, 6, 64, (40, 8)), (900, 6, 64, (3, 57)), (900, 6, 64, (60, 4)),
                                         (65536, 4, 16, None), (65537, 4, 16, None)])
def test_sort_of_a_large_batch(ops, oracle, t, k, e, local):
    rng = np.random.default_rng(t + e)
    ids = rng.integers(0, e, size=(t, k), dtype=np.int32)
    ids[: t // 3] = ids[0, 0]
    w = rng.random((t, k), dtype=np.float32)
    off, le = local or (0, e)
    got = _route_tables(ops, ids, w, e, off, le)
    for name, g, r in zip(("counts", "indptr", "route_rows", "row_tokens", "row_scales"), got, oracle.route_sort(ids, w, off, le)):
        assert np.array_equal(g, r), name


def test_silu_and_mul(ops, oracle, golden):
    case = golden["silu_and_mul"]
    gate = bf16(case["gate"]).reshape(case["tokens"], case["intermediate"])
    up = bf16(case["up"]).reshape(case["tokens"], case["intermediate"])
    out = torch.full(gate.shape, 12345.0, dtype=torch.bfloat16, device="cuda")
    ops.silu_and_mul_bf16(to_dev(gate), to_dev(up), out)
    g, u = f32(gate).astype(np.float64), f32(up).astype(np.float64)
    assert np.max(np.abs(f32(to_np(out)) - g / (1 + np.exp(-g)) * u)) <= case["tolerance"]
    # larger, vectorised shape against the oracle: at most one bf16 step apart (fast exp on device)
    rng = np.random.default_rng(11)
    gate = bf16(rng.standard_normal((67, 512), dtype=np.float32) * 3)
    up = bf16(rng.standard_normal((67, 512), dtype=np.float32))
    out = torch.empty((67, 512), dtype=torch.bfloat16, device="cuda")
    ops.silu_and_mul_bf16(to_dev(gate), to_dev(up), out)
    ref = f32(oracle.silu_and_mul_bf16(gate, up))
    got = f32(to_np(out))
    assert np.all(np.abs(got - ref) <= np.abs(ref) * 2.0 ** -7 + 1e-30)


def test_shared_expert_gate_add(ops, oracle, golden):
    case = golden["shared_expert_gate_add"]
    rows, hidden = case["rows"], case["hidden"]
    shared = bf16(case["shared"]).reshape(rows, hidden)
    out0 = bf16(case["out"]).reshape(rows, hidden)
    for gate_t in (to_dev(np.array(case["gate"], np.float32).reshape(rows, 1)),
                   to_dev(bf16(case["gate"]).reshape(rows, 1))):
        out = to_dev(out0)
        ops.shared_expert_gate_add_bf16(gate_t, to_dev(shared), out)
        ref = f32(oracle.shared_gate_add_bf16(np.array(case["gate"], np.float32), shared, out0))
        assert np.max(np.abs(f32(to_np(out)) - ref)) <= case["tolerance"]


# sizes of the launch that routes and sorts a small batch: one token, a full block of warps, one more, more experts than
# its larger batches take; part of the experts local
@pytest.mark.parametrize("t,e,k,local", [(1, 8, 2, None), (16, 128, 8, None), (17, 128, 8, None), (8, 512, 10, (100, 300)),
                                         (9, 512, 10, None), (3, 40, 4, (32, 8))])
def test_router_and_sort_of_a_small_batch(ops, oracle, t, e, k, local):
    h, i = 128, 64
    off, le = local or (0, e)
    d = make_moe_inputs(90 + t, t, h, e, i)
    ctx = ops.Context()
    plan = ops.MoePlan(ctx, ops.MoePlanConfig(max_num_tokens=t, hidden_size=h, intermediate_size=i, num_experts=e, top_k=k,
                                              local_expert_offset=off, local_num_experts=le))
    ws = torch.zeros(plan.layer_workspace_size(t, 0), dtype=torch.uint8, device="cuda")
    out = torch.empty((t, h), dtype=torch.bfloat16, device="cuda")
    ids = torch.empty((t, k), dtype=torch.int32, device="cuda")
    w = torch.empty((t, k), dtype=torch.float32, device="cuda")
    logits = torch.empty((t, e), dtype=torch.float32, device="cuda")
    ops.moe_layer_execute(plan, to_dev(d["hidden"]), to_dev(d["router"]), to_dev(d["gate_up"][off:off + le]),
                          to_dev(d["down"][off:off + le]), out, ws, topk_ids=ids, topk_weights=w, router_logits=logits)
    torch.cuda.synchronize()
    ids_ref, w_ref = oracle.router_topk(to_np(logits), k, 0, True, 1.0)
    assert np.array_equal(to_np(ids), ids_ref)
    np.testing.assert_allclose(to_np(w), w_ref, rtol=1e-5)
    tables = [to_np(x) for x in plan.routing_tables(ws, t)]
    for g, r in zip(tables, oracle.route_sort(to_np(ids), to_np(w), off, le)):
        assert np.array_equal(g, r)


def _tile_tables(counts, choose):
    """Host restatement of the padded segments and tiles that the NVFP4 GEMMs read: 128-row tiles and their pairs, or, where
    the sort may choose and they come out cheaper, 64-row tiles."""
    tiles = lambda h: (counts + h - 1) // h
    small = choose and 5 * tiles(64).sum() < 7 * tiles(128).sum()
    h = 64 if small else 128
    pad = np.concatenate([[0], np.cumsum(tiles(h) * h)])
    table = [(e, pad[e] + m * h, min(h, n - m * h)) for e, n in enumerate(counts) for m in range((n + h - 1) // h)]
    pairs = [] if small else [(e, pad[e] + m * 256, min(256, n - m * 256)) for e, n in enumerate(counts) for m in range((n + 127) // 256)]
    # (an expert's odd last tile; the singles fill the table from its end)
    singles = [] if small else [(e, pad[e] + (n - 1) // 128 * 128, (n - 1) % 128 + 1)
                                for e, n in enumerate(counts) if (n + 127) // 128 % 2]
    return small, pad, table, pairs, singles


# the two-launch sort at the ends of its range, for the tables of the NVFP4 GEMMs: whole chunks and one more or less, one
# expert's tiles beside another block's, both tile heights where the sort chooses, none where it may not (few routes; experts
# with more than 80 routes on average), experts held by another rank
@pytest.mark.parametrize("t,k,e,local,skew", [
    (2400, 10, 1023, None, False), (2400, 10, 1024, None, True), (2560, 10, 1024, None, False), (321, 8, 9, None, False),
    (1024, 3, 8, None, False), (513, 6, 64, None, False), (513, 6, 64, None, True), (700, 6, 64, (5, 50), False),
    (1025, 6, 257, None, False), (6000, 3, 200, (100, 100), False)])
def test_tile_tables_of_a_large_batch(ops, oracle, t, k, e, local, skew):
    off, le = local or (0, e)
    rng = np.random.default_rng(t + e)
    ids = rng.integers(0, e, size=(t, k), dtype=np.int32)
    if skew: # to a sixteenth of the experts
        ids = (off + ids % (le // 16)).astype(np.int32)
    w = rng.random((t, k), dtype=np.float32)
    h = i = 256
    ctx = ops.Context()
    plan = ops.MoePlan(ctx, ops.MoePlanConfig(max_num_tokens=t, hidden_size=h, intermediate_size=i, num_experts=e, top_k=k,
                                              local_expert_offset=off, local_num_experts=le,
                                              backend=ops.capi.MOE_BACKEND_NVFP4))
    ws = torch.full((plan.workspace_size(t),), 0xff, dtype=torch.uint8, device="cuda")
    zeros = lambda *shape: torch.zeros(shape, dtype=torch.uint8, device="cuda")
    ops.moe_execute_nvfp4(plan, zeros(t, h // 2), zeros(t, h // 16), to_dev(ids), to_dev(w), zeros(le, 2 * i, h // 2),
                          zeros(le, 2 * i, h // 16), zeros(le, h, i // 2), zeros(le, h, i // 16),
                          torch.empty((t, h), dtype=torch.bfloat16, device="cuda"), ws)
    torch.cuda.synchronize()
    assert ctx.read_device_error() == 0
    # the tables' places, in the order and alignment of the workspace
    routes = t * k
    assert routes > 2560 and routes > 22 * le    # two launches, tiles of 128 rows or a choice
    up = lambda v, a: (v + a - 1) // a * a
    seg, choose = min(routes, le), routes <= 80 * le
    max_tiles = (up(routes, 128) + seg * 128) // 128
    room = max(max_tiles, up(routes if choose else 80 * le, 64) // 64 + seg)
    sizes = [le, le + 1, le + 1, routes, routes, routes, routes, room, room, room, 1, 1, max_tiles, max_tiles, max_tiles, 2]
    at, tables = 0, []
    for n in sizes:
        at = up(at, 256)
        tables.append(to_np(ws[at:at + 4 * n].view(torch.int32)))
        at += 4 * n
    counts, indptr, pad, rows, prows, tokens, _, tile_e, tile_r, tile_n, total, alt, pair_e, pair_r, pair_n, pair_counts = tables
    want = oracle.route_sort(ids, w, off, le)
    assert np.array_equal(counts, want[0]) and np.array_equal(indptr, want[1]) and np.array_equal(rows, want[2])
    small, want_pad, table, pairs, singles = _tile_tables(want[0].astype(np.int64), choose)
    assert small == (choose and not skew)          # the case means both heights to occur
    assert np.array_equal(pad, want_pad)
    local_ids = ids.ravel() - off
    held = (local_ids >= 0) & (local_ids < le)
    assert np.array_equal(prows[held], (rows - np.asarray(want[1])[local_ids * held] + want_pad[local_ids * held])[held])
    assert np.all(prows[~held] == -1)
    assert np.array_equal(np.stack([tile_e, tile_r, tile_n], 1)[:len(table)], np.array(table).reshape(-1, 3))
    assert total[0] == (0 if small else len(table))
    if choose:
        assert alt[0] == (len(table) if small else 0)
    assert pair_counts.tolist() == [len(pairs), len(singles)]
    got = np.stack([pair_e, pair_r, pair_n], 1)
    assert np.array_equal(got[:len(pairs)], np.array(pairs).reshape(-1, 3))
    assert np.array_equal(got[::-1][:len(singles)], np.array(singles).reshape(-1, 3))
