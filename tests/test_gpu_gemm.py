"""GPU parity of the dense bf16 GEMM entry (qscb_gemm_bf16: router logits and the
shared-expert projections) against the CPU oracle."""
import numpy as np
import pytest
import torch

from helpers import bf16, f32, to_dev, to_np

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gemm():
    from qs3_b200 import ops
    return ops.GemmContext()


def _ref(x, w):
    return f32(x).astype(np.float64) @ f32(w).astype(np.float64).T


def test_identity_known_answer(gemm):
    # one 128 x 128 x 64 tile: x = eye-like, weight rows = distinct small integers
    x = np.zeros((128, 64), np.float32)
    x[np.arange(128), np.arange(128) % 64] = 1.0
    w = (np.arange(128 * 64).reshape(128, 64) % 251 - 125).astype(np.float32)
    out = torch.zeros((128, 128), dtype=torch.float32, device="cuda")
    gemm.gemm_bf16(to_dev(bf16(x)), to_dev(bf16(w)), out)
    torch.cuda.synchronize()
    want = x.astype(np.float64) @ f32(bf16(w)).astype(np.float64).T
    assert np.array_equal(to_np(out), want.astype(np.float32))


@pytest.mark.parametrize("shape", [(2, 64, 128), (16, 256, 8), (130, 2048, 512), (64, 200, 96),
                                   (300, 72, 130), (8192 // 8, 2048, 512), (5, 12, 7), (128, 4096, 64)])
@pytest.mark.parametrize("out_dtype", ["f32", "bf16"])
def test_gemm_matches_oracle(gemm, oracle, shape, out_dtype):
    rows, k, n = shape
    rng = np.random.default_rng(rows * 7 + k + n)
    x = bf16(rng.standard_normal((rows, k), dtype=np.float32))
    w = bf16(rng.standard_normal((n, k), dtype=np.float32) * 0.05)
    ref64 = _ref(x, w)
    if out_dtype == "f32":
        out = torch.full((rows, n), 777.0, dtype=torch.float32, device="cuda")
        gemm.gemm_bf16(to_dev(x), to_dev(w), out)
        got = to_np(out).astype(np.float64)
        # tensor-core accumulation is a little below IEEE f32: ~2e-6 of the norm at k = 2048
        assert np.linalg.norm(got - ref64) <= 1e-5 * np.linalg.norm(ref64) + 1e-12
        o = oracle.gemm_bf16(x, w, "f32").astype(np.float64)
        assert np.linalg.norm(got - o) <= 1e-5 * np.linalg.norm(ref64) + 1e-12
    else:
        out = torch.full((rows, n), 777.0, dtype=torch.bfloat16, device="cuda")
        gemm.gemm_bf16(to_dev(x), to_dev(w), out)
        got = f32(to_np(out)).astype(np.float64)
        assert np.all(np.abs(got - ref64) <= np.abs(ref64) * 2.0 ** -8 + 1e-4)


def test_alpha_beta_and_padded_strides(gemm):
    # upstream tests_cuda_qscb_gemm.inc:719-921: f32 output with beta and padded row strides,
    # sentinel padding must survive
    rows, k, n = 37, 264, 48
    rng = np.random.default_rng(9)
    x_full = torch.full((rows, k + 8), 3.0, dtype=torch.bfloat16, device="cuda")
    w_full = torch.full((n, k + 16), -2.0, dtype=torch.bfloat16, device="cuda")
    o_full = torch.full((rows, n + 4), 5.0, dtype=torch.float32, device="cuda")
    x = bf16(rng.standard_normal((rows, k), dtype=np.float32))
    w = bf16(rng.standard_normal((n, k), dtype=np.float32) * 0.1)
    c = rng.standard_normal((rows, n), dtype=np.float32)
    x_full[:, :k] = to_dev(x)
    w_full[:, :k] = to_dev(w)
    o_full[:, :n] = to_dev(c)
    gemm.gemm_bf16(x_full[:, :k], w_full[:, :k], o_full[:, :n], alpha=0.5, beta=-1.5)
    got = to_np(o_full)
    want = 0.5 * _ref(x, w) - 1.5 * c
    assert np.allclose(got[:, :n], want, atol=2e-4, rtol=1e-5)
    assert np.all(got[:, n:] == 5.0)
    # bf16 output with beta
    ob = torch.full((rows, n), 0.0, dtype=torch.bfloat16, device="cuda")
    ob.copy_(to_dev(bf16(c)))
    gemm.gemm_bf16(x_full[:, :k], w_full[:, :k], ob, alpha=2.0, beta=1.0)
    want = 2.0 * _ref(x, w) + f32(bf16(c))
    assert np.all(np.abs(f32(to_np(ob)) - want) <= np.abs(want) * 2.0 ** -8 + 1e-5)


def test_validation_errors(gemm):
    from qs3_b200 import ops
    x = torch.zeros((4, 64), dtype=torch.bfloat16, device="cuda")
    w = torch.zeros((8, 64), dtype=torch.bfloat16, device="cuda")
    with pytest.raises(ops.Qs3Error) as e:
        gemm.gemm_bf16(x, w, torch.zeros((4, 9), dtype=torch.float32, device="cuda"))
    assert e.value.status == 1 and "shape mismatch" in e.value.message
    with pytest.raises(ops.Qs3Error) as e:
        gemm.gemm_bf16(x.float(), w, torch.zeros((4, 8), dtype=torch.float32, device="cuda"))
    assert e.value.status == 1


@pytest.mark.parametrize("kind", ["bf16", "fp8", "nvfp4"])
def test_tensor_peak_probe_runs(kind):
    # the probe is a measurement aid: it must finish, report a plausible positive rate
    # and leave the device error word clear (all its waits are bounded)
    from qs3_b200 import ops
    ctx = ops.Context()
    tf = ops.tensor_peak_probe(ctx, kind, n=128, iters=2000)
    assert 10.0 < tf < 40000.0
    assert ctx.read_device_error() == 0


# split k: one row, every tile height and its neighbours, n and k tails, splits past the end of k (k = 576: nine
# blocks over eight ranks of two), several row tiles
@pytest.mark.parametrize("shape", [(1, 2048, 512), (17, 576, 130), (33, 2056, 100), (64, 128, 2048), (65, 2048, 131),
                                   (257, 512, 512)])
@pytest.mark.parametrize("beta", [0.0, 0.5])
def test_splitk_kernel(gemm, shape, beta):
    rows, k, n = shape
    rng = np.random.default_rng(rows + k + n)
    x = bf16(rng.standard_normal((rows, k), dtype=np.float32))
    w = bf16(rng.standard_normal((n, k), dtype=np.float32) * 0.05)
    c = rng.standard_normal((rows, n), dtype=np.float32)
    full = torch.full((rows, n + 3), 7.0, dtype=torch.float32, device="cuda")
    out = full[:, :n]
    out.copy_(torch.from_numpy(c))
    gemm.gemm_bf16(to_dev(x), to_dev(w), out, alpha=0.25, beta=beta)
    want = 0.25 * _ref(x, w) + beta * c.astype(np.float64)
    got = to_np(out).astype(np.float64)
    assert np.linalg.norm(got - want) <= 1e-5 * np.linalg.norm(want)
    assert torch.all(full[:, n:] == 7.0)
    again = out.clone()
    out.copy_(torch.from_numpy(c))
    gemm.gemm_bf16(to_dev(x), to_dev(w), out, alpha=0.25, beta=beta)
    assert torch.equal(again, out)


# f32 results of few rows: on the CUDA cores (few features), split k with 16-, 32- and 64-row tiles, a k tail, more tiles
# than SMs. A sum in one tensor-core chain truncates in every instruction and is off by 2e-6 at k = 2048; chains of two
# instructions (at most 2^-23 of the value each, half of that on average) and a rounding stay within 1e-7.
@pytest.mark.parametrize("shape", [(1, 2048, 128), (64, 1024, 64), (1, 2048, 512), (17, 576, 300), (33, 2048, 512),
                                   (64, 2048, 1100), (24, 2056, 4096), (40, 2048, 5000), (64, 512, 38000)])
def test_f32_sums_of_few_rows(gemm, shape):
    rows, k, n = shape
    g = torch.Generator(device="cuda").manual_seed(rows + k + n)
    x = torch.randn((rows, k), generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn((n, k), generator=g, device="cuda") * 0.02).to(torch.bfloat16)
    out = torch.empty((rows, n), dtype=torch.float32, device="cuda")
    gemm.gemm_bf16(x, w, out)
    want = x.double() @ w.double().t()
    assert float((out.double() - want).norm()) <= 1e-7 * float(want.norm())
    # an infinity stays one, two of different sign make a NaN, and other rows and columns keep their sums
    x2, w2 = x.clone(), w.clone()
    x2[0, k - 1] = float("inf")
    x2[rows - 1, 3] = float("-inf")
    w2[5, 70] = float("inf")
    again = torch.empty_like(out)
    gemm.gemm_bf16(x2, w2, again)
    special = ~torch.isfinite(again)
    ref = x2.double() @ w2.double().t()
    assert torch.equal(special, ~torch.isfinite(ref))
    assert torch.equal(torch.isnan(again), torch.isnan(ref))
    assert torch.equal(again[special & ~torch.isnan(ref)].double(), ref[special & ~torch.isnan(ref)])
    assert torch.equal(again[~special], out[~special])


# at most 64 rows and at least 148 units of features: weights streamed as the M side, unit height chosen for full
# rounds (37889 = 148 * 256 + 1 features: the last unit holds one), both row tile heights, rows in fours up to 48 and in
# boxes of 32 beyond (the second partly past the end); 128 rows: the dense kernel with a width chosen the same way
@pytest.mark.parametrize("rows,k,n", [(1, 64, 37889), (33, 200, 40000), (48, 64, 37633), (49, 128, 37700), (63, 200, 40000),
                                      (64, 72, 50007), (128, 128, 50007)])
def test_feature_streaming_kernel(gemm, rows, k, n):
    rng = np.random.default_rng(rows + k)
    x = bf16(rng.standard_normal((rows, k), dtype=np.float32))
    w = bf16(rng.standard_normal((n, k), dtype=np.float32) * 0.05)
    full = torch.full((rows, n + 1), 7.0, dtype=torch.bfloat16, device="cuda")
    gemm.gemm_bf16(to_dev(x), to_dev(w), full[:, :n])
    want = torch.from_numpy(_ref(x, w)).to(torch.bfloat16).float().numpy()
    got = full[:, :n].float().cpu().numpy()
    assert np.max(np.abs(got - want)) <= 2.0 ** -7 * np.max(np.abs(want))
    assert torch.all(full[:, n] == 7.0)


@pytest.mark.parametrize("shape", [(65, 64, 128), (129, 64, 257), (257, 192, 300), (700, 1024, 2304), (128, 2048, 5000),
                                   (2100, 256, 2400), (2305, 128, 2048)])   # the last two: CTA-pair kernel
@pytest.mark.parametrize("out_dtype", ["f32", "bf16"])
def test_dense_kernel_edges_and_epilogue(gemm, shape, out_dtype):
    """More than 64 rows, k a multiple of 64, n >= 128: the persistent 128 x 256 kernel, or with at
    least 74 tiles of 256 x 256 its CTA-pair variant. Ragged rows and columns, alpha / beta, padded
    row strides (sentinel padding must survive)."""
    rows, k, n = shape
    rng = np.random.default_rng(rows + 3 * k + 5 * n)
    x = bf16(rng.standard_normal((rows, k), dtype=np.float32))
    w = bf16(rng.standard_normal((n, k), dtype=np.float32) * 0.05)
    c = bf16(rng.standard_normal((rows, n), dtype=np.float32))
    dt = torch.float32 if out_dtype == "f32" else torch.bfloat16
    x_full = torch.full((rows, k + 8), 3.0, dtype=torch.bfloat16, device="cuda")
    w_full = torch.full((n, k + 24), -2.0, dtype=torch.bfloat16, device="cuda")
    o_full = torch.full((rows, n + 8), 5.0, dtype=dt, device="cuda")
    x_full[:, :k] = to_dev(x)
    w_full[:, :k] = to_dev(w)
    o_full[:, :n] = to_dev(c).to(dt)
    gemm.gemm_bf16(x_full[:, :k], w_full[:, :k], o_full[:, :n], alpha=0.5, beta=-1.5)
    torch.cuda.synchronize()
    got = o_full.float().cpu().numpy().astype(np.float64)
    want = 0.5 * _ref(x, w) - 1.5 * f32(c).astype(np.float64)
    if out_dtype == "f32":
        assert np.linalg.norm(got[:, :n] - want) <= 1e-5 * np.linalg.norm(want) + 1e-9
    else:
        assert np.all(np.abs(got[:, :n] - want) <= np.abs(want) * 2.0 ** -7 + 2e-3)
    assert np.all(got[:, n:] == 5.0)


# Outputs gathered in shared memory and written by TMA: last tiles of 8 columns and of one row, a row pitch beyond the
# columns, columns that end inside 16 bytes (stored row by row instead); tiles of 32 to 256 columns by one CTA or two, and
# split k with as many stages as a rank has k blocks.
@pytest.mark.parametrize("shape", [(129, 64, 136, 0), (72, 512, 4096, 8), (300, 512, 2504, 8), (257, 128, 2500, 12),
                                   (500, 2048, 2048, 0), (1290, 192, 2561, 7), (1025, 2048, 4104, 24), (2049, 512, 4096, 0),
                                   (130, 4096, 2048, 0), (80, 4096, 512, 16), (190, 704, 520, 8)])
@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("beta", [0.0, 0.5])
def test_dense_output_edges(gemm, shape, out_dtype, beta):
    rows, k, n, pad = shape
    gen = torch.Generator().manual_seed(rows + n)
    x = torch.randn((rows, k), generator=gen).to(torch.bfloat16)
    w = torch.randn((n, k), generator=gen).to(torch.bfloat16)
    full = torch.full((rows + 2, n + pad), 7.0, dtype=out_dtype, device="cuda")
    gemm.gemm_bf16(x.cuda(), w.cuda(), full[:rows, :n], alpha=0.5, beta=beta)
    got = full.cpu()
    assert torch.all(got[rows:] == 7.0) and torch.all(got[:, n:] == 7.0)
    # products of bf16 are exact in f32. The tensor core drops what lies below 2^-24 or so of an accumulator each time it adds
    # one of k / 16 terms: k / 16 * 2^-24 of the sum of the magnitudes bounds that; a bf16 result is then rounded by 2^-9.
    want = 0.5 * (x.double() @ w.double().T) + beta * 7.0
    size = 0.5 * (x.double().abs() @ w.double().abs().T) + beta * 7.0
    bound = size * (k / 16 + 4) * 2.0 ** -24
    if out_dtype == torch.bfloat16:
        bound += want.abs() * 2.0 ** -8
    assert torch.all((got[:rows, :n].double() - want).abs() <= bound)


# short problems whose output is read as well: split over k, where the other kernels would go through the output row by row
@pytest.mark.parametrize("shape", [(127, 1024, 512, 0), (1500, 512, 128, 8), (257, 512, 250, 7)])
@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
def test_short_dense_problems_with_beta(gemm, shape, out_dtype):
    test_dense_output_edges(gemm, shape, out_dtype, 0.75)
