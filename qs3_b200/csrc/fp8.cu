// FP8 block-scaled expert path (e4m3 weights with one f32 scale per 128 x 128 block,
// e4m3 activations with one f32 scale per token per 128 elements): quantisers
// and the choice of the grouped GEMM (tcgen05, kind::f8f6f4).
//
// Upstream has no FP8 MoE surface (only the dtype enum values, qs_tensor.h:20-24); the
// conventions are this library's and are restated by the CPU oracle:
//   scale = max(amax / 448, 1e-30);  code = e4m3_rn_sat(x * (1 / scale))
//
// 128 x 128 block scales are not a tcgen05 block-scale format, so every 128-wide k block is accumulated on its own in
// tensor memory and promoted into f32 registers as acc += partial * (w_scale[block] * x_scale[token, k block]):
// fp8_stream.cu (weight streaming, experts with few rows) and fp8_rows.cu (token rows on the M side).
#include "fp8.cuh"
#include "tcgen05.cuh"

#include <algorithm>

namespace qs3 {

namespace {

using namespace tc;

// ---- quantisers -------------------------------------------------------------------------

// codes[row, :] / scales[row, :] = quantise(x[row, :]); 16 lanes per (row, 128-element group), eight elements per lane.
__global__ void __launch_bounds__(256)
fp8_quantize_rows_kernel(const __nv_bfloat16* __restrict__ x, uint32_t rows, uint32_t k, uint8_t* __restrict__ codes,
                         float* __restrict__ scales)
{
    chain_begin();
    fp8_quantize_groups(x, rows, k, codes, scales, static_cast<uint64_t>(blockIdx.x) * 8 + (threadIdx.x >> 5));
}

// One block per (k block, row block, expert): 128 x 128 weights -> codes + one scale. Sixteen lanes read the
// 256 bytes of a row together, so a load or store instruction touches whole sectors. Bound by HBM: 2 bytes in,
// 1 byte out per weight.
__global__ void __launch_bounds__(256)
fp8_quantize_weight_kernel(const __nv_bfloat16* __restrict__ w, uint32_t rows, uint32_t k,
                           uint8_t* __restrict__ codes, float* __restrict__ scales)
{
    __shared__ float s_part[8];
    const uint32_t kb = blockIdx.x, rb = blockIdx.y, e = blockIdx.z;
    const uint32_t r0 = rb * 128 + threadIdx.x / 16; // rows r0, r0 + 16, ...
    const uint32_t c0 = kb * 128 + (threadIdx.x % 16) * 8;
    const size_t base = (static_cast<size_t>(e) * rows + r0) * k + c0;
    uint4 v[8];
    float amax = 0.0f;
#pragma unroll
    for (uint32_t i = 0; i < 8; ++i)
        v[i] = r0 + 16 * i < rows ? *reinterpret_cast<const uint4*>(w + base + static_cast<size_t>(16 * i) * k)
                                  : make_uint4(0, 0, 0, 0);
#pragma unroll
    for (uint32_t i = 0; i < 8; ++i) {
        const uint32_t ws[4] = { v[i].x, v[i].y, v[i].z, v[i].w };
#pragma unroll
        for (int j = 0; j < 4; ++j)
            amax = fmaxf(amax, fmaxf(fabsf(bf16_bits_to_f32(ws[j] & 0xffffu)), fabsf(bf16_bits_to_f32(ws[j] >> 16))));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    if ((threadIdx.x & 31) == 0)
        s_part[threadIdx.x >> 5] = amax;
    __syncthreads();
    amax = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i)
        amax = fmaxf(amax, s_part[i]);
    const float s = fp8_scale_of(amax);
    const float inv = __fdiv_rn(1.0f, s);
#pragma unroll
    for (uint32_t i = 0; i < 8; ++i) {
        if (r0 + 16 * i < rows) {
            const float f[8] = { bf16_bits_to_f32(v[i].x & 0xffffu), bf16_bits_to_f32(v[i].x >> 16),
                                 bf16_bits_to_f32(v[i].y & 0xffffu), bf16_bits_to_f32(v[i].y >> 16),
                                 bf16_bits_to_f32(v[i].z & 0xffffu), bf16_bits_to_f32(v[i].z >> 16),
                                 bf16_bits_to_f32(v[i].w & 0xffffu), bf16_bits_to_f32(v[i].w >> 16) };
            *reinterpret_cast<uint2*>(codes + base + static_cast<size_t>(16 * i) * k)
                = make_uint2(pack_e4m3x4(f, inv), pack_e4m3x4(f + 4, inv));
        }
    }
    if (threadIdx.x == 0)
        scales[(static_cast<size_t>(e) * gridDim.y + rb) * gridDim.x + kb] = s;
}

} // namespace

uint32_t fp8_tile_rows(uint32_t routes, uint32_t experts)
{
    // Weight streaming reads an expert's weights once per 64 rows. Layer times, 128 experts top-8, 64- against 128-row
    // tiles: even routing 16 routes per expert 0.136 against 0.152 ms, 44: 0.164 against 0.172, 64: 0.186 against
    // 0.177; skewed routing 19: 0.102 against 0.103, 38: 0.139 against 0.137, 64: 0.182 against 0.160.
    return routes <= 40u * experts ? 64u : static_cast<uint32_t>(kTileM);
}

cudaError_t launch_fp8_quantize_rows(const __nv_bfloat16* x, uint32_t rows, uint32_t k, uint8_t* codes, float* scales,
                                     cudaStream_t stream)
{
    if (rows == 0)
        return cudaSuccess;
    const uint64_t units = static_cast<uint64_t>(rows) * (k / 128);
    return launch_chained(fp8_quantize_rows_kernel, dim3(static_cast<uint32_t>((units + 15) / 16)), 256, 0, stream, x, rows, k,
                          codes, scales);
}

cudaError_t launch_fp8_quantize_weight(const __nv_bfloat16* w, uint32_t experts, uint32_t rows, uint32_t k,
                                       uint8_t* codes, float* scales, cudaStream_t stream)
{
    const dim3 grid(k / 128, (rows + 127) / 128, experts);
    fp8_quantize_weight_kernel<<<grid, 256, 0, stream>>>(w, rows, k, codes, scales);
    note_launch();
    return cudaGetLastError();
}

cudaError_t launch_fp8_gemm(const Fp8Gemm& g, cudaStream_t stream, const char** why)
{
    const auto fail = [&](const char* msg) {
        if (why != nullptr)
            *why = msg;
        return cudaErrorNotSupported;
    };
    if (g.n % 128 != 0 || g.k % 128 != 0 || g.n == 0 || g.k == 0)
        return fail("FP8 GEMM needs n and k divisible by 128");
    if (g.k > 4096)
        return fail("FP8 GEMM supports k <= 4096");
    if (g.tile_rows != 64 && g.tile_rows != kTileM)
        return fail("FP8 GEMM token tiles are 64 or 128 rows");
    if ((reinterpret_cast<uintptr_t>(g.x) & 15u) != 0 || (reinterpret_cast<uintptr_t>(g.w) & 15u) != 0)
        return fail("FP8 GEMM operands must be 16-byte aligned");
    if (g.max_tiles == 0 || g.max_tiles > 65535)
        return fail("FP8 GEMM launch grid is too large");
    return g.tile_rows == kTileM ? launch_fp8_rows_gemm(g, stream, why) : launch_fp8_stream_gemm(g, stream, why);
}

} // namespace qs3
