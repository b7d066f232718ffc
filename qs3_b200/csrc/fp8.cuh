// Device-side FP8 (e4m3) quantiser: one f32 scale per 128 elements.
#pragma once

#include "common.cuh"
#include "nvfp4.cuh"

namespace qs3 {

__device__ __forceinline__ float fp8_scale_of(float amax)
{
    return fmaxf(__fdiv_rn(amax, 448.0f), 1.0e-30f);
}

__device__ __forceinline__ uint32_t pack_e4m3x4(const float* f, float inv)
{
    uint32_t r = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i)
        r |= static_cast<uint32_t>(f32_to_e4m3_sat(__fmul_rn(f[i], inv))) << (8 * i);
    return r;
}

// codes / scales of two 128-element groups of [rows, k] by a warp: 16 lanes per group, eight elements per lane. Rows and
// groups follow each other without gaps; `warp` numbers the pairs of groups.
__device__ __forceinline__ void fp8_quantize_groups(const __nv_bfloat16* __restrict__ x, uint32_t rows, uint32_t k,
                                                    uint8_t* __restrict__ codes, float* __restrict__ scales, uint64_t warp)
{
    const uint32_t groups = k / 128;
    const uint64_t unit = warp * 2 + (threadIdx.x >> 4 & 1);
    const uint32_t sub = threadIdx.x & 15;
    const bool live = unit < static_cast<uint64_t>(rows) * groups;
    const size_t at = static_cast<size_t>(unit) * 128 + sub * 8; // rows and groups follow each other without gaps
    uint2 v2[2] = { make_uint2(0, 0), make_uint2(0, 0) };
    if (live) { // (the entry points promise 8-byte aligned rows)
        const uint2* src = reinterpret_cast<const uint2*>(x + at);
        v2[0] = src[0];
        v2[1] = src[1];
    }
    const uint32_t w[4] = { v2[0].x, v2[0].y, v2[1].x, v2[1].y };
    float f[8];
    float amax = 0.0f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        f[2 * j] = bf16_bits_to_f32(w[j] & 0xffffu);
        f[2 * j + 1] = bf16_bits_to_f32(w[j] >> 16);
        amax = fmaxf(amax, fmaxf(fabsf(f[2 * j]), fabsf(f[2 * j + 1])));
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1)
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    if (!live)
        return;
    const float s = fp8_scale_of(amax);
    const float inv = __fdiv_rn(1.0f, s);
    uint32_t* dst = reinterpret_cast<uint32_t*>(codes + at);
    dst[0] = pack_e4m3x4(f, inv);
    dst[1] = pack_e4m3x4(f + 4, inv);
    if (sub == 0)
        scales[unit] = s;
}

} // namespace qs3
