// The routed (and shared) experts of a handful of tokens as matrix-vector products: two launches, gate_up and down +
// combine, instead of routing, two grouped GEMMs and a combine. Every (token, slot) streams its expert's weights by
// itself: with so few rows there is next to nothing to share, and what such a call waits for is the chain of dependent
// launches and table loads.
//
//   gate_up  persistent, two blocks per SM. Block 0 routes all tokens, writes ids and weights and sorts the routes into the
//            tables; every other block stages and quantises the tokens before the predecessor ends, routes them itself, a
//            warp per token, and takes units of 32 features of one slot, the shared expert's first, which do not wait.
//            (The down launch waits for all of them, block 0 among them, whose ids it reads; a combine reads its tables)
//   down     blocks (features, tokens), a warp per slot, then the weighted sum over the slots in shared memory, in
//            ascending order as the combine kernel adds them
//
//   nvfp4    a lane takes one 16-element block of four rows at a time; its products are summed in f16 eight at a time,
//            which is exact (multiples of 1/4 up to 288), and scaled in f32
//   fp8      16 rows by mma.sync m16n8k32, the token in one of its columns; 128 elements, then the scales
//   bf16     a lane takes 16 bytes of four rows at a time, f32
//
// Bound by latency for one token (three launches; routing, expert, weights, table after table), then by the weights, which
// arrive at 3 to 5 TB/s. Layer of one token over 512 experts top-10 + shared, NVFP4: 0.0368 -> 0.0229 ms a call, 0.0335 ->
// 0.0213 replayed from a graph, as are the following; 128 experts top-8, FP8: 0.0279 -> 0.0201, bf16 0.0351 -> 0.0215; 16
// tokens over 8 experts, 256 x 128, bf16: 0.0199 -> 0.0121 a call. Routing in every block of a grid (features, tokens)
// instead: 4 tokens NVFP4 0.052 against 0.043. Decoding e2m1 by byte permutation into
// e4m3 for mma.sync 0.0278, into f16 0.0265 against 0.0225 with the conversion instruction; e4m3 into f16 by shifts for
// mma.sync m16n8k16: FP8 0.0231 against 0.0180.
#include "nvfp4.cuh"
#include "route_sort.cuh"
#include "topk.cuh"

#include <cuda_fp16.h>

#include <algorithm>

namespace qs3 {
namespace {

constexpr uint32_t kGvWarps = kBlockSortWarps;
constexpr uint32_t kGvFeatures = 2 * kGvWarps; // of a gate_up block
constexpr uint32_t kGvXPitch = 48;             // bytes between a token's chunks of 32 in shared memory: no conflicts
constexpr uint32_t kGvMaxSlots = 17;
constexpr uint32_t kGvFewSlots = 12; // two down blocks per SM with 80 registers a thread instead of 56
constexpr uint32_t kGvMaxSmem = 96 * 1024;      // of a gate_up block's tokens: two blocks per SM
constexpr uint32_t kGvDefaultSmem = 40 * 1024; // with the kernel's own below 48 KB

template <int FMT> struct Gv {
    static constexpr uint32_t kOut = FMT == GEMV_FP8 ? 16 : 8;    // features of a down block
    static constexpr uint32_t kSplits = FMT == GEMV_FP8 ? 4 : 1; // of k, in a gate_up block
};

__device__ __forceinline__ uint4 load16(const void* p) { return __ldg(static_cast<const uint4*>(p)); }

// eight e2m1 codes -> four pairs of halves, in order
__device__ __forceinline__ void e2m1_to_f16(uint32_t w, uint32_t* h)
{
    asm("{\n\t.reg .b8 b0, b1, b2, b3;\n\t"
        "mov.b32 {b0, b1, b2, b3}, %4;\n\t"
        "cvt.rn.f16x2.e2m1x2 %0, b0;\n\t"
        "cvt.rn.f16x2.e2m1x2 %1, b1;\n\t"
        "cvt.rn.f16x2.e2m1x2 %2, b2;\n\t"
        "cvt.rn.f16x2.e2m1x2 %3, b3;\n\t}"
        : "=r"(h[0]), "=r"(h[1]), "=r"(h[2]), "=r"(h[3])
        : "r"(w));
}
// The same by byte permutation, for codes that this kernel has just packed (ptxas made zeros of cvt after cvt).
__device__ __forceinline__ void packed_e2m1_to_f16(uint32_t w, uint32_t* h)
{
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const uint32_t v = w >> (16 * i);
        uint32_t magnitude, sign; // upper bytes of 0 .5 1 1.5 2 3 4 6; a selector's bit 3 repeats the byte's top bit: 0xff
        asm("prmt.b32 %0, %1, %2, %3;" : "=r"(magnitude) : "r"(0x3e3c3800u), "r"(0x46444240u), "r"(v & 0x7777u));
        asm("prmt.b32 %0, %1, %1, %2;" : "=r"(sign) : "r"(0x80808080u), "r"(v));
        const uint32_t upper = magnitude | (sign << 1 & 0x80808080u);
        asm("prmt.b32 %0, %1, 0, 0x1404;" : "=r"(h[2 * i]) : "r"(upper));
        asm("prmt.b32 %0, %1, 0, 0x3424;" : "=r"(h[2 * i + 1]) : "r"(upper));
    }
}
__device__ __forceinline__ __half2 as_half2(uint32_t v) { return *reinterpret_cast<const __half2*>(&v); }

// Sum of a block of 16 e2m1 products: weights by code, token decoded.
__device__ __forceinline__ float dot_nvfp4(const uint2& w, const uint32_t (&x)[8])
{
    uint32_t h[8];
    e2m1_to_f16(w.x, h);
    e2m1_to_f16(w.y, h + 4);
    __half2 s = __hmul2(as_half2(h[0]), as_half2(x[0]));
#pragma unroll
    for (int i = 1; i < 8; ++i)
        s = __hfma2(as_half2(h[i]), as_half2(x[i]), s);
    return __low2float(s) + __high2float(s);
}
// The scale of a lane's block out of the word with those of four.
__device__ __forceinline__ float block_scale(uint32_t word) { return e4m3_to_f32(static_cast<uint8_t>(word >> (threadIdx.x % 4 * 8))); }

// c += a (16 rows, 32 k) . b (32 k, 8 columns). Lane (g, t) = (lane / 4, lane % 4): a0 / a1 rows g and g + 8, a2 / a3 the same
// rows' other 16 k; b0 / b1 column g; c0, c1 row g columns 2 t and 2 t + 1, c2, c3 row g + 8.
__device__ __forceinline__ void mma_e4m3(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1)
{
    asm("mma.sync.aligned.m16n8k32.row.col.f32.e4m3.e4m3.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// 128 elements of two FP8 rows (lane: bytes 16 t and 64 + 16 t onwards of rows g and g + 8) by one vector: `x` the same bytes
// of it in the lanes of column 0, zero in the others. The k positions of the instruction are permuted so that a lane's
// bytes are its fragments.
__device__ __forceinline__ void dot_fp8(float (&c)[4], const uint4 (&lo)[2], const uint4 (&hi)[2], const uint32_t (&x)[8])
{
    const uint32_t a[8] = { lo[0].x, lo[0].y, lo[0].z, lo[0].w, lo[1].x, lo[1].y, lo[1].z, lo[1].w };
    const uint32_t b[8] = { hi[0].x, hi[0].y, hi[0].z, hi[0].w, hi[1].x, hi[1].y, hi[1].z, hi[1].w };
#pragma unroll
    for (int s = 0; s < 4; ++s)
        mma_e4m3(c, a[2 * s], b[2 * s], a[2 * s + 1], b[2 * s + 1], x[2 * s], x[2 * s + 1]);
}
__device__ __forceinline__ void unpack_bf16x2(uint32_t w, float* f)
{
    f[0] = __uint_as_float(w << 16);
    f[1] = __uint_as_float(w & 0xffff0000u);
}

// acc + (eight bf16 weights . x)
__device__ __forceinline__ float dot_bf16(float acc, const uint4& w, const float (&x)[8])
{
    const uint32_t v[4] = { w.x, w.y, w.z, w.w };
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float f[2];
        unpack_bf16x2(v[i], f);
        acc = fmaf(f[0], x[2 * i], acc);
        acc = fmaf(f[1], x[2 * i + 1], acc);
    }
    return acc;
}

// Sums of four values over the warp: lane 8 i of the result holds value i.
__device__ __forceinline__ float reduce4(const float (&v)[4])
{
    const uint32_t lane = threadIdx.x & 31;
    const bool hi = lane & 16;
    const float a = (hi ? v[2] : v[0]) + __shfl_xor_sync(0xffffffffu, hi ? v[0] : v[2], 16);
    const float b = (hi ? v[3] : v[1]) + __shfl_xor_sync(0xffffffffu, hi ? v[1] : v[3], 16);
    const bool odd = lane & 8;
    float s = (odd ? b : a) + __shfl_xor_sync(0xffffffffu, odd ? a : b, 8);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1)
        s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}

// Four values of a 128-element group (the others are in the warp) -> their e4m3 codes, and the group's scale.
__device__ __forceinline__ uint32_t quantise_e4m3(const float (&f)[4], float* scale)
{
    const float m = fmaxf(fmaxf(fabsf(f[0]), fabsf(f[1])), fmaxf(fabsf(f[2]), fabsf(f[3])));
    const float amax = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(m)));
    const float s = fmaxf(__fdiv_rn(amax, 448.0f), 1.0e-30f), inv = __fdiv_rn(1.0f, s);
    uint32_t codes = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i)
        codes |= static_cast<uint32_t>(f32_to_e4m3_sat(__fmul_rn(f[i], inv))) << (8 * i);
    *scale = s;
    return codes;
}

// Bytes of a staged token, and where the scales are.
__host__ __device__ constexpr uint32_t token_bytes(int fmt, uint32_t hidden)
{
    return fmt == GEMV_FP8 ? hidden + (hidden / 128 * 4 + 15) / 16 * 16 // (16-byte vectors)
                           : fmt == GEMV_NVFP4 ? hidden / 16 * (kGvXPitch + 4) : hidden / 8 * kGvXPitch;
}
template <int FMT> __device__ __forceinline__ float* scales_of(uint8_t* s_x, uint32_t hidden)
{
    return reinterpret_cast<float*>(s_x + (FMT == GEMV_FP8 ? hidden : hidden / 16 * kGvXPitch));
}

// A token into shared memory: bf16 as floats and NVFP4's code values as halves, a chunk of 32 bytes at every kGvXPitch;
// FP8's codes; with the scales of its blocks.
template <int FMT>
__device__ __forceinline__ void stage_token(const GemvParams& p, uint32_t token, uint8_t* s_x)
{
    float* s_scale = scales_of<FMT>(s_x, p.hidden_size);
    const __nv_bfloat16* x = p.hidden + static_cast<size_t>(token) * p.hidden_size;
    if constexpr (FMT == GEMV_NVFP4) {
        for (uint32_t c = threadIdx.x; c < p.hidden_size / 16; c += blockDim.x) {
            uint32_t lo, hi, code, out[8];
            if (p.hidden_packed != nullptr) {
                const uint2 v = *reinterpret_cast<const uint2*>(p.hidden_packed + static_cast<size_t>(token) * (p.hidden_size / 2) + c * 8);
                lo = v.x, hi = v.y;
                code = p.hidden_sf[tiled_scale_offset(token, c, p.hidden_size / 64)];
            } else {
                float v[16];
                load16_bf16(x + c * 16, v);
                code = quantize_block16(v, p.act_global, &lo, &hi);
            }
            packed_e2m1_to_f16(lo, out);
            packed_e2m1_to_f16(hi, out + 4);
            uint4* dst = reinterpret_cast<uint4*>(s_x + c * kGvXPitch);
            dst[0] = make_uint4(out[0], out[1], out[2], out[3]);
            dst[1] = make_uint4(out[4], out[5], out[6], out[7]);
            s_scale[c] = e4m3_to_f32(static_cast<uint8_t>(code));
        }
    } else if constexpr (FMT == GEMV_FP8) { // a warp per 128 elements
        for (uint32_t kb = threadIdx.x / 32; kb < p.hidden_size / 128; kb += kGvWarps) {
            const uint2 v = reinterpret_cast<const uint2*>(x + kb * 128)[threadIdx.x % 32];
            float f[4];
            unpack_bf16x2(v.x, f);
            unpack_bf16x2(v.y, f + 2);
            float scale;
            reinterpret_cast<uint32_t*>(s_x)[kb * 32 + threadIdx.x % 32] = quantise_e4m3(f, &scale);
            s_scale[kb] = scale;
        }
    } else {
        for (uint32_t c = threadIdx.x; c < p.hidden_size / 8; c += blockDim.x) {
            const uint4 v = *reinterpret_cast<const uint4*>(x + c * 8);
            const uint32_t w[4] = { v.x, v.y, v.z, v.w };
            float4* dst = reinterpret_cast<float4*>(s_x + c * kGvXPitch);
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                float f[4];
                unpack_bf16x2(w[2 * i], f);
                unpack_bf16x2(w[2 * i + 1], f + 2);
                dst[i] = make_float4(f[0], f[1], f[2], f[3]);
            }
        }
    }
}

__device__ __forceinline__ uint64_t tiled_bytes(uint32_t rows, uint32_t k)
{
    return static_cast<uint64_t>((rows + 127) / 128) * (k / 64) * 512;
}

template <int FMT, int ITEMS> // ITEMS: experts per lane of the router; 0: ids and weights are given
__global__ void __launch_bounds__(kBlockSortThreads, 2)
gemv_gate_up_kernel(const GemvParams p, const RouterParams r, const RouteTables rt)
{
    using G = Gv<FMT>;
    extern __shared__ __align__(16) uint8_t s_dyn[];
    __shared__ uint32_t s_cand[ITEMS > 0 ? kGvWarps : 1][64];
    __shared__ int s_expert[kGvWarps * kGvMaxSlots]; // [tokens][top_k], local
    __shared__ float s_part[2][G::kSplits][kGvFeatures][2]; // gate and up sums over a part of k; two units in turn
    __shared__ float s_act[kGvFeatures];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t routes = p.num_tokens * p.top_k;

    if (blockIdx.x == 0) {
        chain_begin();
        const BlockSortSmem s = block_sort_carve(s_dyn, p.experts);
        if constexpr (ITEMS > 0) {
            if (warp < p.num_tokens) {
                int id;
                float weight;
                topk_row<float, ITEMS>(r.logits + static_cast<size_t>(warp) * r.num_experts, r.bias, r.num_experts, p.top_k,
                                       r.sigmoid_score, r.renormalize, r.scaling, s_cand[warp], &id, &weight);
                if (lane < p.top_k) {
                    const uint32_t route = warp * p.top_k + lane;
                    const int local = id - static_cast<int>(p.local_offset);
                    r.ids[route] = id;
                    r.weights[route] = weight;
                    s.ids[route] = static_cast<int16_t>(local < 0 || local >= static_cast<int>(p.experts) ? -1 : local);
                }
            }
        } else {
            for (uint32_t i = threadIdx.x; i < routes; i += kBlockSortThreads)
                s.ids[i] = static_cast<int16_t>(local_expert(p.ids, i, routes, p.local_offset, p.experts));
        }
        block_sort(s, ITEMS > 0 ? r.weights : p.weights, routes, p.top_k, p.experts, rt); // (starts with a barrier)
        return;
    }

    // units: the shared expert's features of all tokens, then the slots'; those before the first wait of a block are the
    // shared expert's only
    const uint32_t blocks = p.inter / kGvFeatures, per_token = blocks * p.num_tokens;
    const uint32_t units = (p.top_k + p.shared) * per_token;
    const uint32_t x_bytes = token_bytes(FMT, p.hidden_size);
    bool routed = false; // the experts are known
    if (!p.early)
        chain_begin();
    for (uint32_t i = 0; i < p.num_tokens; ++i)
        stage_token<FMT>(p, i, s_dyn + i * x_bytes);
    __syncthreads();
    uint32_t turn = 0;
    for (uint32_t unit = blockIdx.x - 1; unit < units; unit += gridDim.x - 1) {
        const bool shared = p.shared && unit < per_token;
        if (!shared && !routed) {
            routed = true;
            if (p.early)
                chain_begin();
            if constexpr (ITEMS > 0) {
                if (warp < p.num_tokens) {
                    int id;
                    float weight;
                    topk_row<float, ITEMS>(r.logits + static_cast<size_t>(warp) * r.num_experts, r.bias, r.num_experts, p.top_k,
                                           r.sigmoid_score, r.renormalize, r.scaling, s_cand[warp], &id, &weight);
                    if (lane < p.top_k)
                        s_expert[warp * p.top_k + lane] = id - static_cast<int>(p.local_offset);
                }
            } else {
                for (uint32_t i = threadIdx.x; i < routes; i += kBlockSortThreads)
                    s_expert[i] = p.ids[i] - static_cast<int>(p.local_offset);
            }
            __syncthreads();
        }
        const uint32_t fb = unit % blocks, token = unit / blocks % p.num_tokens;
        const uint32_t slot = shared ? p.top_k : unit / per_token - p.shared;
        const int expert = shared ? 0 : s_expert[token * p.top_k + slot];
        if (expert < 0 || (!shared && expert >= static_cast<int>(p.experts))) // (uniform)
            continue;
        turn ^= 1; // (the last unit's sums are still being read)
        uint8_t* s_x = s_dyn + token * x_bytes;
        const float* s_scale = scales_of<FMT>(s_x, p.hidden_size);

        const GemvWeights& w = shared ? p.shared_weights : p.routed;
        const uint32_t g = lane / 4, t = lane % 4;
        const uint32_t j64 = fb / 2, half = fb % 2; // NVFP4: features 16 half and 32 + 16 half onwards of a 64-feature block
        const size_t group_row = static_cast<size_t>(expert) * 2 * p.inter;
        if constexpr (FMT == GEMV_NVFP4) {
            // a warp: the gate rows r and r + 32 and the up rows r + 64 and r + 96 of the block's scale tile, whose scales of 64
            // elements are 16 bytes of it
            const uint32_t chunks = p.hidden_size / 16, r = half * 16 + warp;
            const size_t row_bytes = p.hidden_size / 2;
            const uint8_t* src = w.gate_up + (group_row + j64 * 64 + r) * row_bytes;
            const uint8_t* row[4];
#pragma unroll
            for (uint32_t q = 0; q < 4; ++q)
                row[q] = src + (static_cast<size_t>(q & 1) * 32 + static_cast<size_t>(q >> 1) * p.inter) * row_bytes;
            const uint8_t* sf = static_cast<const uint8_t*>(w.gate_up_scale) + expert * tiled_bytes(2 * p.inter, p.hidden_size)
                + static_cast<uint64_t>(j64) * (p.hidden_size / 64) * 512 + r * 16;
            float acc[4] = {};
            constexpr uint32_t kUnroll = 2;
            for (uint32_t c0 = lane; c0 < chunks; c0 += 32 * kUnroll) {
                uint2 v[kUnroll][4];
                uint4 sv[kUnroll];
#pragma unroll
                for (uint32_t u = 0; u < kUnroll; ++u) {
                    const uint32_t c = c0 + 32 * u;
                    if (c < chunks) {
#pragma unroll
                        for (uint32_t q = 0; q < 4; ++q)
                            v[u][q] = __ldg(reinterpret_cast<const uint2*>(row[q] + c * 8));
                        sv[u] = load16(sf + static_cast<size_t>(c / 4) * 512);
                    }
                }
#pragma unroll
                for (uint32_t u = 0; u < kUnroll; ++u) {
                    const uint32_t c = c0 + 32 * u;
                    if (c < chunks) {
                        const uint4* xp = reinterpret_cast<const uint4*>(s_x + c * kGvXPitch);
                        const uint4 x0 = xp[0], x1 = xp[1];
                        const uint32_t x[8] = { x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w };
                        const float xs = s_scale[c];
                        const uint32_t sw[4] = { sv[u].x, sv[u].y, sv[u].z, sv[u].w };
#pragma unroll
                        for (uint32_t q = 0; q < 4; ++q)
                            acc[q] = fmaf(dot_nvfp4(v[u][q], x), xs * block_scale(sw[q]), acc[q]);
                    }
                }
            }
            // lanes 0 and 8: gate of the two features, lanes 16 and 24: up
            const float sum = reduce4(acc);
            if (lane % 8 == 0)
                s_part[turn][0][(lane / 8 & 1) * 16 + warp][lane / 16] = sum;
        } else if constexpr (FMT == GEMV_FP8) {
            const uint32_t split = warp / 4, kbs = p.hidden_size / 128, rbs = p.inter / 128;
            const uint32_t f = fb * kGvFeatures + warp % 4 * 8 + g;
            const size_t row_bytes = p.hidden_size, up = static_cast<size_t>(p.inter) * row_bytes;
            const uint8_t* src = w.gate_up + (group_row + f) * row_bytes + t * 16;
            const float* ws0 = static_cast<const float*>(w.gate_up_scale) + (static_cast<size_t>(expert) * 2 * rbs + f / 128) * kbs;
            const float* ws1 = ws0 + static_cast<size_t>(rbs) * kbs;
            float acc[2] = {};
#pragma unroll 1
            for (uint32_t kb = split; kb < kbs; kb += G::kSplits) {
                uint4 gate[2], upw[2];
#pragma unroll
                for (uint32_t q = 0; q < 2; ++q) {
                    gate[q] = load16(src + kb * 128 + q * 64);
                    upw[q] = load16(src + up + kb * 128 + q * 64);
                }
                const float s0 = __ldg(ws0 + kb), s1 = __ldg(ws1 + kb), xs = s_scale[kb];
                uint32_t x[8] = {};
                if (g == 0) {
                    const uint4* xp = reinterpret_cast<const uint4*>(s_x) + kb * 8 + t;
                    const uint4 x0 = xp[0], x1 = xp[4];
                    x[0] = x0.x, x[1] = x0.y, x[2] = x0.z, x[3] = x0.w, x[4] = x1.x, x[5] = x1.y, x[6] = x1.z, x[7] = x1.w;
                }
                float c[4] = {};
                dot_fp8(c, gate, upw, x);
                acc[0] = fmaf(c[0], s0 * xs, acc[0]); // (column 0: lanes t = 0)
                acc[1] = fmaf(c[2], s1 * xs, acc[1]);
            }
            if (t == 0) {
                s_part[turn][split][warp % 4 * 8 + g][0] = acc[0];
                s_part[turn][split][warp % 4 * 8 + g][1] = acc[1];
            }
        } else { // a warp: the gate and up rows of features `warp` and `warp` + 16
            const uint32_t chunks = p.hidden_size / 8;
            const __nv_bfloat16* src = reinterpret_cast<const __nv_bfloat16*>(w.gate_up) + (group_row + fb * kGvFeatures + warp) * p.hidden_size;
            const __nv_bfloat16* row[4];
#pragma unroll
            for (uint32_t q = 0; q < 4; ++q)
                row[q] = src + (static_cast<size_t>(q & 1) * 16 + static_cast<size_t>(q >> 1) * p.inter) * p.hidden_size;
            float acc[4] = {};
            constexpr uint32_t kUnroll = 2;
            for (uint32_t c0 = lane; c0 < chunks; c0 += 32 * kUnroll) {
                uint4 v[kUnroll][4];
#pragma unroll
                for (uint32_t u = 0; u < kUnroll; ++u)
                    if (c0 + 32 * u < chunks)
#pragma unroll
                        for (uint32_t q = 0; q < 4; ++q)
                            v[u][q] = load16(row[q] + (c0 + 32 * u) * 8);
#pragma unroll
                for (uint32_t u = 0; u < kUnroll; ++u) {
                    if (c0 + 32 * u < chunks) {
                        const float4* xp = reinterpret_cast<const float4*>(s_x + (c0 + 32 * u) * kGvXPitch);
                        const float4 x0 = xp[0], x1 = xp[1];
                        const float x[8] = { x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w };
#pragma unroll
                        for (uint32_t q = 0; q < 4; ++q)
                            acc[q] = dot_bf16(acc[q], v[u][q], x);
                    }
                }
            }
            // lanes 0 and 8: gate of the two features, lanes 16 and 24: up
            const float sum = reduce4(acc);
            if (lane % 8 == 0)
                s_part[turn][0][(lane / 8 & 1) * 16 + warp][lane / 16] = sum;
        }
        __syncthreads();

        if (warp == 0) { // a lane per feature: of an NVFP4 block, 16 neighbouring ones twice
            const size_t act_row = static_cast<size_t>(token) * (p.top_k + p.shared) + slot;
            float gv = s_part[turn][0][lane][0], uv = s_part[turn][0][lane][1];
#pragma unroll
            for (uint32_t s = 1; s < G::kSplits; ++s) {
                gv += s_part[turn][s][lane][0];
                uv += s_part[turn][s][lane][1];
            }
            if constexpr (FMT == GEMV_BF16) {
                gv = __bfloat162float(__float2bfloat16(gv));
                uv = __bfloat162float(__float2bfloat16(uv));
                reinterpret_cast<__nv_bfloat16*>(p.act)[act_row * p.inter + fb * kGvFeatures + lane]
                    = __float2bfloat16(gv * sigmoid_fast(gv) * uv);
            } else if constexpr (FMT == GEMV_FP8) {
                reinterpret_cast<float*>(p.act)[act_row * p.inter + fb * kGvFeatures + lane] = __fdividef(gv, 1.0f + __expf(-gv)) * uv;
            } else {
                float scale = p.act_global, scale_up = p.act_global;
                if (w.gate_up_global != nullptr)
                    scale *= w.gate_up_global[expert];
                scale_up *= w.gate_up_global_up != nullptr ? w.gate_up_global_up[expert]
                                                           : (w.gate_up_global != nullptr ? w.gate_up_global[expert] : 1.0f);
                gv *= scale;
                uv *= scale_up;
                s_act[lane] = __fdividef(gv, 1.0f + __expf(-gv)) * uv;
                __syncwarp();
                if (lane < 2) { // the block's features are two 16-element blocks of the next product
                    uint32_t lo, hi;
                    const uint32_t blk = j64 * 4 + lane * 2 + half;
                    const uint8_t code = quantize_block16(s_act + lane * 16, p.act2_global, &lo, &hi);
                    *reinterpret_cast<uint2*>(p.act + act_row * (p.inter / 2) + blk * 8) = make_uint2(lo, hi);
                    p.act_scale[act_row * (p.inter / 16) + blk] = code;
                }
                __syncwarp();
            }
        }
    }
    if (p.early && !routed)
        chain_begin();
}

template <int FMT, uint32_t SLOTS> // at most that many
__global__ void __launch_bounds__(SLOTS * 32, 2) gemv_down_kernel(const GemvParams p)
{
    constexpr uint32_t kOut = Gv<FMT>::kOut;
    __shared__ float s_y[kGvMaxSlots][kOut];
    __shared__ float s_dot[kGvMaxSlots];
    __shared__ float s_weight[kGvMaxSlots]; // routing weight
    __shared__ int s_valid[kGvMaxSlots];
    const uint32_t slot = threadIdx.x >> 5, lane = threadIdx.x & 31, token = blockIdx.y;
    const uint32_t slots = p.top_k + p.shared;
    const bool shared = slot == p.top_k;
    const bool combine = p.y2 == nullptr;
    if (p.shared && combine) {
        // gate logit of the shared expert (hidden and gate weight are older than the predecessor)
        const uint4* x = reinterpret_cast<const uint4*>(p.hidden + static_cast<size_t>(token) * p.hidden_size);
        const uint4* w = reinterpret_cast<const uint4*>(p.shared_gate);
        float dot = 0.0f;
        for (uint32_t i = threadIdx.x; i < p.hidden_size / 8; i += blockDim.x) {
            const uint4 xv = x[i], wv = w[i];
            const uint32_t xs[4] = { xv.x, xv.y, xv.z, xv.w }, ws[4] = { wv.x, wv.y, wv.z, wv.w };
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                float a[2], b[2];
                unpack_bf16x2(xs[j], a);
                unpack_bf16x2(ws[j], b);
                dot += a[0] * b[0];
                dot += a[1] * b[1];
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            dot += __shfl_xor_sync(0xffffffffu, dot, o);
        if (lane == 0)
            s_dot[slot] = dot;
    }
    chain_begin();
    int expert = 0;
    float weight = 0.0f;
    if (!shared) {
        expert = p.ids[token * p.top_k + slot] - static_cast<int>(p.local_offset);
        weight = p.weights[token * p.top_k + slot];
    }
    const bool valid = expert >= 0 && expert < static_cast<int>(p.experts);
    // The block's features: bf16 and FP8 kOut in a row; NVFP4 two in a row and those 32, 64 and 96 further on, whose scales
    // of 64 elements lie side by side in the scale tile.
    const uint32_t f0 = FMT == GEMV_NVFP4 ? blockIdx.x / 16 * 128 + blockIdx.x % 16 * 2 : blockIdx.x * kOut;
    const auto feature = [&](uint32_t i) { return FMT == GEMV_NVFP4 ? f0 + i / 4 + i % 4 * 32 : f0 + i; };
    if (valid) {
        const GemvWeights& w = shared ? p.shared_weights : p.routed;
        const uint32_t g = lane / 4, t = lane % 4;
        const size_t act_row = static_cast<size_t>(token) * slots + slot;
        const size_t row0 = static_cast<size_t>(expert) * p.hidden_size;
        float y[kOut / 4]; // lanes 0, 8, 16, 24: features 4 i .. 4 i + 3; FP8: lanes t = 0, features g and g + 8
        if constexpr (FMT == GEMV_NVFP4) {
            const uint32_t chunks = p.inter / 16;
            const size_t row_bytes = p.inter / 2;
            const uint8_t* src = w.down + (row0 + f0) * row_bytes;
            const uint8_t* sf = static_cast<const uint8_t*>(w.down_scale) + expert * tiled_bytes(p.hidden_size, p.inter)
                + static_cast<uint64_t>(f0 / 128) * (p.inter / 64) * 512 + (f0 % 128) * 16;
            float acc[kOut / 4][4] = {};
            for (uint32_t c = lane; c < chunks; c += 32) {
                uint2 v[kOut / 4][4];
                uint4 sv[kOut / 4];
#pragma unroll
                for (uint32_t i = 0; i < kOut / 4; ++i) {
#pragma unroll
                    for (uint32_t q = 0; q < 4; ++q)
                        v[i][q] = __ldg(reinterpret_cast<const uint2*>(src + (i + q * 32) * row_bytes + c * 8));
                    sv[i] = load16(sf + static_cast<size_t>(c / 4) * 512 + i * 16);
                }
                const uint2 codes = *reinterpret_cast<const uint2*>(p.act + act_row * (p.inter / 2) + c * 8);
                uint32_t x[8];
                e2m1_to_f16(codes.x, x);
                e2m1_to_f16(codes.y, x + 4);
                const float xs = e4m3_to_f32(p.act_scale[act_row * (p.inter / 16) + c]);
#pragma unroll
                for (uint32_t i = 0; i < kOut / 4; ++i) {
                    const uint32_t sw[4] = { sv[i].x, sv[i].y, sv[i].z, sv[i].w };
#pragma unroll
                    for (uint32_t q = 0; q < 4; ++q)
                        acc[i][q] = fmaf(dot_nvfp4(v[i][q], x), xs * block_scale(sw[q]), acc[i][q]);
                }
            }
            float scale = p.act2_global;
            if (w.down_global != nullptr)
                scale *= w.down_global[expert];
#pragma unroll
            for (uint32_t i = 0; i < kOut / 4; ++i)
                y[i] = reduce4(acc[i]) * scale;
        } else if constexpr (FMT == GEMV_FP8) {
            const size_t row_bytes = p.inter;
            const uint32_t kbs = p.inter / 128;
            const uint8_t* src = w.down + (row0 + f0 + g) * row_bytes + t * 16;
            const float* ws = static_cast<const float*>(w.down_scale)
                + (static_cast<size_t>(expert) * (p.hidden_size / 128) + f0 / 128) * kbs;
            const float4* act = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(p.act) + act_row * p.inter);
            y[0] = y[1] = 0.0f;
            constexpr uint32_t kAhead = SLOTS <= kGvFewSlots ? 3 : 1;
#pragma unroll kAhead
            for (uint32_t kb = 0; kb < kbs; ++kb) {
                uint4 lo[2], hi[2];
#pragma unroll
                for (uint32_t q = 0; q < 2; ++q) {
                    lo[q] = load16(src + kb * 128 + q * 64);
                    hi[q] = load16(src + 8 * row_bytes + kb * 128 + q * 64);
                }
                const float4 v = act[kb * 32 + lane];
                const float f[4] = { v.x, v.y, v.z, v.w };
                float xs;
                const uint32_t codes = quantise_e4m3(f, &xs);
                uint32_t x[8];
#pragma unroll
                for (uint32_t i = 0; i < 8; ++i) {
                    const uint32_t word = __shfl_sync(0xffffffffu, codes, i / 4 * 16 + t * 4 + i % 4);
                    x[i] = g == 0 ? word : 0u;
                }
                const float s = __ldg(ws + kb) * xs;
                float c[4] = {};
                dot_fp8(c, lo, hi, x);
                y[0] = fmaf(c[0], s, y[0]);
                y[1] = fmaf(c[2], s, y[1]);
            }
        } else {
            const uint32_t chunks = p.inter / 8;
            const __nv_bfloat16* src = reinterpret_cast<const __nv_bfloat16*>(w.down) + (row0 + f0) * p.inter;
            const uint4* act = reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(p.act) + act_row * p.inter);
            float acc[2][4] = {};
            for (uint32_t c = lane; c < chunks; c += 32) {
                uint4 v[8];
#pragma unroll
                for (uint32_t q = 0; q < 8; ++q)
                    v[q] = load16(src + static_cast<size_t>(q) * p.inter + c * 8);
                const uint4 a = act[c];
                const uint32_t aw[4] = { a.x, a.y, a.z, a.w };
                float x[8];
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    unpack_bf16x2(aw[i], x + 2 * i);
#pragma unroll
                for (uint32_t q = 0; q < 8; ++q)
                    acc[q / 4][q % 4] = dot_bf16(acc[q / 4][q % 4], v[q], x);
            }
            y[0] = reduce4(acc[0]);
            y[1] = reduce4(acc[1]);
        }
        if (FMT == GEMV_FP8 ? t == 0 : lane % 8 == 0) {
#pragma unroll
            for (uint32_t i = 0; i < (FMT == GEMV_FP8 ? 2 : kOut / 4); ++i) {
                const uint32_t at = FMT == GEMV_FP8 ? i * 8 + g : i * 4 + lane / 8;
                const __nv_bfloat16 v = __float2bfloat16(y[i]);
                if (combine) {
                    s_y[slot][at] = __bfloat162float(v);
                } else {
                    const size_t row = !shared ? static_cast<size_t>(p.route_prows[token * p.top_k + slot])
                        : token + (p.shared_row0 != nullptr ? static_cast<size_t>(*p.shared_row0) : 0);
                    (shared ? p.y2_shared : p.y2)[row * p.hidden_size + feature(at)] = v;
                }
            }
        }
    }
    if (!combine)
        return;
    if (lane == 0) {
        s_weight[slot] = weight;
        s_valid[slot] = valid;
    }
    __syncthreads();
    if (threadIdx.x < kOut) {
        float sum = 0.0f;
        for (uint32_t k = 0; k < p.top_k; ++k)
            if (s_valid[k]) // a skipped route adds nothing (not even a signed zero)
                sum += s_weight[k] * s_y[k][threadIdx.x];
        if (p.shared) {
            float dot = 0.0f;
            for (uint32_t w = 0; w < slots; ++w)
                dot += s_dot[w];
            if (FMT == GEMV_BF16)
                sum = __bfloat162float(__float2bfloat16(sum));
            sum = sum + sigmoid_fast(dot) * s_y[p.top_k][threadIdx.x];
        }
        p.out[static_cast<size_t>(token) * p.hidden_size + feature(threadIdx.x)] = __float2bfloat16(sum);
    }
}

template <int FMT>
cudaError_t launch_instance(const GemvParams& p, const RouterParams* router, const RouteTables& rt, cudaStream_t stream)
{
    const uint32_t slots = p.top_k + p.shared;
    const size_t smem = std::max<size_t>(block_sort_smem(p.experts), static_cast<size_t>(p.num_tokens) * token_bytes(FMT, p.hidden_size));
    auto kernel = gemv_gate_up_kernel<FMT, 16>;
    if (router != nullptr) {
        const uint32_t per_lane = (router->num_experts + 31) / 32;
        if (per_lane <= 8)
            kernel = per_lane <= 1 ? gemv_gate_up_kernel<FMT, 1> : per_lane <= 4 ? gemv_gate_up_kernel<FMT, 4> : gemv_gate_up_kernel<FMT, 8>;
    } else if constexpr (FMT == GEMV_BF16) {
        kernel = gemv_gate_up_kernel<FMT, 0>;
    } else {
        return cudaErrorNotSupported; // (no entry point gives ids with a bf16 token)
    }
    if (smem > kGvDefaultSmem) {
        const cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kGvMaxSmem);
        if (err != cudaSuccess)
            return err;
    }
    const cudaError_t err = launch_chained(kernel, dim3(1 + std::min(slots * (p.inter / kGvFeatures) * p.num_tokens, 2 * device_sm_count() - 1)),
                                           kBlockSortThreads, smem, stream, p, router != nullptr ? *router : RouterParams {}, rt);
    if (err != cudaSuccess)
        return err;
    stage_mark(stream, STAGE_DOWN_GEMM);
    return launch_chained(slots <= kGvFewSlots ? gemv_down_kernel<FMT, kGvFewSlots> : gemv_down_kernel<FMT, kGvMaxSlots>,
                          dim3(p.hidden_size / Gv<FMT>::kOut, p.num_tokens), slots * 32, 0, stream, p);
}

// Where the products win. Their time grows with the weights that the slots multiply, again for every slot of one expert, with
// the rows of a slot (more of them for the same weights where hidden is small), and with the tokens and experts that every
// block routes; the grouped GEMMs stream an expert once, over five launches, and are quickest with a skewed router. The cost
// is in millions of weights; the limits are where, over 125 shapes (hidden 256..4096, 4..512 experts top-1..16, intermediate
// 128..1536, with and without a shared expert, even and skewed router, 1..16 tokens), the first calls come out slower
// than they were before these products: of the 1698 taken three are, by 3 to 4 %. By the weights alone, up to 110, 115 and
// 140 million, and fewer where the experts have several routes each, 78 of 1848 were, by 3 to 56 %
// (layer of 12 tokens, 128 experts top-8, 256 x 1024, FP8: 23.6 us grouped, 36.7 this; 8 tokens, 512 experts top-10, 2048 x
// 256, bf16: 37.9 and 54.9; 16 tokens, 128 experts top-4, 512 x 768, NVFP4: 25.7 and 34.0). Layer (hidden, experts top-k,
// intermediate; tokens: grouped / this, us; of a skewed router in brackets):
//                              bf16                            nvfp4                          fp8
//   2048, 128 top-8, 768       3: 48 / 42 (39 / 34),                                          3: 35 / 31 (28 / 28),
//                              4: 59 / 54 (41 / 43)                                           4: 41 / 43 (29 / 37)
//   2048, 512 top-10, 512 + 1  3: 54 / 55 (49 / 46),           2: 32 / 28 (31 / 27),
//                              4: 72 / 71 (51 / 55)            3: 34 / 35 (31 / 33)
struct GemvCost {
    float rows, slot, token, experts, most; // of a thousand intermediate features of a slot, a slot, a token, a hundred experts
};
constexpr GemvCost kGvCost[] = { { 2, 2, 4, 0, 220 }, { 3, 1, 4, 10, 220 }, { 3, 0.5f, 6, 0, 180 } }; // by GemvFormat
bool gemv_pays(int fmt, uint32_t tokens, uint32_t slots, uint32_t experts, uint32_t hidden, uint32_t inter)
{
    const GemvCost& c = kGvCost[fmt];
    const float rows = 1e-3f * static_cast<float>(slots) * static_cast<float>(inter);
    return rows * (3e-3f * static_cast<float>(hidden) + c.rows) + c.slot * slots + c.token * tokens + c.experts * 0.01f * experts <= c.most;
}

} // namespace

bool gemv_supported(int fmt, uint32_t num_tokens, uint32_t top_k, uint32_t num_experts, uint32_t experts, uint32_t hidden,
                    uint32_t inter, uint32_t shared_inter)
{
    // whole blocks of features; the tokens in shared memory; a warp per slot; one router block
    return inter % kGvFeatures == 0 && hidden % 128 == 0 && hidden <= 65536 && num_tokens * token_bytes(fmt, hidden) <= kGvMaxSmem
        && top_k + 1 <= kGvMaxSlots && num_tokens <= kGvWarps
        && (shared_inter == 0 || shared_inter == inter) && router_sort_supported(num_tokens, num_experts, top_k, experts)
        && (fmt == GEMV_BF16 || inter % 128 == 0)
        && (fmt != GEMV_FP8 || (hidden <= 4096 && inter <= 4096)) // (as far as FP8 plans go: larger batches are refused beyond)
        && gemv_pays(fmt, num_tokens, num_tokens * (top_k + (shared_inter != 0)), num_experts, hidden, inter);
}

cudaError_t launch_gemv(int fmt, const GemvParams& p, const RouterParams* router, const RouteTables& rt, cudaStream_t stream)
{
    return fmt == GEMV_NVFP4 ? launch_instance<GEMV_NVFP4>(p, router, rt, stream)
        : fmt == GEMV_FP8    ? launch_instance<GEMV_FP8>(p, router, rt, stream)
                             : launch_instance<GEMV_BF16>(p, router, rt, stream);
}

} // namespace qs3
