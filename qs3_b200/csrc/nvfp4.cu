// NVFP4 quantisers and scale-layout kernels: weight preparation (the layout the
// upstream weight loader never produced, src/weight_loader.rs:33-66), activation
// quantisation in token order, the gather of its codes by expert, and linear -> tiled scale re-tiling.
#include "common.cuh"
#include "nvfp4.cuh"

#include <cooperative_groups.h>

#include <algorithm>
#include <utility>

namespace qs3 {

namespace {

// Weight quantisation in ONE launch: a cluster of kQwCluster blocks per expert finds the expert's amax
// (pass 1, exchanged through distributed shared memory) and then quantises it (pass 2, whose reads come
// from L2: about seventeen experts are in flight, 70 MB for 4-MB gate_up experts, against 126 MB of L2).
// 2 bytes in, 0.63 bytes out per weight; bound by its two passes taking turns: all clusters read HBM first, then L2 and
// compute, and clusters of 16 leave SMs out (active for 83 % of the busiest one's cycles, some for none). Of the rest half the
// issue slots are taken, 26 of 64 warps resident, HBM at 38 %. Separate amax / finish / quantise kernels read the
// weights twice from HBM and sent every warp's amax to one address per expert; 64 experts of 1024 x 2048:
// 0.453 -> 0.108 ms (3.3 TB/s); half the arithmetic of pass 2 changed nothing.
constexpr uint32_t kQwCluster = 16;
constexpr uint32_t kQwThreads = 512;
constexpr uint32_t kQwChunk = 512;   // k elements of one unit of pass 2: a 16-element block per lane
constexpr uint32_t kQwPitch = 36;    // bytes per row of the scale staging (odd word count: no bank conflicts)

__device__ __forceinline__ float global_scale_of(float amax) { return amax > 0.0f ? __fdiv_rn(amax, 6.0f * 448.0f) : 1.0f; }

// Units of 128 tiled rows x kQwChunk elements of expert `e`, every `step`-th from `first`; a warp takes eight rows, a lane one
// block of a row. `s_code` is 128 * kQwPitch bytes of shared memory.
__device__ __forceinline__ void quantize_units(const __nv_bfloat16* __restrict__ w, uint32_t e, uint32_t rows, uint32_t k, float g,
                                               uint8_t* __restrict__ packed, uint8_t* __restrict__ scale_linear,
                                               uint8_t* __restrict__ scale_tiled, uint64_t tiled_bytes, int gated,
                                               uint32_t first, uint32_t step, uint8_t* s_code)
{
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t kb_per_row = k / 16, kgroups = k / 64;
    const uint32_t k_chunks = (k + kQwChunk - 1) / kQwChunk;
    const uint32_t units = (rows + 127) / 128 * k_chunks;
    for (uint32_t unit = first; unit < units; unit += step) {
        const uint32_t rb = unit / k_chunks, kc = unit % k_chunks;
        const uint32_t kb = kc * (kQwChunk / 16) + lane;
        constexpr uint32_t kRows = 128 / (kQwThreads / 32);
#pragma unroll
        for (uint32_t i0 = 0; i0 < kRows; i0 += 4) {
            uint4 va[4], vb[4];
            uint64_t grow[4];
            bool live[4];
#pragma unroll
            for (uint32_t q = 0; q < 4; ++q) {
                const uint32_t tr = warp + (i0 + q) * (kQwThreads / 32); // row of the tile
                const uint32_t row = gated ? rb * 64 + (tr & 63) + (tr >= 64 ? rows / 2 : 0) : rb * 128 + tr;
                live[q] = row < rows && kb < kb_per_row;
                grow[q] = static_cast<uint64_t>(e) * rows + row;
                const uint4* p = reinterpret_cast<const uint4*>(w + grow[q] * k + static_cast<uint64_t>(kb) * 16);
                va[q] = live[q] ? p[0] : make_uint4(0, 0, 0, 0);
                vb[q] = live[q] ? p[1] : make_uint4(0, 0, 0, 0);
            }
#pragma unroll
            for (uint32_t q = 0; q < 4; ++q) {
                float x[16];
                unpack16_bf16(va[q], vb[q], x);
                const __nv_bfloat162 zero = __floats2bfloat162_rn(0.0f, 0.0f);
                const float block_amax = bf16x2_max(bf16x2_amax(bf16x2_amax(zero, va[q]), vb[q]));
                uint32_t lo, hi;
                const uint8_t code = quantize_block16(x, block_amax, g, &lo, &hi);
                if (live[q]) {
                    *reinterpret_cast<uint2*>(packed + grow[q] * (k / 2) + static_cast<uint64_t>(kb) * 8) = make_uint2(lo, hi);
                    if (scale_linear != nullptr)
                        scale_linear[grow[q] * kb_per_row + kb] = code;
                }
                s_code[(warp + (i0 + q) * (kQwThreads / 32)) * kQwPitch + lane] = live[q] ? code : 0;
            }
        }
        __syncthreads();
        if (scale_tiled != nullptr && threadIdx.x < 256) {
            // thread = (k group, lane of the scale tile): rows lane, lane + 32, lane + 64, lane + 96
            const uint32_t kg = kc * (kQwChunk / 64) + warp;
            if (kg < kgroups) {
                uint32_t word[4];
#pragma unroll
                for (uint32_t q = 0; q < 4; ++q)
                    word[q] = *reinterpret_cast<const uint32_t*>(s_code + (lane + 32 * q) * kQwPitch + warp * 4);
                *reinterpret_cast<uint4*>(scale_tiled + static_cast<uint64_t>(e) * tiled_bytes
                                          + (static_cast<uint64_t>(rb) * kgroups + kg) * 512 + lane * 16)
                    = make_uint4(word[0], word[1], word[2], word[3]);
            }
        }
        __syncthreads(); // the staging is reused by the next unit
    }
}

__global__ void __launch_bounds__(kQwThreads, 2)
quantize_weight_kernel(const __nv_bfloat16* __restrict__ w, uint32_t rows, uint32_t k, float* __restrict__ global_scale,
                       uint8_t* __restrict__ packed, uint8_t* __restrict__ scale_linear,
                       uint8_t* __restrict__ scale_tiled, uint64_t tiled_bytes, int gated)
{
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    // a block's shared memory may be written by a peer only once the block runs: awaited before the exchange, behind pass 1
    auto started = cluster.barrier_arrive();
    const uint32_t rank = cluster.block_rank();
    const uint32_t e = blockIdx.x / kQwCluster;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __shared__ float s_part[kQwThreads / 32];
    __shared__ float s_amax[kQwCluster];
    __shared__ __align__(16) uint8_t s_code[128 * kQwPitch];

    // pass 1: amax of the expert
    const uint64_t per_expert = static_cast<uint64_t>(rows) * k;
    const uint4* src = reinterpret_cast<const uint4*>(w + static_cast<uint64_t>(e) * per_expert);
    const uint64_t vecs = per_expert / 8;
    constexpr uint64_t kStep = static_cast<uint64_t>(kQwCluster) * kQwThreads;
    __nv_bfloat162 m2 = __floats2bfloat162_rn(0.0f, 0.0f);
    for (uint64_t i0 = static_cast<uint64_t>(rank) * kQwThreads + threadIdx.x; i0 < vecs; i0 += 4 * kStep) {
        uint4 v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q)
            v[q] = i0 + q * kStep < vecs ? src[i0 + q * kStep] : make_uint4(0, 0, 0, 0);
#pragma unroll
        for (int q = 0; q < 4; ++q)
            m2 = bf16x2_amax(m2, v[q]);
    }
    float m = bf16x2_max(m2);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (lane == 0)
        s_part[warp] = m;
    __syncthreads();
    cluster.barrier_wait(std::move(started));
    if (warp == 0) {
        m = lane < kQwThreads / 32 ? s_part[lane] : 0.0f;
#pragma unroll
        for (int o = 8; o > 0; o >>= 1)
            m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        m = __shfl_sync(0xffffffffu, m, 0);
        if (lane < kQwCluster) // this block's amax into slot `rank` of block `lane`
            *cluster.map_shared_rank(&s_amax[rank], lane) = m;
    }
    cluster.sync();
    float amax = 0.0f;
#pragma unroll
    for (uint32_t r = 0; r < kQwCluster; ++r)
        amax = fmaxf(amax, s_amax[r]);
    const float g = global_scale_of(amax);
    if (rank == 0 && threadIdx.x == 0)
        global_scale[e] = g;

    // pass 2
    quantize_units(w, e, rows, k, g, packed, scale_linear, scale_tiled, tiled_bytes, gated, rank, kQwCluster, s_code);
}

// The same over the whole grid, blockIdx.y = expert, for experts too few and too large for their clusters: bound by HBM, 1 x
// 32768 x 2048 0.401 -> 0.063 ms (3.5 TB/s; the second pass comes from L2 where the weights fit it).
// amax_bits[e] = bits of the expert's amax (non-negative floats order like their bit patterns), zeroed before.
__global__ void __launch_bounds__(kQwThreads)
expert_amax_kernel(const __nv_bfloat16* __restrict__ w, uint64_t per_expert, uint32_t* __restrict__ amax_bits)
{
    const uint4* src = reinterpret_cast<const uint4*>(w + blockIdx.y * per_expert);
    const uint64_t vecs = per_expert / 8, step = static_cast<uint64_t>(gridDim.x) * kQwThreads;
    __nv_bfloat162 m2 = __floats2bfloat162_rn(0.0f, 0.0f);
    for (uint64_t i0 = static_cast<uint64_t>(blockIdx.x) * kQwThreads + threadIdx.x; i0 < vecs; i0 += 4 * step) {
        uint4 v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q)
            v[q] = i0 + q * step < vecs ? src[i0 + q * step] : make_uint4(0, 0, 0, 0);
#pragma unroll
        for (int q = 0; q < 4; ++q)
            m2 = bf16x2_amax(m2, v[q]);
    }
    const uint32_t m = __reduce_max_sync(0xffffffffu, __float_as_uint(bf16x2_max(m2)));
    __shared__ uint32_t s_part[kQwThreads / 32];
    if ((threadIdx.x & 31) == 0)
        s_part[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x < 32) {
        const uint32_t all = __reduce_max_sync(0xffffffffu, threadIdx.x < kQwThreads / 32 ? s_part[threadIdx.x] : 0u);
        if (threadIdx.x == 0)
            atomicMax(amax_bits + blockIdx.y, all);
    }
}

__global__ void finish_global_scale_kernel(float* scale, uint32_t experts)
{
    const uint32_t e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e < experts)
        scale[e] = global_scale_of(scale[e]);
}

__global__ void __launch_bounds__(kQwThreads, 2)
quantize_weight_flat_kernel(const __nv_bfloat16* __restrict__ w, uint32_t rows, uint32_t k, const float* __restrict__ global_scale,
                            uint8_t* __restrict__ packed, uint8_t* __restrict__ scale_linear,
                            uint8_t* __restrict__ scale_tiled, uint64_t tiled_bytes, int gated)
{
    __shared__ __align__(16) uint8_t s_code[128 * kQwPitch];
    quantize_units(w, blockIdx.y, rows, k, global_scale[blockIdx.y], packed, scale_linear, scale_tiled, tiled_bytes, gated,
                   blockIdx.x, gridDim.x, s_code);
}

// Activation rows to the declared (linear) layout; one thread per block.
__global__ void quantize_act_linear_kernel(const __nv_bfloat16* __restrict__ x, uint32_t k,
                                           uint64_t total_blocks, float g, uint8_t* __restrict__ packed,
                                           uint8_t* __restrict__ scale_linear)
{
    const uint64_t idx = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (idx >= total_blocks)
        return;
    float v[16];
    load16_bf16(x + idx * 16, v);
    uint32_t lo, hi;
    const uint8_t code = quantize_block16(v, g, &lo, &hi);
    *reinterpret_cast<uint2*>(packed + idx * 8) = make_uint2(lo, hi);
    scale_linear[idx] = code;
}

// Token rows, in token order, to codes and tiled scales (quantize_row_chunk). A warp takes 512 elements of one row, a lane one
// 16-element block: a load instruction covers contiguous sectors and four neighbouring lanes share the 32-bit
// scale word of a 64-element group (a thread per group read with a 128-byte stride between lanes). Bound by
// HBM (2 bytes in, 0.56 out): 8192 x 2048 beside the router GEMM 0.027 -> 0.023 ms.
__global__ void __launch_bounds__(256)
quantize_rows_kernel(const __nv_bfloat16* __restrict__ x, uint32_t rows, uint32_t k, float g,
                     uint8_t* __restrict__ packed, uint8_t* __restrict__ scale_tiled)
{
    chain_begin();
    quantize_row_chunk(x, rows, k, g, packed, scale_tiled, static_cast<uint64_t>(blockIdx.x) * 8 + (threadIdx.x >> 5));
}

// Gather of already-quantised rows into the padded permuted layout, organised by destination tile (128-row token
// tiles; the kernel for smaller tiles fetches its rows itself): block (k chunk, tile) moves the rows of one token tile of one expert for 512 elements of k. The codes of a row chunk are 256 contiguous
// bytes (16 threads x 16 bytes), and a scale tile of the destination (512 bytes: 32 lanes x
// four 32-row groups) is written with one 16-byte store per lane instead of 128 scattered
// 4-byte stores. Rows are found through the
// routing tables: padded row -> dense row -> token.
constexpr uint32_t kGatherChunk = 512; // elements of k per block

__global__ void __launch_bounds__(256)
gather_packed_tiles_kernel(const uint8_t* __restrict__ hidden_packed, const uint8_t* __restrict__ hidden_scale,
                           const RouteTables rt, uint32_t hidden_size, uint8_t* __restrict__ packed,
                           uint8_t* __restrict__ scale_tiled, int src_scale_tiled)
{
    chain_begin();
    const uint32_t tile = blockIdx.y;
    if (static_cast<int>(tile) >= *rt.total_tiles)
        return;
    const int expert = rt.tile_expert[tile];
    const uint32_t row0 = static_cast<uint32_t>(rt.tile_row0[tile]);
    const uint32_t nrows = static_cast<uint32_t>(rt.tile_nrows[tile]);
    // dense (unpadded) row of the tile's first row: same offset inside the expert's segment
    const uint32_t dense0 = static_cast<uint32_t>(rt.indptr[expert])
        + (row0 - static_cast<uint32_t>(rt.pad_indptr[expert]));
    const uint32_t kgroups = hidden_size / 64;
    const uint32_t row_bytes = hidden_size / 2;
    const uint32_t chunk_bytes = kGatherChunk / 2;
    const uint32_t c0 = blockIdx.x * chunk_bytes;

    // codes: 16 threads per row, 16 rows per pass
    const uint32_t sub = threadIdx.x & 15;
    if (c0 + sub * 16 < row_bytes) {
        for (uint32_t j = threadIdx.x >> 4; j < nrows; j += 16) {
            const uint64_t token = static_cast<uint64_t>(rt.row_tokens[dense0 + j]);
            const uint4 v = *reinterpret_cast<const uint4*>(hidden_packed + token * row_bytes + c0 + sub * 16);
            *reinterpret_cast<uint4*>(packed + static_cast<uint64_t>(row0 + j) * row_bytes + c0 + sub * 16) = v;
        }
    }
    // scales: this block's k groups
    const uint32_t kg0 = blockIdx.x * (kGatherChunk / 64);
    const auto src_word = [&](uint32_t j, uint32_t kg) -> uint32_t {
        if (j >= nrows)
            return 0u;
        const uint64_t token = static_cast<uint64_t>(rt.row_tokens[dense0 + j]);
        const uint64_t off = src_scale_tiled ? tiled_scale_offset(token, 4ull * kg, kgroups)
                                             : token * (hidden_size / 16) + kg * 4;
        return *reinterpret_cast<const uint32_t*>(hidden_scale + off);
    };
    // thread = (k group, lane of the scale tile): the words of rows lane, lane + 32, lane + 64, lane + 96
    const uint32_t kg = kg0 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (kg < kgroups) {
        const uint4 v = make_uint4(src_word(lane, kg), src_word(lane + 32, kg), src_word(lane + 64, kg),
                                   src_word(lane + 96, kg));
        *reinterpret_cast<uint4*>(scale_tiled + (static_cast<uint64_t>(row0 >> 7) * kgroups + kg) * 512 + lane * 16)
            = v;
    }
}

// linear [experts, rows, k/16] -> tiled; one thread per (row, k group).
__global__ void tile_scales_kernel(const uint8_t* __restrict__ linear, uint32_t rows, uint32_t k,
                                   uint64_t total, uint8_t* __restrict__ tiled, uint64_t tiled_bytes,
                                   int gated)
{
    const uint64_t idx = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (idx >= total)
        return;
    const uint32_t kgroups = k / 64;
    const uint32_t kg = static_cast<uint32_t>(idx % kgroups);
    const uint64_t grow = idx / kgroups;
    const uint32_t e = static_cast<uint32_t>(grow / rows);
    const uint32_t row = static_cast<uint32_t>(grow % rows);
    const uint32_t sf = *reinterpret_cast<const uint32_t*>(linear + grow * (k / 16) + kg * 4);
    const uint64_t tr = gated ? gated_tiled_row(row, rows / 2) : row;
    *reinterpret_cast<uint32_t*>(tiled + static_cast<uint64_t>(e) * tiled_bytes
                                 + tiled_scale_offset(tr, 4ull * kg, kgroups))
        = sf;
}

uint32_t blocks_for(uint64_t total, uint32_t threads)
{
    return static_cast<uint32_t>((total + threads - 1) / threads);
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// Fewer blocks than SMs and more than a few microseconds' work for each: the whole grid per expert instead of a cluster,
// which costs a memset and two launches. Experts x bytes of each, cluster / whole grid in us: 1 x 4 MB 14 / 13, 1 x 17
// 44 / 14, 1 x 134 401 / 63, 4 x 8 25 / 18, 4 x 67 223 / 109, 8 x 8 37 / 27, 12 x 8 47 / 50, 16 x 34 278 / 254, 20 x 34
// 302 / 330.
bool quantize_flat_pays(uint64_t experts, uint64_t per_expert)
{
    return experts * kQwCluster < kSmCount && per_expert > (2u << 20);
}

} // namespace

cudaError_t launch_nvfp4_quantize_rows(const __nv_bfloat16* x, uint32_t rows, uint32_t k, float global_scale,
                                       uint8_t* packed, uint8_t* scale_tiled, cudaStream_t stream)
{
    const uint64_t units = static_cast<uint64_t>(rows) * ((k + 511) / 512);
    return launch_chained(quantize_rows_kernel, dim3(blocks_for(units, 8)), 256, 0, stream, x, rows, k,
                          global_scale == 0.0f ? 1.0f : global_scale, packed, scale_tiled);
}

cudaError_t launch_nvfp4_gather_tiles(const uint8_t* hidden_packed, const uint8_t* hidden_scale, const RouteTables& rt,
                                      uint32_t hidden_size, uint8_t* packed, uint8_t* scale_tiled, cudaStream_t stream,
                                      int src_scale_tiled)
{
    if (rt.max_tiles == 0)
        return cudaSuccess;
    const dim3 grid((hidden_size + kGatherChunk - 1) / kGatherChunk, rt.max_tiles, 1);
    return launch_chained(gather_packed_tiles_kernel, grid, 256, 0, stream, hidden_packed, hidden_scale, rt, hidden_size,
                          packed, scale_tiled, src_scale_tiled);
}

cudaError_t launch_tile_scales(const uint8_t* linear, uint32_t experts, uint32_t rows, uint32_t k,
                               int gated, uint8_t* tiled, cudaStream_t stream)
{
    const uint64_t total = static_cast<uint64_t>(experts) * rows * (k / 64);
    tile_scales_kernel<<<blocks_for(total, 256), 256, 0, stream>>>(
        linear, rows, k, total, tiled, qs3_nvfp4_tiled_scale_bytes(rows, k), gated);
    note_launch();
    return cudaGetLastError();
}

} // namespace qs3

using namespace qs3;

extern "C" {

qsfi_status qs3_nvfp4_quantize_weight(qsfi_context* ctx, const qs3_nvfp4_quantize_weight_desc* d)
{
    if (ctx == nullptr)
        return QSFI_STATUS_INVALID_ARGUMENT;
    clear_error(&ctx->last_error);
    qsfi_status status = activate_context(ctx);
    if (status != QSFI_STATUS_OK)
        return status;
    if (d == nullptr)
        return set_invalid_arg(ctx, "desc is null");
    if (d->weight.data == nullptr || d->weight.dtype != QSFI_DTYPE_BF16 || !contiguous3(d->weight))
        return set_invalid_arg(ctx, "weight must be a contiguous bf16 [experts, rows, k] tensor");
    const int64_t experts = d->weight.shape[0], rows = d->weight.shape[1], k = d->weight.shape[2];
    if (experts <= 0 || rows <= 0 || k <= 0 || k % 64 != 0)
        return set_invalid_arg(ctx, "NVFP4 weight quantisation requires k divisible by 64");
    if (d->gated_rows != 0 && rows % 128 != 0)
        return set_invalid_arg(ctx, "gated NVFP4 weights require 2*intermediate divisible by 128");
    if (d->packed.data == nullptr || d->packed.dtype != QSFI_DTYPE_U8 || !contiguous3(d->packed)
        || d->packed.shape[0] != experts || d->packed.shape[1] != rows || d->packed.shape[2] != k / 2)
        return set_invalid_arg(ctx, "packed must be a contiguous u8 [experts, rows, k/2] tensor");
    if (d->global_scale.data == nullptr || d->global_scale.dtype != QSFI_DTYPE_F32
        || d->global_scale.shape[0] != experts || !contiguous1(d->global_scale))
        return set_invalid_arg(ctx, "global_scale must be a contiguous f32 [experts] tensor");
    if (d->scale_linear.data != nullptr
        && (d->scale_linear.dtype != QSFI_DTYPE_FP8_E4M3 || !contiguous3(d->scale_linear)
            || d->scale_linear.shape[0] != experts || d->scale_linear.shape[1] != rows
            || d->scale_linear.shape[2] != k / 16))
        return set_invalid_arg(ctx, "scale_linear must be a contiguous e4m3 [experts, rows, k/16] tensor");
    const uint64_t tiled_bytes = qs3_nvfp4_tiled_scale_bytes(rows, k);
    if (d->scale_tiled.data != nullptr
        && (d->scale_tiled.dtype != QSFI_DTYPE_U8 || !contiguous1(d->scale_tiled)
            || static_cast<uint64_t>(d->scale_tiled.shape[0]) < tiled_bytes * experts))
        return set_invalid_arg(ctx, "scale_tiled is too small");
    if (!aligned16(d->weight.data) || !aligned16(d->packed.data)
        || (d->scale_tiled.data != nullptr && !aligned16(d->scale_tiled.data)))
        return set_invalid_arg(ctx, "NVFP4 quantisation buffers must be 16-byte aligned");

    // rows of the last 128-row block that do not exist get scale 0 from the kernels themselves
    const uint64_t per_expert = static_cast<uint64_t>(rows) * k;
    if (quantize_flat_pays(static_cast<uint64_t>(experts), per_expert)) {
        cudaStream_t st = ctx->stream;
        const uint32_t want = 2 * kSmCount, e32 = static_cast<uint32_t>(experts);
        const uint64_t units = (rows + 127) / 128 * ((k + kQwChunk - 1) / kQwChunk);
        cudaError_t err = cudaMemsetAsync(d->global_scale.data, 0, sizeof(float) * e32, st);
        if (err != cudaSuccess)
            return set_cuda_error(ctx, err, "cudaMemsetAsync global_scale");
        expert_amax_kernel<<<dim3((2 * want + e32 - 1) / e32, e32), kQwThreads, 0, st>>>(
            static_cast<const __nv_bfloat16*>(d->weight.data), per_expert, static_cast<uint32_t*>(d->global_scale.data));
        finish_global_scale_kernel<<<1, 32, 0, st>>>(static_cast<float*>(d->global_scale.data), e32);
        quantize_weight_flat_kernel<<<dim3(static_cast<uint32_t>(std::min<uint64_t>(units, (want + e32 - 1) / e32)), e32),
                                      kQwThreads, 0, st>>>(
            static_cast<const __nv_bfloat16*>(d->weight.data), static_cast<uint32_t>(rows), static_cast<uint32_t>(k),
            static_cast<const float*>(d->global_scale.data), static_cast<uint8_t*>(d->packed.data),
            static_cast<uint8_t*>(d->scale_linear.data), static_cast<uint8_t*>(d->scale_tiled.data), tiled_bytes,
            static_cast<int>(d->gated_rows != 0));
        note_launch(3);
        return set_cuda_error(ctx, cudaGetLastError(), "qs3_nvfp4_quantize_weight");
    }
    static bool configured[64] = {};
    const int dev = ctx->device_ordinal;
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        const cudaError_t err
            = cudaFuncSetAttribute(quantize_weight_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        if (err != cudaSuccess)
            return set_cuda_error(ctx, err, "NVFP4 weight quantiser cluster size");
        if (dev >= 0 && dev < 64)
            configured[dev] = true;
    }
    cudaLaunchConfig_t cfg {};
    cudaLaunchAttribute attr {};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim = { kQwCluster, 1, 1 };
    cfg.gridDim = dim3(kQwCluster * static_cast<uint32_t>(experts));
    cfg.blockDim = dim3(kQwThreads);
    cfg.stream = ctx->stream;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    const cudaError_t err = cudaLaunchKernelEx(
        &cfg, quantize_weight_kernel, static_cast<const __nv_bfloat16*>(d->weight.data), static_cast<uint32_t>(rows),
        static_cast<uint32_t>(k), static_cast<float*>(d->global_scale.data), static_cast<uint8_t*>(d->packed.data),
        static_cast<uint8_t*>(d->scale_linear.data), static_cast<uint8_t*>(d->scale_tiled.data), tiled_bytes,
        static_cast<int>(d->gated_rows != 0));
    note_launch();
    return set_cuda_error(ctx, err, "qs3_nvfp4_quantize_weight");
}

qsfi_status qs3_nvfp4_quantize_act(qsfi_context* ctx, const qs3_nvfp4_quantize_act_desc* d)
{
    if (ctx == nullptr)
        return QSFI_STATUS_INVALID_ARGUMENT;
    clear_error(&ctx->last_error);
    qsfi_status status = activate_context(ctx);
    if (status != QSFI_STATUS_OK)
        return status;
    if (d == nullptr)
        return set_invalid_arg(ctx, "desc is null");
    if (d->x.data == nullptr || d->x.dtype != QSFI_DTYPE_BF16 || !contiguous2(d->x)
        || d->x.shape[0] != d->rows || d->x.shape[1] <= 0 || d->x.shape[1] % 16 != 0)
        return set_invalid_arg(ctx, "x must be a contiguous bf16 [rows, k] tensor with k divisible by 16");
    const int64_t k = d->x.shape[1];
    if (d->packed.data == nullptr || d->packed.dtype != QSFI_DTYPE_U8 || !contiguous2(d->packed)
        || d->packed.shape[0] != d->rows || d->packed.shape[1] != k / 2)
        return set_invalid_arg(ctx, "packed must be a contiguous u8 [rows, k/2] tensor");
    if (d->scale_linear.data == nullptr || d->scale_linear.dtype != QSFI_DTYPE_FP8_E4M3
        || !contiguous2(d->scale_linear) || d->scale_linear.shape[0] != d->rows
        || d->scale_linear.shape[1] != k / 16)
        return set_invalid_arg(ctx, "scale_linear must be a contiguous e4m3 [rows, k/16] tensor");
    if (!aligned16(d->x.data) || !aligned16(d->packed.data))
        return set_invalid_arg(ctx, "NVFP4 quantisation buffers must be 16-byte aligned");
    const uint64_t total = static_cast<uint64_t>(d->rows) * (k / 16);
    quantize_act_linear_kernel<<<blocks_for(total, 256), 256, 0, ctx->stream>>>(
        static_cast<const __nv_bfloat16*>(d->x.data), static_cast<uint32_t>(k), total,
        d->global_scale == 0.0f ? 1.0f : d->global_scale, static_cast<uint8_t*>(d->packed.data),
        static_cast<uint8_t*>(d->scale_linear.data));
    note_launch();
    return set_cuda_error(ctx, cudaGetLastError(), "qs3_nvfp4_quantize_act");
}

qsfi_status qs3_nvfp4_tile_scales(qsfi_context* ctx, const qs3_nvfp4_tile_scales_desc* d)
{
    if (ctx == nullptr)
        return QSFI_STATUS_INVALID_ARGUMENT;
    clear_error(&ctx->last_error);
    qsfi_status status = activate_context(ctx);
    if (status != QSFI_STATUS_OK)
        return status;
    if (d == nullptr)
        return set_invalid_arg(ctx, "desc is null");
    if (d->scale_linear.data == nullptr || d->scale_linear.dtype != QSFI_DTYPE_FP8_E4M3
        || !contiguous3(d->scale_linear) || d->scale_linear.shape[2] <= 0
        || d->scale_linear.shape[2] % 4 != 0)
        return set_invalid_arg(ctx, "scale_linear must be a contiguous e4m3 [experts, rows, k/16] tensor with k divisible by 64");
    const int64_t experts = d->scale_linear.shape[0], rows = d->scale_linear.shape[1];
    const int64_t k = d->scale_linear.shape[2] * 16;
    if (d->gated_rows != 0 && rows % 128 != 0)
        return set_invalid_arg(ctx, "gated NVFP4 weights require 2*intermediate divisible by 128");
    const uint64_t tiled_bytes = qs3_nvfp4_tiled_scale_bytes(rows, k);
    if (d->scale_tiled.data == nullptr || d->scale_tiled.dtype != QSFI_DTYPE_U8
        || static_cast<uint64_t>(d->scale_tiled.shape[0]) < tiled_bytes * experts)
        return set_invalid_arg(ctx, "scale_tiled is too small");
    if ((reinterpret_cast<uintptr_t>(d->scale_linear.data) & 3u) != 0 || !aligned16(d->scale_tiled.data))
        return set_invalid_arg(ctx, "scale buffers are misaligned");
    if (rows % 128 != 0) {
        cudaError_t err = cudaMemsetAsync(d->scale_tiled.data, 0, tiled_bytes * experts, ctx->stream);
        if (err != cudaSuccess)
            return set_cuda_error(ctx, err, "cudaMemsetAsync scale_tiled");
    }
    cudaError_t err = launch_tile_scales(static_cast<const uint8_t*>(d->scale_linear.data),
                                         static_cast<uint32_t>(experts), static_cast<uint32_t>(rows),
                                         static_cast<uint32_t>(k), d->gated_rows != 0,
                                         static_cast<uint8_t*>(d->scale_tiled.data), ctx->stream);
    return set_cuda_error(ctx, err, "qs3_nvfp4_tile_scales");
}

} // extern "C"
