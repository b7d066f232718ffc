// Tensor-pipe peak probe: every SM issues back-to-back tcgen05.mma instructions on
// operand tiles that already sit in shared memory (no loads inside the timed loop), so
// the measured rate is the tensor-pipe ceiling of one instruction shape on this device.
// It provides the FP4 / FP8 / BF16 denominators for the "fraction of tensor peak"
// figures; it is not part of the MoE data path.
#include "tcgen05.cuh"

#include <cooperative_groups.h>

namespace qs3 {
namespace {

using namespace tc;

enum ProbeKind { PROBE_BF16 = 0, PROBE_FP8 = 1, PROBE_NVFP4 = 2 };

// One CTA per SM: A tile 128 rows x 128 bytes, B tile n rows x 128 bytes, 128-byte swizzle
// layout (contents are pseudo-random bytes; the result is never read). Each iteration
// issues the MMAs that consume one 128-byte k-block: 4 instructions of K = 32 bytes.
// cps_main / cps_side (NVFP4 only): scale-tile copies (tcgen05.cp, 512 bytes each) per
// iteration issued by the MMA thread ahead of its four MMAs, into the scale columns those
// MMAs read / by a second thread that runs free of the first. They measure what the scale
// copies of a block-scaled main loop cost the tensor pipe.
__global__ void __launch_bounds__(128, 1)
tensor_peak_kernel(int kind, uint32_t n, uint32_t iters, uint32_t* err, uint32_t cps_main, uint32_t cps_side)
{
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    uint8_t* a_tile = smem;
    uint8_t* b_tile = smem + kTileBytes;                 // up to 256 rows = 32 KB
    uint8_t* sf_tile = b_tile + 2 * kTileBytes;          // 512 bytes of scale 1.0
    uint64_t* done_bar = reinterpret_cast<uint64_t*>(sf_tile + 1024);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done_bar + 1);
    volatile uint32_t* abort_flag = tmem_slot + 1;

    uint32_t x = 0x9e3779b9u * (blockIdx.x + 1) + threadIdx.x;
    for (uint32_t i = threadIdx.x; i < 3 * kTileBytes / 4; i += blockDim.x) {
        x = x * 1664525u + 1013904223u;
        // keep exponents small so that no format produces Inf/NaN in the accumulator
        reinterpret_cast<uint32_t*>(smem)[i] = x & 0x37373737u;
    }
    for (uint32_t i = threadIdx.x; i < 512; i += blockDim.x)
        sf_tile[i] = 0x38; // e4m3 1.0
    if (threadIdx.x == 0) {
        mbar_init(done_bar, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    if (threadIdx.x < 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(512u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (threadIdx.x < 32 && elect_one()) {
        const uint32_t nm = ((n >> 3) << 17) | ((kBM >> 4) << 24);
        const uint32_t idesc = kind == PROBE_BF16 ? ((1u << 4) | (1u << 7) | (1u << 10) | nm)
            : kind == PROBE_FP8                  ? ((1u << 4) | nm) // e4m3 x e4m3, f32 accumulate
                                                 : ((1u << 7) | (1u << 10) | nm);
        const uint64_t da = operand_desc(smem_u32(a_tile));
        const uint64_t db = operand_desc(smem_u32(b_tile));
        const uint32_t sfa = tmem_base + 256, sfb = tmem_base + 272;
        if (kind == PROBE_NVFP4) {
            for (uint32_t c = 0; c < 40; ++c) // scale 1.0 everywhere the MMAs may look
                tc_cp_scales(sfa + 4 * c, scale_desc(smem_u32(sf_tile)));
        }
        const uint64_t sdesc = scale_desc(smem_u32(sf_tile));
        for (uint32_t it = 0; it < iters; ++it) {
            // the copies alternate between two groups of scale columns, as a main loop does
            const uint32_t sfb_it = cps_main != 0 ? sfb + 64 * (it & 1) : sfb;
            for (uint32_t c = 0; c < cps_main; ++c)
                tc_cp_scales(sfb_it + 4 * c, sdesc);
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j) {
                const uint32_t acc = (it | j) != 0 ? 1u : 0u;
                if (kind == PROBE_BF16)
                    tc_mma_bf16(tmem_base, da + 2 * j, db + 2 * j, idesc, acc);
                else if (kind == PROBE_FP8)
                    tc_mma_f8(tmem_base, da + 2 * j, db + 2 * j, idesc, acc);
                else
                    tc_mma_nvfp4(tmem_base, da + 2 * j, db + 2 * j, idesc, acc, sfa, sfb_it + 8 * (j & 1));
            }
        }
        tc_commit(done_bar);
        mbar_wait<true>(done_bar, 0, abort_flag, err, 0x53000001u);
    } else if (threadIdx.x / 32 == 1 && elect_one() && cps_side != 0 && kind == PROBE_NVFP4) {
        const uint64_t sdesc = scale_desc(smem_u32(sf_tile));
        const uint32_t side = tmem_base + 416; // columns no MMA of this probe reads
        for (uint32_t it = 0; it < iters; ++it)
            for (uint32_t c = 0; c < cps_side; ++c)
                tc_cp_scales(side + 4 * c, sdesc);
    }
    tc_fence_before();
    __syncthreads();
    if (threadIdx.x < 32) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u)
                     : "memory");
    }
}

// The same loop with CTA pairs: a cluster of two CTAs issues cta_group::2 instructions of
// 256 x n (128 rows of A and n / 2 rows of B from each CTA's shared memory; each CTA's
// tensor memory receives its 128 rows of the result). Only the first CTA of the pair
// issues; the other one provides its shared and tensor memory.
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(128, 1)
tensor_peak_pair_kernel(int kind, uint32_t n, uint32_t iters, uint32_t* err)
{
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    const uint32_t cta_rank = cluster.block_rank();

    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    uint8_t* a_tile = smem;
    uint8_t* b_tile = smem + kTileBytes;                 // n / 2 <= 128 rows
    uint8_t* sf_tile = b_tile + 2 * kTileBytes;
    uint64_t* done_bar = reinterpret_cast<uint64_t*>(sf_tile + 1024);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done_bar + 1);
    volatile uint32_t* abort_flag = tmem_slot + 1;

    uint32_t x = 0x9e3779b9u * (blockIdx.x + 1) + threadIdx.x;
    for (uint32_t i = threadIdx.x; i < 3 * kTileBytes / 4; i += blockDim.x) {
        x = x * 1664525u + 1013904223u;
        reinterpret_cast<uint32_t*>(smem)[i] = x & 0x37373737u;
    }
    for (uint32_t i = threadIdx.x; i < 512; i += blockDim.x)
        sf_tile[i] = 0x38;
    if (threadIdx.x == 0) {
        mbar_init(done_bar, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    cluster.sync(); // both CTAs are resident before the paired allocation
    if (threadIdx.x < 32) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(512u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    cluster.sync();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (cta_rank == 0 && threadIdx.x < 32 && elect_one()) {
        const uint32_t nm = ((n >> 3) << 17) | ((256u >> 4) << 24);
        const uint32_t idesc = kind == PROBE_BF16 ? ((1u << 4) | (1u << 7) | (1u << 10) | nm)
            : kind == PROBE_FP8                  ? ((1u << 4) | nm)
                                                 : ((1u << 7) | (1u << 10) | nm);
        const uint64_t da = operand_desc(smem_u32(a_tile));
        const uint64_t db = operand_desc(smem_u32(b_tile));
        const uint32_t sfa = tmem_base + 256, sfb = tmem_base + 272;
        if (kind == PROBE_NVFP4) {
            for (uint32_t c = 0; c < 12; ++c)
                asm volatile("tcgen05.cp.cta_group::2.32x128b.warpx4 [%0], %1;" ::"r"(sfa + 4 * c),
                             "l"(scale_desc(smem_u32(sf_tile)))
                             : "memory");
        }
        for (uint32_t it = 0; it < iters; ++it) {
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j) {
                const uint32_t acc = (it | j) != 0 ? 1u : 0u;
                if (kind == PROBE_BF16)
                    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                                 "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_base),
                                 "l"(da + 2 * j), "l"(db + 2 * j), "r"(idesc), "r"(acc)
                                 : "memory");
                else if (kind == PROBE_FP8)
                    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                                 "tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_base),
                                 "l"(da + 2 * j), "l"(db + 2 * j), "r"(idesc), "r"(acc)
                                 : "memory");
                else
                    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                                 "tcgen05.mma.cta_group::2.kind::mxf4nvf4.block_scale.scale_vec::4X"
                                 " [%0], %1, %2, %3, [%5], [%6], p;\n\t}" ::"r"(tmem_base),
                                 "l"(da + 2 * j), "l"(db + 2 * j), "r"(idesc), "r"(acc), "r"(sfa), "r"(sfb)
                                 : "memory");
            }
        }
        asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                         smem_u32(done_bar))
                     : "memory");
        mbar_wait<true>(done_bar, 0, abort_flag, err, 0x53000002u);
    }
    tc_fence_before();
    cluster.sync(); // the pair's tensor memory is idle in both CTAs
    if (threadIdx.x < 32) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u)
                     : "memory");
    }
}

// Operand-delivery probe: every SM streams `tiles` tiles of `tile_bytes` from a buffer that fits the L2
// into its shared memory with bulk copies, `stages` of them in flight, and does nothing with them.
// CTA b walks the buffer from its own offset, so all SMs read different lines at any time and every line
// is read by several SMs over the run, as the weight stream of a grouped GEMM is.
//
// pattern 0: a tile is `tile_bytes` contiguous bytes (one cp.async.bulk): operands stored as shared-memory
// images. pattern 1: the buffer is a row-major matrix with 1 KiB rows and a tile is a 128-row x 128-byte
// box of it with the 128-byte swizzle (one cp.async.bulk.tensor.2d): what a k-major operand with k = 2048
// FP4 elements per row looks like to the copy engine (128 separate 128-byte segments per tile).
__global__ void __launch_bounds__(32, 1)
operand_stream_kernel(const __grid_constant__ CUtensorMap map, const uint8_t* __restrict__ buf, uint64_t buf_bytes,
                      uint32_t tile_bytes, uint32_t stages, uint32_t tiles, uint32_t pattern, uint32_t* err)
{
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + static_cast<size_t>(stages) * tile_bytes);
    __shared__ uint32_t abort_flag;
    if (threadIdx.x != 0)
        return;
    abort_flag = 0;
    for (uint32_t s = 0; s < stages; ++s)
        mbar_init(&bars[s], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    const uint64_t n_tiles = buf_bytes / tile_bytes;
    uint64_t at = (static_cast<uint64_t>(blockIdx.x) * 9973u) % n_tiles;
    for (uint32_t i = 0; i < tiles + stages; ++i) {
        const uint32_t s = i % stages;
        if (i >= stages && !mbar_wait(&bars[s], ((i / stages) - 1) & 1, &abort_flag, err, 0x57000001u))
            break;
        if (i < tiles) {
            mbar_expect_tx(&bars[s], tile_bytes);
            if (pattern == 0)
                bulk_load(smem + static_cast<size_t>(s) * tile_bytes, buf + at * tile_bytes, tile_bytes, &bars[s]);
            else // eight boxes side by side per 128 rows
                tma_load_2d(smem + static_cast<size_t>(s) * tile_bytes, &map, &bars[s],
                            static_cast<int>(at % 8) * 128, static_cast<int>(at / 8) * 128);
            at = at + 1 == n_tiles ? 0 : at + 1;
        }
    }
}

} // namespace
} // namespace qs3

using namespace qs3;

extern "C" qsfi_status qs3_tensor_peak_probe(qsfi_context* ctx, uint32_t kind, uint32_t n, uint32_t iters,
                                             double* tflops)
{
    if (ctx == nullptr || tflops == nullptr)
        return QSFI_STATUS_INVALID_ARGUMENT;
    clear_error(&ctx->last_error);
    qsfi_status status = activate_context(ctx);
    if (status != QSFI_STATUS_OK)
        return status;
    const bool pair = (kind & 16u) != 0; // + 16: CTA pairs issuing cta_group::2 instructions of 256 x n
    const uint32_t cps_main = (kind >> 8) & 15u, cps_side = (kind >> 12) & 15u;
    kind &= 15u;
    if ((cps_main | cps_side) != 0 && (pair || kind != 2 || cps_main > 8 || cps_side > 8))
        return set_invalid_arg(ctx, "peak probe: scale copies go with the single-CTA NVFP4 probe, at most 8 per iteration");
    if (kind > 2 || n < 16 || n > 256 || n % 16 != 0 || iters == 0 || iters > (1u << 22) || (pair && n % 32 != 0))
        return set_invalid_arg(ctx, "peak probe: kind in {0,1,2} (+16), n a multiple of 16 in [16, 256], iters in [1, 2^22]");
    int dev = 0, sms = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err == cudaSuccess)
        err = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const size_t smem = 3 * kTileBytes + 1024 + 64 + 1024;
    if (err == cudaSuccess)
        err = cudaFuncSetAttribute(tensor_peak_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   static_cast<int>(smem));
    if (err == cudaSuccess)
        err = cudaFuncSetAttribute(tensor_peak_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   static_cast<int>(smem));
    if (pair)
        sms &= ~1; // whole pairs only
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    if (err == cudaSuccess)
        err = cudaEventCreate(&e0);
    if (err == cudaSuccess)
        err = cudaEventCreate(&e1);
    if (err != cudaSuccess)
        return set_cuda_error(ctx, err, "peak probe setup");
    uint32_t* errw = device_error_word();
    const auto launch = [&](uint32_t count) {
        if (pair)
            tensor_peak_pair_kernel<<<sms, 128, smem, ctx->stream>>>(static_cast<int>(kind), n, count, errw);
        else
            tensor_peak_kernel<<<sms, 128, smem, ctx->stream>>>(static_cast<int>(kind), n, count, errw, cps_main,
                                                                cps_side);
    };
    launch(64); // warm-up
    cudaEventRecord(e0, ctx->stream);
    launch(iters);
    cudaEventRecord(e1, ctx->stream);
    note_launch(2);
    err = cudaEventSynchronize(e1);
    float ms = 0.0f;
    if (err == cudaSuccess)
        err = cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (err != cudaSuccess)
        return set_cuda_error(ctx, err, "peak probe");
    // K elements per instruction: 32 bytes of K -> 16 bf16, 32 fp8, 64 fp4
    const double k_per_mma = kind == 0 ? 16.0 : kind == 1 ? 32.0 : 64.0;
    // a pair instruction is 256 x n and is issued by every second CTA
    const double flops = 2.0 * (pair ? 256.0 * 0.5 : 128.0) * n * k_per_mma * 4.0 * iters * sms;
    *tflops = flops / (static_cast<double>(ms) * 1e-3) / 1e12;
    return QSFI_STATUS_OK;
}

extern "C" qsfi_status qs3_operand_stream_probe(qsfi_context* ctx, void* buffer, uint64_t buffer_bytes,
                                                uint32_t tile_bytes, uint32_t stages, uint32_t tiles,
                                                uint32_t pattern, double* gbs)
{
    if (ctx == nullptr || gbs == nullptr)
        return QSFI_STATUS_INVALID_ARGUMENT;
    clear_error(&ctx->last_error);
    qsfi_status status = activate_context(ctx);
    if (status != QSFI_STATUS_OK)
        return status;
    if (buffer == nullptr || (reinterpret_cast<uintptr_t>(buffer) & 15u) != 0 || tile_bytes < 1024
        || tile_bytes % 1024 != 0 || stages == 0 || stages > 32 || tiles == 0 || tiles > (1u << 24)
        || static_cast<uint64_t>(stages) * tile_bytes > 200u * 1024u || buffer_bytes < 2ull * tile_bytes
        || pattern > 1 || (pattern == 1 && (tile_bytes != 16384 || buffer_bytes % (128u * 1024u) != 0)))
        return set_invalid_arg(ctx, "operand stream probe: 16-byte aligned buffer of at least two tiles, tile a "
                                    "multiple of 1 KiB, stages * tile <= 200 KiB, 1..32 stages, 1..2^24 tiles");
    int dev = 0, sms = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err == cudaSuccess)
        err = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const size_t smem = static_cast<size_t>(stages) * tile_bytes + 1024 + 8 * stages;
    if (err == cudaSuccess)
        err = cudaFuncSetAttribute(operand_stream_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   static_cast<int>(smem));
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    if (err == cudaSuccess)
        err = cudaEventCreate(&e0);
    if (err == cudaSuccess)
        err = cudaEventCreate(&e1);
    if (err != cudaSuccess)
        return set_cuda_error(ctx, err, "operand stream probe setup");
    uint32_t* errw = device_error_word();
    const uint8_t* buf = static_cast<const uint8_t*>(buffer);
    CUtensorMap map {};
    if (pattern == 1 && !make_operand_map(&map, true, buffer, 1024, buffer_bytes / 1024, 1024, 128))
        return set_invalid_arg(ctx, "operand stream probe: cuTensorMapEncodeTiled failed");
    // first pass brings the buffer into L2 (when it fits), the second one is timed
    operand_stream_kernel<<<sms, 32, smem, ctx->stream>>>(map, buf, buffer_bytes, tile_bytes, stages, tiles, pattern,
                                                         errw);
    cudaEventRecord(e0, ctx->stream);
    operand_stream_kernel<<<sms, 32, smem, ctx->stream>>>(map, buf, buffer_bytes, tile_bytes, stages, tiles, pattern,
                                                         errw);
    cudaEventRecord(e1, ctx->stream);
    note_launch(2);
    err = cudaEventSynchronize(e1);
    float ms = 0.0f;
    if (err == cudaSuccess)
        err = cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (err != cudaSuccess)
        return set_cuda_error(ctx, err, "operand stream probe");
    *gbs = static_cast<double>(sms) * tiles * tile_bytes / (static_cast<double>(ms) * 1e-3) / 1e9;
    return QSFI_STATUS_OK;
}
