// Dense bf16 GEMM with few output tiles  D[m, n] = alpha * sum_k A[m, k] * B[n, k] (+ beta * D) (+ bias[n]):
// router logits, and projections of a decode batch. One CTA per output tile would stream all of k through a handful
// of SMs (128 x 512 x 2048: four), so k is split over the CTAs of a cluster, whose partial tiles are summed through
// distributed shared memory in rank order (the result does not depend on timing) without a scratch buffer or a
// second launch.
//
//   grid    (splits, ceil(n / 128), ceil(m / NT)), clusters of `splits` CTAs
//   tile    128 weight rows (M side) x NT rows of A (N side, 16..128): accumulator lane = feature, column = row
//   smem    ring of stages: B 128 x 64 + A NT x 64; then the f32 partial tile [NT][128] (the ring is idle by then)
//   warps   0-3 (and 6 upwards) accumulator -> shared memory, 4 producer (TMA), 5 MMA issuer; all sum and store
//
// f32 results of few rows: the tensor core truncates what it adds to an accumulator, about 1.5e-8 of the result for every
// instruction in the chain. So two instructions at most meet in an accumulator (each k block fills two), and warps add them
// up in registers, compensated, as do the sums over the ranks. Error against 64 bits (2-norm) and time of 2048 x 512:
//   rows                            1          16         64
//   one chain per rank              24e-8 4.4  24e-8 4.4  23e-8 5.7 us
//   short chains, compensated       6.8e-8 4.4 6.5e-8 5.0 6.6e-8 5.8
//   CUDA cores, a block per feature 7.5e-8 5.6 8.1e-8 8.5 7.9e-8 28.6 (gemm_skinny_kernel: few features)
// and of 65000 features, where no tile is split, 64 rows: one chain 2.1e-6 56 us, compensated 5.8e-8 98, CUDA cores 7.9e-8
// 3710.
//
// Bound by latency: launch, one trip to HBM for the weights (and, at decode sizes, the code), two cluster barriers.
// Router logits, hidden 2048: 512 experts, 128 tokens 0.0153 -> 0.0098 ms (split over grid.z with a reduction pass), 1021
// tokens 0.0194 -> 0.0112; 128 experts, 4096 tokens 0.0204 -> 0.0128.
#include "tcgen05.cuh"

#include <cooperative_groups.h>

#include <algorithm>

namespace qs3 {
namespace {

using namespace tc;

constexpr uint32_t kSkMaxStages = 8;
constexpr uint32_t kSkRing = 192 * 1024; // shared memory of the stages, at most
constexpr uint32_t kSkMaxSplits = 8; // the largest portable cluster
constexpr uint32_t kSkPitch = 132; // floats per row of the partial tile

enum : uint32_t {
    ERR_SK_FULL_WAIT = 0x5a000001u,
    ERR_SK_EMPTY_WAIT = 0x5a000002u,
    ERR_SK_ACC_WAIT = 0x5a000003u,
    ERR_SK_ACC_EMPTY_WAIT = 0x5a000004u,
};

struct SplitkParams {
    uint32_t m, n;
    uint32_t k_blocks, kb_per_split;
    uint32_t stages;
    void* out;
    uint64_t out_pitch;
    float alpha, beta;
    const float* bias;
    uint32_t* err;
};

template <int NT> struct SkSmem {
    static constexpr uint32_t kStageBytes = kTileBytes + NT * 128;
    static constexpr uint32_t kPartial = NT * kSkPitch * 4;
    static constexpr uint32_t kMostStages = kSkRing / kStageBytes < kSkMaxStages ? kSkRing / kStageBytes : kSkMaxStages;
    __host__ __device__ static uint32_t bytes(uint32_t stages)
    {
        return stages * kStageBytes > kPartial ? stages * kStageBytes : kPartial;
    }
};

// How the products of a row are summed (see above).
enum SkSum { SUM_CHAIN = 0, SUM_SHORT_CHAINS = 1, SUM_COMPENSATED = 2 };

// Stages of the ring, 0: as many as splitk_stages() says. Of f32 results of more than 64 rows a constant: 130 x 2048 x 1536 6.7
// us, with a number that only the launch knows 7.3, and 1021 x 7168 x 256 with eight 15.2 instead of 14.8.
template <bool F32, int SUM> constexpr uint32_t kSkStages = F32 && SUM != SUM_COMPENSATED ? 4 : 0;

// Tensor-memory buffers: short chains two accumulators per k block, in turn; else one accumulator for all of k.
template <int NT, int SUM> struct SkTmem {
    static constexpr uint32_t kBufs = SUM == SUM_CHAIN ? 1 : NT <= 32 ? 4 : 2;
    static constexpr uint32_t kUsed = SUM == SUM_CHAIN ? NT : 2 * NT * kBufs;
    static constexpr uint32_t kCols = kUsed <= 32 ? 32 : kUsed <= 64 ? 64 : kUsed <= 128 ? 128 : 256; // a power of two
    // warps that empty them, in fours, one per quarter of the lanes; compensated sums take a warp for 16 columns
    static constexpr uint32_t kAdders = SUM == SUM_COMPENSATED ? NT / 4 : 4;
    static constexpr uint32_t kThreads = (kAdders + 2) * 32;
    static constexpr uint32_t kMine = NT * 4 / kAdders; // columns of an adding warp
};

// Compensated (Kahan) sums of two neighbouring values at a time: s - c is the sum of the values added so far to within a
// rounding of it. An infinity makes c a NaN: a plain sum beside it tells.
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b)
{
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
constexpr uint64_t kNegate2 = 0x8000000080000000ull;
__device__ __forceinline__ void kahan2(uint64_t& s, uint64_t& c, uint64_t x)
{
    const uint64_t y = add2(x, c ^ kNegate2), t = add2(s, y);
    c = add2(add2(t, s ^ kNegate2), y ^ kNegate2);
    s = t;
}
__device__ __forceinline__ void kahan(float& s, float& c, float x)
{
    const float y = __fadd_rn(x, -c), t = __fadd_rn(s, y);
    c = __fadd_rn(__fadd_rn(t, -s), -y);
    s = t;
}
__device__ __forceinline__ float half2(uint64_t v, uint32_t i) { return __uint_as_float(static_cast<uint32_t>(v >> (32 * i))); }
__device__ __forceinline__ uint64_t pack2(uint32_t a, uint32_t b) { return static_cast<uint64_t>(b) << 32 | a; }

template <int NT, bool F32, int SUM>
__global__ void __launch_bounds__(SkTmem<NT, SUM>::kThreads)
gemm_splitk_kernel(const __grid_constant__ CUtensorMap map_b, const __grid_constant__ CUtensorMap map_a,
                   const SplitkParams p)
{
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    const uint32_t rank = cluster.block_rank(), splits = cluster.num_blocks();
    constexpr uint32_t kStageBytes = SkSmem<NT>::kStageBytes;
    constexpr uint32_t kTmemCols = SkTmem<NT, SUM>::kCols, kBufs = SkTmem<NT, SUM>::kBufs;
    constexpr uint32_t kAdders = SkTmem<NT, SUM>::kAdders, kMine = SkTmem<NT, SUM>::kMine;

    const uint32_t stages = kSkStages<F32, SUM> != 0 ? kSkStages<F32, SUM> : p.stages;

    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    float* part = reinterpret_cast<float*>(smem); // [NT][kSkPitch], after the ring
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + SkSmem<NT>::bytes(stages));
    uint64_t* empty_bar = full_bar + kSkMaxStages;
    uint64_t* acc_full = empty_bar + kSkMaxStages;
    uint64_t* acc_empty = acc_full + kBufs; // short chains
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + kBufs);
    volatile uint32_t* abort_flag = tmem_slot + 1;

    const uint32_t warp = threadIdx.x >> 5;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t n0 = blockIdx.y * 128, m0 = blockIdx.z * NT;
    const uint32_t kb0 = min(rank * p.kb_per_split, p.k_blocks), kb1 = min(kb0 + p.kb_per_split, p.k_blocks);

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < stages; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        for (uint32_t b = 0; b < kBufs; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], kAdders);
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 5) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    chain_begin();

    bool ready = true;
    if (warp == 4) {
        // ------------------------------------------------------------ producer --
        if (elect_one()) {
            uint32_t s = 0, ph = 0;
            for (uint32_t i = 0; i < kb1 - kb0; ++i) {
                if (!mbar_wait<true>(&empty_bar[s], ph ^ 1, abort_flag, p.err, ERR_SK_EMPTY_WAIT))
                    break;
                uint8_t* sb = smem + s * kStageBytes;
                mbar_expect_tx(&full_bar[s], kStageBytes);
                const int c0 = static_cast<int>(kb0 + i) * 64;
                tma_load_2d(sb, &map_b, &full_bar[s], c0, static_cast<int>(n0));
                tma_load_2d(sb + kTileBytes, &map_a, &full_bar[s], c0, static_cast<int>(m0));
                if (++s == stages) {
                    s = 0;
                    ph ^= 1;
                }
            }
        }
    } else if (warp == 5) {
        // ---------------------------------------------------------- MMA issuer --
        if (elect_one()) {
            // M = 128 weight rows, N = NT rows of A, bf16 x bf16 -> f32, both operands K-major
            constexpr uint32_t kIdesc
                = (1u << 4) | (1u << 7) | (1u << 10) | ((static_cast<uint32_t>(NT) >> 3) << 17) | ((kBM >> 4) << 24);
            bool ok = true;
            uint32_t s = 0, ph = 0;
            for (uint32_t i = 0; i < kb1 - kb0; ++i) {
                const uint32_t b = i % kBufs;
                if (SUM != SUM_CHAIN && !mbar_wait<true>(&acc_empty[b], ((i / kBufs) & 1) ^ 1, abort_flag, p.err, ERR_SK_ACC_EMPTY_WAIT)) {
                    ok = false;
                    break;
                }
                if (!mbar_wait<true>(&full_bar[s], ph, abort_flag, p.err, ERR_SK_FULL_WAIT)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t sb = smem_u32(smem + s * kStageBytes);
                const uint64_t db = operand_desc(sb), da = operand_desc(sb + kTileBytes);
#pragma unroll
                for (uint32_t j = 0; j < 4; ++j)
                    tc_mma_bf16(SUM != SUM_CHAIN ? tmem_base + (2 * b + j / 2) * NT : tmem_base, db + 2 * j, da + 2 * j, kIdesc,
                                (SUM != SUM_CHAIN ? j % 2 : i + j) > 0 ? 1u : 0u);
                tc_commit(&empty_bar[s]);
                if (SUM != SUM_CHAIN)
                    tc_commit(&acc_full[b]);
                if (++s == stages) {
                    s = 0;
                    ph ^= 1;
                }
            }
            if (ok && SUM == SUM_CHAIN)
                tc_commit(acc_full);
        }
    } else {
        // ------------------------------------- accumulators -> partial tile in smem --
        // this warp's lanes, and its first column
        const uint32_t quarter = warp % 4, c0 = (warp < 4 ? 0 : (warp - 2) / 4) * kMine;
        const uint32_t lanes = tmem_base + ((quarter * 32) << 16) + c0;
        float* const mine = part + c0 * kSkPitch + quarter * 32 + lane;
        if constexpr (SUM != SUM_CHAIN) {
            constexpr bool KAHAN = SUM == SUM_COMPENSATED;
            constexpr uint32_t kKept = KAHAN ? kMine / 2 : 1;
            uint64_t plain[kMine / 2], sum[kKept] = {}, rest[kKept] = {};
#pragma unroll
            for (uint32_t t = 0; t < kMine / 2; ++t)
                plain[t] = 0;
            for (uint32_t i = 0; i < kb1 - kb0; ++i) {
                const uint32_t b = i % kBufs;
                ready = __all_sync(0xffffffffu, mbar_wait(&acc_full[b], (i / kBufs) & 1, abort_flag, p.err, ERR_SK_ACC_WAIT));
                if (!ready)
                    break;
                tc_fence_after();
#pragma unroll
                for (uint32_t c = 0; c < kMine / 16; ++c) {
                    if (m0 + c0 + c * 16 < p.m) { // uniform
                        uint32_t v[16], w[16];
                        tc_ld16(lanes + 2 * b * NT + c * 16, v);
                        tc_ld16(lanes + (2 * b + 1) * NT + c * 16, w);
                        tc_ld_wait();
#pragma unroll
                        for (uint32_t t = 0; t < 8; ++t) {
                            const uint64_t x = add2(pack2(v[2 * t], v[2 * t + 1]), pack2(w[2 * t], w[2 * t + 1]));
                            plain[c * 8 + t] = add2(plain[c * 8 + t], x);
                            if constexpr (KAHAN)
                                kahan2(sum[c * 8 + t], rest[c * 8 + t], x);
                        }
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0)
                    mbar_arrive(&acc_empty[b]);
            }
            // every load of this CTA has been consumed (all adding warps have seen the last block): the ring is free
            ready = group_all(1, kAdders * 32, ready);
#pragma unroll
            for (uint32_t t = 0; t < kMine; ++t)
                if (ready && m0 + c0 + t < p.m) {
                    const float whole = half2(plain[t / 2], t % 2);
                    mine[t * kSkPitch]
                        = KAHAN && isfinite(whole) ? half2(sum[KAHAN ? t / 2 : 0], t % 2) - half2(rest[KAHAN ? t / 2 : 0], t % 2) : whole;
                }
        } else {
            ready = __all_sync(0xffffffffu, mbar_wait(acc_full, 0, abort_flag, p.err, ERR_SK_ACC_WAIT));
            tc_fence_after();
            if (ready) { // every load has been consumed: the ring is free
                const bool some = kb1 > kb0; // a rank past the end of k adds zeros
#pragma unroll
                for (uint32_t c = 0; c < NT / 16; ++c) {
                    if (m0 + c * 16 >= p.m)
                        break;
                    uint32_t v[16];
                    tc_ld16(lanes + c * 16, v);
                    tc_ld_wait();
#pragma unroll
                    for (uint32_t t = 0; t < 16; ++t)
                        mine[(c * 16 + t) * kSkPitch] = some ? __uint_as_float(v[t]) : 0.0f;
                }
            }
            tc_fence_before();
        }
    }
    cluster.sync(); // every partial tile is complete
    // rows of the tile are dealt out over the cluster's warps; a lane sums four features over the ranks, in order
    // (kept short: at decode sizes the code itself comes from HBM, and unrolling this over rows took longer)
    const float alpha = p.alpha == 0.0f ? 1.0f : p.alpha;
    const uint32_t rows = min(static_cast<uint32_t>(NT), p.m - m0);
    const uint32_t f = n0 + lane * 4;
    constexpr uint32_t kWarps = kAdders + 2;
    for (uint32_t t = rank * kWarps + warp; t < rows && *abort_flag == 0; t += splits * kWarps) {
        float4 v[kSkMaxSplits];
#pragma unroll
        for (uint32_t s = 0; s < kSkMaxSplits; ++s)
            v[s] = s < splits ? *reinterpret_cast<const float4*>(cluster.map_shared_rank(part, s) + t * kSkPitch + lane * 4)
                              : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        float a[4] = { v[0].x, v[0].y, v[0].z, v[0].w };
#pragma unroll
        for (uint32_t s = 1; s < kSkMaxSplits; ++s) {
            a[0] += v[s].x;
            a[1] += v[s].y;
            a[2] += v[s].z;
            a[3] += v[s].w;
        }
        if constexpr (SUM == SUM_COMPENSATED) {
            float sum[4] = { v[0].x, v[0].y, v[0].z, v[0].w }, rest[4] = {};
#pragma unroll
            for (uint32_t s = 1; s < kSkMaxSplits; ++s) {
                const float x[4] = { v[s].x, v[s].y, v[s].z, v[s].w };
#pragma unroll
                for (uint32_t q = 0; q < 4; ++q) {
                    kahan(sum[q], rest[q], x[q]);
                }
            }
#pragma unroll
            for (uint32_t q = 0; q < 4; ++q)
                a[q] = isfinite(a[q]) ? sum[q] - rest[q] : a[q];
        }
        const uint64_t at = static_cast<uint64_t>(m0 + t) * p.out_pitch + f;
        const uint32_t left = f < p.n ? min(4u, p.n - f) : 0u;
        if (p.beta != 0.0f || p.bias != nullptr || alpha != 1.0f) {
            for (uint32_t q = 0; q < left; ++q) {
                a[q] *= alpha;
                if (p.beta != 0.0f)
                    a[q] += p.beta * (F32 ? static_cast<const float*>(p.out)[at + q]
                                          : __bfloat162float(static_cast<const __nv_bfloat16*>(p.out)[at + q]));
                if (p.bias != nullptr)
                    a[q] += p.bias[f + q];
            }
        }
        if constexpr (F32) {
            float* o = static_cast<float*>(p.out) + at;
            if (left == 4 && (reinterpret_cast<uintptr_t>(o) & 15u) == 0)
                *reinterpret_cast<float4*>(o) = make_float4(a[0], a[1], a[2], a[3]);
            else
                for (uint32_t q = 0; q < left; ++q)
                    o[q] = a[q];
        } else {
            __nv_bfloat16* o = static_cast<__nv_bfloat16*>(p.out) + at;
            if (left == 4 && (reinterpret_cast<uintptr_t>(o) & 7u) == 0)
                *reinterpret_cast<uint2*>(o) = make_uint2(pack_bf16x2(a[0], a[1]), pack_bf16x2(a[2], a[3]));
            else
                for (uint32_t q = 0; q < left; ++q)
                    o[q] = __float2bfloat16(a[q]);
        }
    }
    cluster.sync(); // no CTA leaves while a peer still reads its partial tile
    if (warp == 5) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols)
                     : "memory");
    }
}

// A CTA alone on its SM takes as many stages as the k blocks of a rank can use (72 x 4096 x 4096: four stages 0.0163 ms,
// eight 0.0136). Two share an SM when there are more tiles than SMs, and when clusters of four or eight would take most of the
// SMs, since not every one finds its SMs free side by side then (33 x 4096 x 2048, 16 clusters of eight: 0.0133 ms with eight
// stages, 0.0090 with four; 809 x 4096 x 512, 36 of four: 0.0159 against 0.0118 with fewer tiles).
uint32_t splitk_stages(uint32_t nt, uint64_t tiles, uint32_t splits, uint32_t kb_per_split, uint64_t sms)
{
    const uint64_t ctas = tiles * splits;
    const bool alone = ctas <= (splits < 4 ? sms : splits == 4 ? sms * 7 / 8 : sms * 3 / 4);
    return std::min({ alone ? kSkMaxStages : 4u, kSkRing / (kTileBytes + nt * 128), kb_per_split });
}

template <int NT, bool F32, int SUM>
cudaError_t launch_splitk_instance(const CUtensorMap& mb, const CUtensorMap& ma, SplitkParams sp, dim3 grid,
                                   cudaStream_t stream)
{
    auto kernel = gemm_splitk_kernel<NT, F32, SUM>;
    sp.stages = kSkStages<F32, SUM> != 0
        ? kSkStages<F32, SUM>
        : splitk_stages(NT, static_cast<uint64_t>(grid.y) * grid.z, grid.x, sp.kb_per_split, device_sm_count());
    const size_t smem = 1024 + SkSmem<NT>::bytes(sp.stages) + 256, most = 1024 + SkSmem<NT>::bytes(SkSmem<NT>::kMostStages) + 256;
    static bool configured[64] = {}; // per instantiation and device
    int dev = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err != cudaSuccess)
        return err;
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(most));
        if (err != cudaSuccess)
            return err;
        if (dev >= 0 && dev < 64)
            configured[dev] = true;
    }
    return launch_chained_cluster(kernel, grid.x, grid, SkTmem<NT, SUM>::kThreads, smem, stream, mb, ma, sp);
}

uint64_t splitk_tiles(const GemmProblem& g, uint32_t nt) { return (g.n + 127ull) / 128 * ((g.a_rows + nt - 1) / nt); }

bool splitk_compensated(const GemmProblem& g) { return g.epilogue == EPI_STORE_F32 && g.a_rows <= 64; }

// Rows of A per tile: the fewest MMA columns that hold them, 64 above that (128 x 4096 x 2048: 0.0125 ms against
// 0.0145 with 128) as long as every tile can still be split. Compensated sums in smaller tiles as long as each can be split in
// four: adding up is what they wait for (33 x 2048 x 512: 0.0054 ms, with 32 rows 0.0066).
uint32_t splitk_tile_rows(const GemmProblem& g)
{
    if (splitk_compensated(g))
        for (uint32_t nt = 16; nt < 64; nt *= 2)
            if (4 * splitk_tiles(g, nt) <= device_sm_count())
                return nt;
    return g.a_rows <= 16 ? 16u : g.a_rows <= 32 ? 32u : 64u;
}

// Compensated sums for f32 results of decode batches, which the CUDA cores summed before; short chains for router logits of
// up to a few row tiles. A larger batch's had one chain over all of k before this kernel, and adding up outside the
// tensor core takes longer than the loads where every SM has a tile (4096 x 2048 x 8: 0.0128 against 0.0120 ms).
SkSum splitk_sum(const GemmProblem& g, uint32_t nt)
{
    if (g.epilogue != EPI_STORE_F32)
        return SUM_CHAIN;
    return splitk_compensated(g) ? SUM_COMPENSATED
        : nt == 64 && splitk_tiles(g, 128) <= 18 ? SUM_SHORT_CHAINS
                                                 : SUM_CHAIN;
}

// As many splits as fit one CTA per SM, two k blocks each at least; none for compensated sums of a short k, which a
// rounding per rank would leave further off (64 x 512 x 512: 6.4e-8, 5.8e-8 unsplit, on CUDA cores 6.2e-8).
uint32_t splitk_splits(const GemmProblem& g, uint32_t nt, uint64_t sms)
{
    const uint64_t tiles = splitk_tiles(g, nt);
    const uint32_t k_blocks = (g.k + 63) / 64;
    uint32_t splits = 1;
    while (splits < kSkMaxSplits && 2 * splits * tiles <= sms && 2 * (2 * splits) <= k_blocks
           && (splitk_sum(g, nt) != SUM_COMPENSATED || k_blocks > 8))
        splits *= 2;
    return splits;
}

// Tile rows of a problem that this kernel takes, 0: it does not. At least two CTAs per tile without exceeding one CTA
// per SM, since more tiles fill the device as they are; a long k is split with 128-row tiles too (2048 x 4096 x 512:
// 0.0207 against 0.0269 ms for the 128 x 256 kernel, but 512 x 2048 x 2048: 0.0163 against 0.0145).
uint32_t splitk_choice(const GemmProblem& g)
{
    const uint32_t nt = splitk_tile_rows(g);
    if (splitk_compensated(g) && g.k <= 4096) // whatever the tiles (longer sums were a chain: 64 x 7168 x 16384 0.071 / 0.056 ms)
        return nt;
    if (g.a_rows > 64 && g.k < 512) // nothing to split (1021 x 256 x 8: 0.0058 against 0.0046 ms in one tile per CTA)
        return 0;
    if (2 * splitk_tiles(g, nt) <= device_sm_count())
        return nt;
    return nt == 64 && g.k >= 2048 && 2 * splitk_tiles(g, 128) <= device_sm_count() ? 128u : 0u;
}

} // namespace

bool gemm_splitk_supported(const GemmProblem& g)
{
    return !g.nvfp4 && !g.gated && g.tile_expert == nullptr && g.groups == 1 && g.group_scale == nullptr && g.k % 8 == 0
        && (g.epilogue == EPI_STORE_BF16 || g.epilogue == EPI_STORE_F32)
        && (reinterpret_cast<uintptr_t>(g.a) & 15u) == 0 && (reinterpret_cast<uintptr_t>(g.b) & 15u) == 0
        && g.a_pitch_bytes % 16 == 0 && g.b_pitch_bytes % 16 == 0
        && splitk_choice(g) != 0;
}

// 200 x 4096 x 2048, 64 rows a tile: 11.8 us both; 130 x 4096 x 2048, 96 rows: 11.1, measured 10.5.
float gemm_splitk_estimate(const GemmProblem& g, uint32_t nt, uint32_t sms)
{
    const uint64_t tiles = splitk_tiles(g, nt);
    if (tiles > sms)
        return 1e30f;
    const uint32_t splits = splitk_splits(g, nt, sms), kbs = ((g.k + 63) / 64 + splits - 1) / splits;
    const float output = g.beta != 0.0f ? 0.01f * nt / splits : 0.0f;
    return 4.6f + output + 0.028f * nt + kbs * (1.1f / splitk_stages(nt, tiles, splits, 8, sms) + 0.0003f * nt + 0.01f);
}

cudaError_t launch_gemm_splitk(const GemmProblem& g, uint32_t rows, cudaStream_t stream, const char** why)
{
    SplitkParams sp {};
    sp.m = static_cast<uint32_t>(g.a_rows);
    sp.n = g.n;
    sp.k_blocks = (g.k + 63) / 64;
    sp.out = g.out;
    sp.out_pitch = g.out_pitch_elems;
    sp.alpha = g.alpha;
    sp.beta = g.beta;
    sp.bias = g.bias;
    sp.err = device_error_word();
    const uint32_t nt = rows != 0 ? rows : splitk_choice(g);
    const uint64_t tiles = splitk_tiles(g, nt);
    const uint32_t splits = splitk_splits(g, nt, device_sm_count());
    sp.kb_per_split = (sp.k_blocks + splits - 1) / splits;
    CUtensorMap mb, ma;
    if (!make_operand_map(&mb, false, g.b, g.k, g.n, g.b_pitch_bytes, 128)
        || !make_operand_map(&ma, false, g.a, g.k, g.a_rows, g.a_pitch_bytes, nt)) {
        if (why != nullptr)
            *why = "cuTensorMapEncodeTiled failed";
        return cudaErrorInvalidValue;
    }
    const dim3 grid(splits, (g.n + 127) / 128, static_cast<uint32_t>((g.a_rows + nt - 1) / nt));
    const auto launch = [&](auto kernel) { return kernel(mb, ma, sp, grid, stream); };
    if (g.epilogue != EPI_STORE_F32)
        return launch(nt == 16 ? launch_splitk_instance<16, false, SUM_CHAIN>
            : nt == 32         ? launch_splitk_instance<32, false, SUM_CHAIN>
            : nt == 64         ? launch_splitk_instance<64, false, SUM_CHAIN>
            : nt == 96         ? launch_splitk_instance<96, false, SUM_CHAIN>
                               : launch_splitk_instance<128, false, SUM_CHAIN>);
    switch (splitk_sum(g, nt)) {
    case SUM_COMPENSATED:
        return launch(nt == 16 ? launch_splitk_instance<16, true, SUM_COMPENSATED>
            : nt == 32         ? launch_splitk_instance<32, true, SUM_COMPENSATED>
                               : launch_splitk_instance<64, true, SUM_COMPENSATED>);
    case SUM_SHORT_CHAINS: return launch(launch_splitk_instance<64, true, SUM_SHORT_CHAINS>);
    default: return launch(nt == 64 ? launch_splitk_instance<64, true, SUM_CHAIN> : launch_splitk_instance<128, true, SUM_CHAIN>);
    }
}

} // namespace qs3
