// Dense bf16 GEMM  D[m, n] = alpha * sum_k A[m, k] * B[n, k] (+ beta * D) (+ bias[n])  for the
// projection lane (qscb_gemm_bf16: router logits, shared expert in bf16 plans, LM head).
//
// The one-tile-per-CTA kernel of gemm.cu issues 128 x 128 instructions and relies on two
// co-resident CTAs to hide its epilogue. This kernel is the large-problem variant:
//
//   persistent   one CTA per SM walks the output tiles (row tile fastest, so the CTAs of a wave
//                share one or two B panels through L2)
//   128 x bn     tcgen05.mma kind::f16 with N = bn columns, 32 to 256 (256: the widest single-CTA instruction), as many as
//                gemm_dense_choice() finds quickest
//   TMEM         two 256-column f32 accumulators: the epilogue of tile i (eight warps, two per
//                lane quadrant) overlaps the main loop of tile i + 1
//   smem         192 KB ring of stages, each A 128 x 64 bf16 (16 KB) + B bn x 64, filled by TMA with the 128-byte swizzle;
//                32 KB through which the output goes (dense_epilogue)
//
// Rows past the end of A or B are zero-filled by TMA and masked in the epilogue. Every wait is
// bounded; on expiry the kernel records a code and leaves through the normal teardown.
#include "tcgen05.cuh"

#include <cooperative_groups.h>

#include <algorithm>

namespace qs3 {
namespace {

using namespace tc;

constexpr int kDnThreads = 320; // warps 0-7 epilogue, 8 producer, 9 MMA issuer
constexpr uint32_t kDnBN = 256;
constexpr uint32_t kDnRing = 12 * kTileBytes; // stages of an A tile + bn rows of B: four of 256 rows, up to eight of fewer
constexpr uint32_t kDnMaxStages = 8;
__host__ __device__ constexpr uint32_t dense_stages(uint32_t bn)
{
    return kDnRing / (kTileBytes + bn * 128) < kDnMaxStages ? kDnRing / (kTileBytes + bn * 128) : kDnMaxStages;
}
constexpr uint32_t kDnTmemCols = 512;
constexpr uint32_t kDnOutBytes = 2048;            // staging of a warp's 32 rows x 64 bytes of output
constexpr uint32_t kDnStaging = 8 * 2 * kDnOutBytes; // two per epilogue warp

enum : uint32_t {
    ERR_DN_FULL_WAIT = 0x55000001u,
    ERR_DN_EMPTY_WAIT = 0x55000002u,
    ERR_DN_ACC_FULL_WAIT = 0x55000003u,
    ERR_DN_ACC_EMPTY_WAIT = 0x55000004u,
};

// Epilogue of one output tile: 128 accumulator lanes (rows from row0) x bn columns (from col0), by eight warps, two per
// quarter of the lanes. A lane holds a row, so a warp's store of 16 bytes a lane touches 32 rows, and every 32-byte sector
// is written twice; of a short k this takes longer than the products. With TMA a warp gathers 64 bytes of each of its rows
// in shared memory (64-byte swizzle, no bank conflicts) and has them written, two such stores in flight: 4096 x 512 x 8192
// 50 -> 39 us, 3001 x 2048 x 4096 42.5 -> 40.9. The last columns of a tile are taken as the last 64 bytes, which may write some
// columns twice, with the same values; rows and columns past the end are clipped. beta reads the output, and an output that
// TMA cannot address is stored row by row.
template <int EPI, bool TMA>
__device__ __forceinline__ void dense_epilogue(const TcParams& p, const CUtensorMap* map_o, uint8_t* staging, uint32_t& stores,
                                               uint32_t tmem_acc, uint32_t warp, uint32_t lane, uint32_t row0, uint32_t col0,
                                               uint32_t bn)
{
    const uint32_t quad = warp & 3, half = warp >> 2;
    if constexpr (!TMA) {
        // the tile's columns as a problem of their own: this epilogue works in units of 128 of them
        TcParams q = p;
        q.n = min(bn, p.n - col0);
        q.out = static_cast<uint8_t*>(p.out) + static_cast<uint64_t>(col0) * (EPI == EPI_STORE_F32 ? 4 : 2);
        if (p.bias != nullptr)
            q.bias = p.bias + col0;
        const int nrows = static_cast<int>(min(static_cast<uint32_t>(kBM), p.dense_rows - row0));
#pragma unroll
        for (uint32_t h = 0; h < 2; ++h)
            epilogue_tile<false, EPI, 2>(q, tmem_acc + h * kBN, quad, lane, 0, static_cast<int>(row0), nrows, h, half);
        return;
    }
    if (row0 + quad * 32 >= p.dense_rows)
        return;
    constexpr uint32_t kCols = EPI == EPI_STORE_F32 ? 16 : 32;
    const uint32_t cols = min(bn, p.n - col0);
    const float scale = p.alpha == 0.0f ? 1.0f : p.alpha;
    for (uint32_t c = half * kCols; c < cols; c += 2 * kCols) {
        const uint32_t at = min(c, bn - kCols);
        uint32_t v[kCols];
        tc_ld16(tmem_acc + ((quad * 32) << 16) + at, v);
        if constexpr (kCols == 32)
            tc_ld16(tmem_acc + ((quad * 32) << 16) + at + 16, v + 16);
        tc_ld_wait();
        float f[kCols];
#pragma unroll
        for (uint32_t i = 0; i < kCols; ++i) {
            f[i] = __uint_as_float(v[i]) * scale;
            if (p.bias != nullptr && col0 + at + i < p.n)
                f[i] += p.bias[col0 + at + i];
        }
        uint8_t* buf = staging + (stores++ & 1) * kDnOutBytes;
        if (lane == 0) // the store before the last has left its buffer
            asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
        __syncwarp();
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j) {
            uint4 w;
            if constexpr (EPI == EPI_STORE_F32)
                w = make_uint4(__float_as_uint(f[4 * j]), __float_as_uint(f[4 * j + 1]), __float_as_uint(f[4 * j + 2]),
                               __float_as_uint(f[4 * j + 3]));
            else
                w = make_uint4(pack_bf16x2(f[8 * j], f[8 * j + 1]), pack_bf16x2(f[8 * j + 2], f[8 * j + 3]),
                               pack_bf16x2(f[8 * j + 4], f[8 * j + 5]), pack_bf16x2(f[8 * j + 6], f[8 * j + 7]));
            *reinterpret_cast<uint4*>(buf + lane * 64 + ((j ^ (lane >> 1 & 3)) << 4)) = w;
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) {
            asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(
                             reinterpret_cast<uint64_t>(map_o)),
                         "r"(smem_u32(buf)), "r"(col0 + at), "r"(row0 + quad * 32)
                         : "memory");
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        }
    }
}

template <int EPI, bool TMA>
__global__ void __launch_bounds__(kDnThreads, 1)
gemm_dense_bf16_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                       const __grid_constant__ CUtensorMap map_o, const TcParams p, const uint32_t tiles_m, const uint32_t tiles_n, const uint32_t bn)
{
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    uint8_t* staging = smem + kDnRing; // [8 warps][2]
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(staging + (TMA ? kDnStaging : 0));
    uint64_t* empty_bar = full_bar + kDnMaxStages;
    uint64_t* acc_full = empty_bar + kDnMaxStages;
    uint64_t* acc_empty = acc_full + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
    volatile uint32_t* abort_flag = tmem_slot + 1;
    const uint32_t stage_bytes = kTileBytes + bn * 128, stages = dense_stages(bn);

    const uint32_t warp = threadIdx.x >> 5;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t total = tiles_m * tiles_n;

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < stages; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], 8); // one arrival per epilogue warp
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 9) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(kDnTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    chain_begin();

    if (warp == 8) {
        // ------------------------------------------------------------ producer --
        if (elect_one()) {
            uint32_t s = 0, ph = 0;
            bool ok = true;
            for (uint32_t t = blockIdx.x; t < total && ok; t += gridDim.x) {
                const int row0 = static_cast<int>((t % tiles_m) * kBM);
                const int col0 = static_cast<int>((t / tiles_m) * bn);
                for (uint32_t kb = 0; kb < p.k_blocks; ++kb) {
                    if (!mbar_wait<true>(&empty_bar[s], ph ^ 1, abort_flag, p.err, ERR_DN_EMPTY_WAIT)) {
                        ok = false;
                        break;
                    }
                    uint8_t* sa = smem + s * stage_bytes;
                    mbar_expect_tx(&full_bar[s], stage_bytes);
                    const int c0 = static_cast<int>(kb) * 64;
                    tma_load_2d(sa, &map_a, &full_bar[s], c0, row0);
                    tma_load_2d(sa + kTileBytes, &map_b, &full_bar[s], c0, col0);
                    tma_load_2d(sa + kTileBytes + bn * 64, &map_b, &full_bar[s], c0, col0 + static_cast<int>(bn / 2));
                    if (++s == stages) {
                        s = 0;
                        ph ^= 1;
                    }
                }
            }
        }
    } else if (warp == 9) {
        // ---------------------------------------------------------- MMA issuer --
        if (elect_one()) {
            // M = 128, N = bn, bf16 x bf16 -> f32, both operands K-major
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((bn >> 3) << 17) | ((kBM >> 4) << 24);
            uint32_t s = 0, ph = 0, u = 0;
            bool ok = true;
            for (uint32_t t = blockIdx.x; t < total && ok; t += gridDim.x, ++u) {
                const uint32_t buf = u & 1;
                if (!mbar_wait<true>(&acc_empty[buf], ((u >> 1) & 1) ^ 1, abort_flag, p.err, ERR_DN_ACC_EMPTY_WAIT))
                    break;
                tc_fence_after();
                const uint32_t d = tmem_base + buf * kDnBN;
                for (uint32_t kb = 0; kb < p.k_blocks; ++kb) {
                    if (!mbar_wait<true>(&full_bar[s], ph, abort_flag, p.err, ERR_DN_FULL_WAIT)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t sa = smem_u32(smem + s * stage_bytes);
                    const uint64_t da = operand_desc(sa);
                    const uint64_t db = operand_desc(sa + kTileBytes); // bn rows: two tiles back to back
#pragma unroll
                    for (uint32_t j = 0; j < 4; ++j)
                        tc_mma_bf16(d, da + 2 * j, db + 2 * j, idesc, (kb > 0 || j > 0) ? 1u : 0u);
                    tc_commit(&empty_bar[s]);
                    if (++s == stages) {
                        s = 0;
                        ph ^= 1;
                    }
                }
                if (ok)
                    tc_commit(&acc_full[buf]);
            }
        }
    } else {
        // ------------------------------------------------------------ epilogue --
        uint32_t u = 0, stores = 0;
        for (uint32_t t = blockIdx.x; t < total; t += gridDim.x, ++u) {
            const uint32_t buf = u & 1;
            const bool ready = __all_sync(
                0xffffffffu, mbar_wait(&acc_full[buf], (u >> 1) & 1, abort_flag, p.err, ERR_DN_ACC_FULL_WAIT));
            if (!ready)
                break;
            tc_fence_after();
            dense_epilogue<EPI, TMA>(p, &map_o, staging + warp * 2 * kDnOutBytes, stores, tmem_base + buf * kDnBN, warp, lane,
                                (t % tiles_m) * kBM, (t / tiles_m) * bn, bn);
            tc_fence_before();
            __syncwarp();
            if (lane == 0)
                mbar_arrive(&acc_empty[buf]);
        }
        if (lane == 0)
            asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); // stores done before shared memory goes away
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 9) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kDnTmemCols)
                     : "memory");
    }
}

// ---- CTA-pair variant ---------------------------------------------------------------------
//
// A 128 x 256 tile needs (128 + 256) operand rows per 2 * 128 * 256 products per k: at 1.3 PFLOP/s
// that is 15 TB/s out of L2, which is what bounds the kernel above. Here two CTAs of a cluster
// (two SMs) compute one 256 x 256 tile with cta_group::2 instructions: each loads its own 128
// rows of A and HALF of the 256 B rows, the tensor cores of both SMs read both halves, and each
// CTA ends up with its 128 output rows in its own tensor memory. Operand traffic per product
// drops by a third. Every load has one destination CTA: each CTA's own TMA loads (cta_group::2
// form) signal the barrier of the pair's first CTA, which issues the MMAs for both.
//
//   barriers  full[s]      first CTA only: its expect_tx covers both CTAs' tiles of the stage
//             empty[s]     one per CTA: the first CTA commits to its own and to its peer's
//             acc_full[b]  one per CTA, same way;  acc_empty[b] first CTA only, 16 arrivals
//                          (eight epilogue warps of each CTA, the peer's through cluster addresses)
constexpr uint32_t kPrKbs = 2;                              // k blocks (of 64) per stage
constexpr uint32_t kPrStageBytes = kPrKbs * 2 * kTileBytes; // per CTA and k block: A 128 x 64, B 128 x 64
constexpr uint32_t kPrStages = 3;

__device__ __forceinline__ uint32_t cluster_addr(const void* local, uint32_t cta_rank)
{
    uint32_t remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_u32(local)), "r"(cta_rank));
    return remote;
}

// TMA tile load whose completion bytes are counted on a barrier that may live in the peer CTA.
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const CUtensorMap* map, uint32_t bar_cluster_addr, int c0,
                                                 int c1)
{
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
                 " [%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(dst)),
                 "l"(reinterpret_cast<uint64_t>(map)), "r"(bar_cluster_addr), "r"(c0), "r"(c1)
                 : "memory");
}

__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar_cluster_addr)
{
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar_cluster_addr) : "memory");
}

__device__ __forceinline__ void tc_commit_pair(uint32_t bar_cluster_addr)
{
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar_cluster_addr)
                 : "memory");
}

template <int EPI, bool TMA>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kDnThreads, 1)
gemm_dense_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                       const __grid_constant__ CUtensorMap map_o, const TcParams p, const uint32_t tiles_m,
                       const uint32_t tiles_n, const uint32_t bn)
{
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    const uint32_t rank = cluster.block_rank(); // 0: issues the MMAs of the pair

    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    uint8_t* staging = smem + kPrStages * kPrStageBytes; // [8 warps][2]
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(staging + (TMA ? kDnStaging : 0));
    uint64_t* empty_bar = full_bar + kPrStages;
    uint64_t* acc_full = empty_bar + kPrStages;
    uint64_t* acc_empty = acc_full + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
    volatile uint32_t* abort_flag = tmem_slot + 1;

    const uint32_t warp = threadIdx.x >> 5;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t total = tiles_m * tiles_n;
    const uint32_t pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < kPrStages; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], 16);
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    cluster.sync(); // both CTAs resident and their barriers initialised before anything is signalled
    if (warp == 9) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(kDnTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    cluster.sync();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    chain_begin();

    if (warp == 8) {
        // ------------------------------------------------------------ producer --
        if (elect_one()) {
            uint32_t s = 0, ph = 0;
            bool ok = true;
            for (uint32_t t = pair; t < total && ok; t += pairs) {
                const int row0 = static_cast<int>((t % tiles_m) * 256 + rank * 128);
                const int col0 = static_cast<int>((t / tiles_m) * bn + rank * (bn / 2));
                for (uint32_t kb = 0; kb < p.k_blocks; kb += kPrKbs) {
                    if (!mbar_wait<true>(&empty_bar[s], ph ^ 1, abort_flag, p.err, ERR_DN_EMPTY_WAIT)) {
                        ok = false;
                        break;
                    }
                    const uint32_t nkb = min(kPrKbs, p.k_blocks - kb);
                    uint8_t* sa = smem + s * kPrStageBytes;
                    if (rank == 0)
                        mbar_expect_tx(&full_bar[s], nkb * (2 * kTileBytes + bn * 128)); // both CTAs' A and B tiles
                    const uint32_t bar = cluster_addr(&full_bar[s], 0);
                    for (uint32_t q = 0; q < nkb; ++q) {
                        const int c0 = static_cast<int>(kb + q) * 64;
                        tma_load_2d_pair(sa + q * 2 * kTileBytes, &map_a, bar, c0, row0);
                        tma_load_2d_pair(sa + q * 2 * kTileBytes + kTileBytes, &map_b, bar, c0, col0);
                    }
                    if (++s == kPrStages) {
                        s = 0;
                        ph ^= 1;
                    }
                }
            }
        }
    } else if (warp == 9) {
        // ---------------------------------------------------------- MMA issuer --
        if (rank == 0 && elect_one()) {
            // M = 256 (128 rows in each CTA), N = bn (half of the B rows from each CTA)
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((bn >> 3) << 17) | ((256u >> 4) << 24);
            uint32_t s = 0, ph = 0, u = 0;
            bool ok = true;
            for (uint32_t t = pair; t < total && ok; t += pairs, ++u) {
                const uint32_t buf = u & 1;
                if (!mbar_wait<true>(&acc_empty[buf], ((u >> 1) & 1) ^ 1, abort_flag, p.err, ERR_DN_ACC_EMPTY_WAIT))
                    break;
                tc_fence_after();
                const uint32_t d = tmem_base + buf * kDnBN;
                for (uint32_t kb = 0; kb < p.k_blocks; kb += kPrKbs) {
                    if (!mbar_wait<true>(&full_bar[s], ph, abort_flag, p.err, ERR_DN_FULL_WAIT)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t nkb = min(kPrKbs, p.k_blocks - kb);
                    for (uint32_t q = 0; q < nkb; ++q) {
                        const uint32_t sa = smem_u32(smem + s * kPrStageBytes + q * 2 * kTileBytes);
                        const uint64_t da = operand_desc(sa);
                        const uint64_t db = operand_desc(sa + kTileBytes);
#pragma unroll
                        for (uint32_t j = 0; j < 4; ++j) {
                            const uint32_t acc = (kb + q > 0 || j > 0) ? 1u : 0u;
                            asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %4, 0;\n\t"
                                         "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, q;\n\t}" ::"r"(d),
                                         "l"(da + 2 * j), "l"(db + 2 * j), "r"(idesc), "r"(acc)
                                         : "memory");
                        }
                    }
                    tc_commit_pair(cluster_addr(&empty_bar[s], 0));
                    tc_commit_pair(cluster_addr(&empty_bar[s], 1));
                    if (++s == kPrStages) {
                        s = 0;
                        ph ^= 1;
                    }
                }
                if (ok) {
                    tc_commit_pair(cluster_addr(&acc_full[buf], 0));
                    tc_commit_pair(cluster_addr(&acc_full[buf], 1));
                }
            }
        }
    } else {
        // ------------------------------------------------------------ epilogue --
        uint32_t u = 0, stores = 0;
        for (uint32_t t = pair; t < total; t += pairs, ++u) {
            const uint32_t buf = u & 1;
            const bool ready = __all_sync(
                0xffffffffu, mbar_wait(&acc_full[buf], (u >> 1) & 1, abort_flag, p.err, ERR_DN_ACC_FULL_WAIT));
            if (!ready)
                break;
            tc_fence_after();
            const uint32_t row0 = (t % tiles_m) * 256 + rank * 128;
            if (row0 < p.dense_rows)
                dense_epilogue<EPI, TMA>(p, &map_o, staging + warp * 2 * kDnOutBytes, stores, tmem_base + buf * kDnBN, warp, lane, row0,
                                    (t / tiles_m) * bn, bn);
            tc_fence_before();
            __syncwarp();
            if (lane == 0)
                mbar_arrive_cluster(cluster_addr(&acc_empty[buf], 0));
        }
        if (lane == 0)
            asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); // stores done before shared memory goes away
    }

    tc_fence_before();
    cluster.sync(); // the pair's tensor memory is idle in both CTAs
    if (warp == 9) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kDnTmemCols)
                     : "memory");
    }
}

template <int EPI, bool TMA>
cudaError_t launch_pair_instance(const CUtensorMap& ma, const CUtensorMap& mb, const CUtensorMap& mo, const TcParams& tp,
                                 uint32_t tiles_m, uint32_t tiles_n, uint32_t bn, cudaStream_t stream)
{
    auto kernel = gemm_dense_pair_kernel<EPI, TMA>;
    constexpr size_t smem = 1024 + kPrStages * kPrStageBytes + (TMA ? kDnStaging : 0) + 256;
    static bool configured[64] = {};
    int dev = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err != cudaSuccess)
        return err;
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
        if (err != cudaSuccess)
            return err;
        if (dev >= 0 && dev < 64)
            configured[dev] = true;
    }
    const uint32_t pairs = std::min(tiles_m * tiles_n, device_sm_count() / 2);
    return launch_chained(kernel, dim3(2 * pairs), kDnThreads, smem, stream, ma, mb, mo, tp, tiles_m, tiles_n, bn);
}

template <int EPI, bool TMA>
cudaError_t launch_dense_instance(const CUtensorMap& ma, const CUtensorMap& mb, const CUtensorMap& mo, const TcParams& tp,
                                  uint32_t tiles_m, uint32_t tiles_n, uint32_t bn, cudaStream_t stream)
{
    auto kernel = gemm_dense_bf16_kernel<EPI, TMA>;
    constexpr size_t smem = 1024 + kDnRing + (TMA ? kDnStaging : 0) + 256;
    static bool configured[64] = {};
    int dev = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err != cudaSuccess)
        return err;
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
        if (err != cudaSuccess)
            return err;
        if (dev >= 0 && dev < 64)
            configured[dev] = true;
    }
    const uint32_t grid = std::min(tiles_m * tiles_n, device_sm_count());
    return launch_chained(kernel, dim3(grid), kDnThreads, smem, stream, ma, mb, mo, tp, tiles_m, tiles_n, bn);
}

} // namespace

bool gemm_dense_bf16_supported(const GemmProblem& g)
{
    return !g.nvfp4 && !g.gated && g.tile_expert == nullptr && g.groups == 1 && g.group_scale == nullptr && g.a_rows > 64
        && g.k % 64 == 0 && g.k >= 64 && g.n >= 128 && (g.epilogue == EPI_STORE_BF16 || g.epilogue == EPI_STORE_F32)
        && (reinterpret_cast<uintptr_t>(g.a) & 15u) == 0 && (reinterpret_cast<uintptr_t>(g.b) & 15u) == 0
        && g.a_pitch_bytes % 16 == 0 && g.b_pitch_bytes % 16 == 0
        && (g.a_rows + kBM - 1) / kBM * ((g.n + 31ull) / 32) < (1ull << 31);
}

// What computes a dense problem of more than 64 rows: the kernel, and the columns (rows of A for the split one) of a tile, by
// an estimate of its time in microseconds. Fitted to 72..3001 rows, k 512..4096, 512..8192 features, operands from HBM; with
// operands in L2 the times are 0.7 to 1.0 of it, for shorter k 0.65 to 1.35. What it has to get right is the order. A CTA's operands come through a ring that holds 192 KB, a trip
// of 1.1 us, so a k block takes 1.1 us / stages however few SMs work: narrow tiles are quick by themselves, wide ones move
// fewer bytes, and the rounds of the SMs decide between them.
//   one CTA per tile of 128 x c   2.9 + c / 80 + rounds (1 + k blocks (1.1 / stages + 0.0003 c))
//   a pair of CTAs, 256 x c       6.8 + rounds (1.5 + k blocks (0.15 + 0.00062 c)), a round not under the 3.5 c / 256 that
//                                 its output takes
//   split k (gemm_splitk.cu)      bf16 results only: f32 results have their own choice there
// With beta the first two read and store the output row by row, 1.5 us more, split k along the rows, 0.01 times its rows a rank
// (127 x 1024 x 512: split 5.8 us, one CTA per tile 8.5; 1500 x 512 x 128: 6.0 and 7.6; over 91 shapes the choice takes 1 %
// longer than the quickest, without beta over 54 as well).
// A sum over all of k in one accumulator is off by 2e-6 at k = 2048, a rank's share by less; rounding to bf16 by 2e-3, which
// is all that 106 shapes show against 64 bits, whichever kernel computes them (within 3e-6 of that error).
// Before, by the number of 128 x 256 tiles: 300 x 4096 x 4096 25.9 -> 16.8 us, 1200 x 4096 x 4096 46.3 -> 37.6,
// 800 x 4096 x 2048 26.0 -> 18.0, 200 x 512 x 2048 6.9 -> 5.7, 2000 x 512 x 8192 26.9 -> 23.
DenseChoice gemm_dense_choice(const GemmProblem& g)
{
    // (32 bits hold the tiles: gemm_dense_bf16_supported; a call of a small problem takes as long on the host as on the device)
    const uint32_t sms = device_sm_count(), m = static_cast<uint32_t>(g.a_rows);
    const float kb = static_cast<float>(g.k / 64), by_rows = g.beta != 0.0f ? 1.5f : 0.0f;
    const auto rounds = [](uint32_t tiles, uint32_t at_once) { return static_cast<float>((tiles + at_once - 1) / at_once); };
    const uint32_t tiles_m = (m + kBM - 1) / kBM, pair_m = (m + 255) / 256;
    DenseChoice best { DENSE_ONE, kDnBN };
    float least = 1e30f;
    const auto offer = [&](DenseKernel kernel, uint32_t width, float time) {
        if (time < least) {
            least = time;
            best = { kernel, width };
        }
    };
    for (uint32_t c = kDnBN; c >= 32; c -= 16) {
        const float r = rounds(tiles_m * ((g.n + c - 1) / c), sms);
        offer(DENSE_ONE, c, 2.9f + by_rows + 0.0125f * c + r * (1.0f + kb * (1.1f / dense_stages(c) + 0.0003f * c)));
    }
    for (uint32_t c = 256; c >= 128; c -= 32) {
        const float r = rounds(pair_m * ((g.n + c - 1) / c), sms / 2);
        offer(DENSE_PAIR, c, 6.8f + by_rows + r * (1.5f + std::max(kb * (0.15f + 0.00062f * c), 3.5f * c / 256)));
    }
    if (g.epilogue == EPI_STORE_BF16)
        for (uint32_t nt : { 64u, 96u, 128u })
            offer(DENSE_SPLIT, nt, gemm_splitk_estimate(g, nt, sms));
    return best;
}

cudaError_t launch_gemm_dense_bf16(const GemmProblem& g, DenseChoice choice, cudaStream_t stream, const char** why)
{
    TcParams tp {};
    tp.n = g.n;
    tp.k_blocks = g.k / 64;
    tp.b_rows = g.n;
    tp.dense_rows = static_cast<uint32_t>(g.a_rows);
    tp.out = g.out;
    tp.out_pitch = g.out_pitch_elems;
    tp.alpha = g.alpha;
    tp.beta = g.beta;
    tp.bias = g.bias;
    tp.err = device_error_word();
    const uint32_t tiles_m = static_cast<uint32_t>((g.a_rows + kBM - 1) / kBM);
    const bool pair = choice.kernel == DENSE_PAIR;
    const uint32_t pair_m = static_cast<uint32_t>((g.a_rows + 255) / 256);
    const uint32_t bn = choice.width, tiles_n = (g.n + bn - 1) / bn;
    // Several row tiles read a B panel from neighbouring SMs; over several rounds a chained start, which lets the next problem
    // begin on the SMs that are done first, sets them out of step (156 rows x 2048 x 151936, 8 rounds: 0.152 against 0.146 ms;
    // 300 x 4096 x 50000, 4 rounds: 0.129 against 0.125). In one or two it pays (1000 x 512 x 8192: 0.0114, unchained 0.0123).
    const UnchainedScope in_step(tiles_m > 1 && static_cast<uint64_t>(tiles_m) * tiles_n > 3ull * device_sm_count());
    CUtensorMap ma, mb;
    if (!make_operand_map(&ma, false, g.a, g.k, g.a_rows, g.a_pitch_bytes, kBM)
        || !make_operand_map(&mb, false, g.b, g.k, g.n, g.b_pitch_bytes, bn / 2)) {
        if (why != nullptr)
            *why = "cuTensorMapEncodeTiled failed";
        return cudaErrorInvalidValue;
    }
    CUtensorMap mo = ma;
    const bool f32 = g.epilogue == EPI_STORE_F32;
    // In a single round nothing hides the way through shared memory, and a smaller block starts sooner: 200 x 512 x 4096
    // 5.0 us, stored directly 4.7; 845 x 512 x 4096 8.3 / 7.6. Not so f32 results (1021 x 2048 x 512: 8.9 / 9.3).
    const bool several = pair || f32 || static_cast<uint64_t>(tiles_m) * tiles_n > device_sm_count();
    const bool tma = several && g.beta == 0.0f && make_output_map(&mo, f32, g.out, g.n, g.a_rows, g.out_pitch_elems);
    const auto launch = [&](auto kernel, uint32_t rows) { return kernel(ma, mb, mo, tp, rows, tiles_n, bn, stream); };
    if (pair)
        return tma ? launch(f32 ? launch_pair_instance<EPI_STORE_F32, true> : launch_pair_instance<EPI_STORE_BF16, true>, pair_m)
                   : launch(f32 ? launch_pair_instance<EPI_STORE_F32, false> : launch_pair_instance<EPI_STORE_BF16, false>, pair_m);
    return tma ? launch(f32 ? launch_dense_instance<EPI_STORE_F32, true> : launch_dense_instance<EPI_STORE_BF16, true>, tiles_m)
               : launch(f32 ? launch_dense_instance<EPI_STORE_F32, false> : launch_dense_instance<EPI_STORE_BF16, false>, tiles_m);
}

} // namespace qs3
