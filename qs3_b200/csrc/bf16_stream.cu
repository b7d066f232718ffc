// Grouped bf16 GEMM of the routed experts: weight streaming with the operands swapped (weight rows are the M side of
// the MMA, the expert's token tile of NT padded rows the N side). The plain variant also takes dense problems of at
// most 64 rows with many features (the LM head of a decode batch): one row tile, no tables.
//
//   unit   one token tile x 256 weight rows of its expert: gated: 128 gate rows and the 128 up rows of the same
//          features (two accumulators with the same lanes, so SwiGLU needs no exchange); plain: 256 features
//   grid   persistent, one CTA per SM, every gridDim.x-th unit: the CTAs of a round hold neighbouring units, so a
//          token tile and the weights of an expert with several tiles are read by several SMs at about the same
//          time (contiguous ranges of units instead: gate_up of the 2048-token case below 0.425 ms)
//   smem   ring of stages: two weight tiles 128 x 64 (32 KB) + token tile NT x 64
//   TMEM   two buffers of two NT-column accumulators (lane = weight row, column = token)
//   warps  0-3 epilogue, 4 producer (TMA; token rows by gather4), 5 MMA issuer
//
// Bound by HBM while experts have few rows: hit experts * weight bytes. A 128 x 128 tile per CTA moved as many token
// (mostly padding) as weight bytes into shared memory and multiplied the padding; here a stage moves NT / 256 as
// many. 33 tokens x 128 experts top-8 (hidden 2048, intermediate 768): gate_up 0.148 -> 0.114 (6.2 TB/s), down
// 0.072 -> 0.059 ms; 2048 tokens x 512 experts top-10 (intermediate 512): gate_up 0.443 -> 0.370 (5.8 TB/s), down
// 0.222 -> 0.174 ms. The token rows of experts with few of them come by gather4 straight from the caller's tensor: a pass
// that copied each route's row first, and the loads of rows that only pad a tile, cost 7 us of the 33-token layer (0.187 ->
// 0.180 ms) and 56 us of the 2048-token one (0.680 -> 0.624). LM head, 2048 -> 151936: 1 row 0.151 -> 0.097 ms, 64 rows 0.116 -> 0.102.
#include "tcgen05.cuh"

#include <algorithm>

namespace qs3 {
namespace {

using namespace tc;

constexpr int kBsThreads = 192;
constexpr uint32_t kBsMaxStages = 6;
constexpr uint32_t kBsBox = 32; // rows of one copy where the token rows lie together

enum : uint32_t {
    ERR_BS_FULL_WAIT = 0x59000001u,
    ERR_BS_EMPTY_WAIT = 0x59000002u,
    ERR_BS_ACC_FULL_WAIT = 0x59000003u,
    ERR_BS_ACC_EMPTY_WAIT = 0x59000004u,
};

struct Bf16StreamParams {
    uint32_t n;            // output features per group (gated: intermediate size)
    uint32_t k_blocks;     // ceil(k / 64)
    uint32_t b_rows;       // weight rows per group (gated: 2 n)
    uint32_t units_per_tile; // gated: ceil(n / 128); plain: ceil(n / 256)
    const int32_t* tile_expert;
    const int32_t* tile_row0;
    const int32_t* tile_nrows;
    const int32_t* total_tiles;
    const int32_t* row_tokens; // NULL: A rows are the padded rows; else dense row -> A row
    const int32_t* indptr;     // with row_tokens: segment starts, dense and padded
    const int32_t* pad_indptr;
    int gathered;              // rows of experts with more than kGatherRows rows are in map_g, padded
    int tables_ready;      // the tables were complete before the predecessor in the stream started
    uint32_t dense_rows;   // no tile tables: one group, row tiles in order
    uint32_t half;         // weight rows of each of a unit's two tiles, 128 (dense: a multiple of 8 up to 128)
    __nv_bfloat16* out;    // [rows, n]
    uint64_t out_pitch;
    uint32_t* err;
};

template <int NT> struct BsRing {
    static constexpr uint32_t kStageBytes = 2 * kTileBytes + NT * 128;
    static constexpr uint32_t kStages = NT == 32 ? kBsMaxStages : NT == 64 ? 5 : 4;
};

template <int NT, bool GATED>
__global__ void __launch_bounds__(kBsThreads, 1)
gemm_bf16_stream_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                        const __grid_constant__ CUtensorMap map_g, // boxes of rows that lie together
                        const Bf16StreamParams p)
{
    constexpr uint32_t kStageBytes = BsRing<NT>::kStageBytes;
    constexpr uint32_t kNumStages = BsRing<NT>::kStages;
    constexpr uint32_t kTmemCols = 4 * NT;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + kNumStages * kStageBytes);
    uint64_t* empty_bar = full_bar + kBsMaxStages;
    uint64_t* acc_full = empty_bar + kBsMaxStages;
    uint64_t* acc_empty = acc_full + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
    volatile uint32_t* abort_flag = tmem_slot + 1;

    const uint32_t warp = threadIdx.x >> 5;
    const uint32_t lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < kNumStages; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], 4); // one arrival per epilogue warp
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
    // weights and tables are complete: a decode batch's loads need not wait (with skewed ends of a longer predecessor the
    // CTAs would no longer read neighbouring rows together: down of 2048 tokens 0.177 -> 0.19 ms)
    const bool early = NT == 32 && p.tables_ready && warp == 4;
    if (!early)
        chain_begin();

    // unit i of this CTA: the CTAs of a round hold neighbouring units, so that a token tile (and the weights of an
    // expert with several tiles) is read by several SMs at about the same time
    const bool grouped = p.tile_expert != nullptr;
    const uint32_t total = (grouped ? static_cast<uint32_t>(*p.total_tiles) : (p.dense_rows + NT - 1) / NT) * p.units_per_tile;
    const uint32_t my_units = blockIdx.x < total ? (total - blockIdx.x - 1) / gridDim.x + 1 : 0;

    if (warp == 4) {
        // ------------------------------------------------------------ producer --
        // Lane 0 loads the weight tiles, lane j part j of the token tile, a box of rows that lie together or four rows
        // found through the routing tables (gather4: no gather pass). Parts past the tile's last row are not moved.
        uint32_t s = 0, ph = 0;
        bool ok = true;
        for (uint32_t i = 0; i < my_units && ok; ++i) {
            const uint32_t u = blockIdx.x + i * gridDim.x, tile = u / p.units_per_tile;
            const uint32_t f0 = u % p.units_per_tile * (GATED ? 1 : 2) * p.half;
            const int row0 = grouped ? p.tile_row0[tile] : static_cast<int>(tile * NT);
            const int nrows = grouped ? p.tile_nrows[tile] : static_cast<int>(min(static_cast<uint32_t>(NT), p.dense_rows - row0));
            const int expert = grouped ? p.tile_expert[tile] : 0;
            // rows of a tile past the last feature belong to something else and are dropped by the epilogue
            const int w_row = expert * static_cast<int>(p.b_rows) + static_cast<int>(f0);
            const int w_row2 = w_row + static_cast<int>(GATED ? p.n : p.half);
            uint32_t ahead = 0; // k blocks whose weights are on their way already
            if (i == 0 && early) {
                if (elect_one()) {
                    for (; ahead < min(kNumStages, p.k_blocks); ++ahead) {
                        uint8_t* sw = smem + ahead * kStageBytes;
                        mbar_expect_tx_only(&full_bar[ahead], 2 * p.half * 128);
                        tma_load_2d(sw, &map_w, &full_bar[ahead], static_cast<int>(ahead) * 64, w_row);
                        tma_load_2d(sw + kTileBytes, &map_w, &full_bar[ahead], static_cast<int>(ahead) * 64, w_row2);
                    }
                }
                __syncwarp();
                chain_begin();
            }
            bool boxes = nrows > static_cast<int>(kGatherRows);
            int row[4];
            if (p.row_tokens == nullptr) { // (four rows of a small tile at a time, which moves no padding)
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    row[q] = row0 + min(static_cast<int>(lane) * 4 + q, nrows - 1);
            } else {
                const int dense = p.indptr[expert], dense0 = dense + row0 - p.pad_indptr[expert];
                boxes = p.gathered && p.indptr[expert + 1] - dense > static_cast<int>(kGatherRows);
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    row[q] = p.row_tokens[dense0 + min(static_cast<int>(lane) * 4 + q, nrows - 1)];
            }
            const uint32_t part_rows = boxes ? kBsBox : 4u, parts = (static_cast<uint32_t>(nrows) + part_rows - 1) / part_rows;
            for (uint32_t kb = 0; kb < p.k_blocks; ++kb) {
                ok = __all_sync(0xffffffffu, mbar_wait<true>(&empty_bar[s], ph ^ 1, abort_flag, p.err, ERR_BS_EMPTY_WAIT));
                if (!ok)
                    break;
                uint8_t* sw = smem + s * kStageBytes;
                const int c0 = static_cast<int>(kb) * 64;
                if (elect_one()) {
                    mbar_expect_tx(&full_bar[s], (kb < ahead ? 0 : 2 * p.half * 128) + parts * part_rows * 128);
                    if (kb >= ahead) {
                        tma_load_2d(sw, &map_w, &full_bar[s], c0, w_row);
                        tma_load_2d(sw + kTileBytes, &map_w, &full_bar[s], c0, w_row2);
                    }
                }
                __syncwarp();
                if (lane < parts) {
                    uint8_t* dst = sw + 2 * kTileBytes + lane * part_rows * 128;
                    if (boxes)
                        tma_load_2d(dst, &map_g, &full_bar[s], c0, row0 + static_cast<int>(lane * kBsBox));
                    else
                        tma_gather4(dst, &map_x, &full_bar[s], c0, row);
                }
                if (++s == kNumStages) {
                    s = 0;
                    ph ^= 1;
                }
            }
        }
        if (early && my_units == 0)
            chain_begin();
    } else if (warp == 5) {
        // ---------------------------------------------------------- MMA issuer --
        if (elect_one()) {
            // M = 128 weight rows, N = NT tokens, bf16 x bf16 -> f32, both operands K-major
            constexpr uint32_t kIdesc
                = (1u << 4) | (1u << 7) | (1u << 10) | ((static_cast<uint32_t>(NT) >> 3) << 17) | ((kBM >> 4) << 24);
            uint32_t s = 0, ph = 0;
            bool ok = true;
            for (uint32_t i = 0; i < my_units && ok; ++i) {
                const uint32_t buf = i & 1;
                if (!mbar_wait<true>(&acc_empty[buf], ((i >> 1) & 1) ^ 1, abort_flag, p.err, ERR_BS_ACC_EMPTY_WAIT))
                    break;
                tc_fence_after();
                const uint32_t d = tmem_base + buf * 2 * NT;
                for (uint32_t kb = 0; kb < p.k_blocks; ++kb) {
                    if (!mbar_wait<true>(&full_bar[s], ph, abort_flag, p.err, ERR_BS_FULL_WAIT)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t sw = smem_u32(smem + s * kStageBytes);
                    const uint64_t dw = operand_desc(sw), dw2 = operand_desc(sw + kTileBytes);
                    const uint64_t dx = operand_desc(sw + 2 * kTileBytes);
#pragma unroll
                    for (uint32_t j = 0; j < 4; ++j) {
                        const uint32_t acc = (kb > 0 || j > 0) ? 1u : 0u;
                        tc_mma_bf16(d, dw + 2 * j, dx + 2 * j, kIdesc, acc);
                        tc_mma_bf16(d + NT, dw2 + 2 * j, dx + 2 * j, kIdesc, acc);
                    }
                    tc_commit(&empty_bar[s]);
                    if (++s == kNumStages) {
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
        const uint32_t lane_base = (warp * 32) << 16;
        for (uint32_t i = 0; i < my_units; ++i) {
            const uint32_t u = blockIdx.x + i * gridDim.x, tile = u / p.units_per_tile;
            const uint32_t f0 = u % p.units_per_tile * (GATED ? 1 : 2) * p.half;
            const uint32_t buf = i & 1;
            const uint32_t row0 = grouped ? static_cast<uint32_t>(p.tile_row0[tile]) : tile * NT;
            const uint32_t nrows = grouped ? static_cast<uint32_t>(p.tile_nrows[tile]) : min(static_cast<uint32_t>(NT), p.dense_rows - row0);
            const uint32_t r = warp * 32 + lane; // weight row of each tile; rows past `half` hold nothing
            const uint32_t f = f0 + r;           // plain: and f + half
            const bool live = r < p.half && f < p.n, live2 = r < p.half && f + p.half < p.n;
            const bool ready = __all_sync(0xffffffffu, mbar_wait(&acc_full[buf], (i >> 1) & 1, abort_flag, p.err,
                                                                 ERR_BS_ACC_FULL_WAIT));
            if (!ready)
                break;
            tc_fence_after();
            const uint32_t src = tmem_base + lane_base + buf * 2 * NT;
            __nv_bfloat16* out = p.out + row0 * p.out_pitch + f;
#pragma unroll 1 // (short code: its first pass is fetched with HBM busy)
            for (uint32_t c = 0; c * 16 < nrows; ++c) {
                uint32_t va[16], vb[16];
                tc_ld16(src + c * 16, va);
                tc_ld16(src + NT + c * 16, vb);
                tc_ld_wait();
#pragma unroll
                for (uint32_t t = 0; t < 16; ++t) {
                    if (c * 16 + t < nrows) { // uniform
                        const float a = __uint_as_float(va[t]), b = __uint_as_float(vb[t]);
                        __nv_bfloat16* o = out + (c * 16 + t) * p.out_pitch;
                        if constexpr (GATED) {
                            // upstream stores the gate_up product as bf16 before SwiGLU (qsfi_moe.cu:638-651,445-463)
                            const float g = round_bf16(a), up = round_bf16(b);
                            if (live)
                                *o = __float2bfloat16(g * sigmoid_fast(g) * up);
                        } else {
                            if (live)
                                *o = __float2bfloat16(a);
                            if (live2)
                                o[p.half] = __float2bfloat16(b);
                        }
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0)
                mbar_arrive(&acc_empty[buf]);
        }
    }

    // ---- teardown ----
    tc_fence_before();
    __syncthreads();
    if (warp == 5) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols)
                     : "memory");
    }
}

template <int NT, bool GATED>
cudaError_t launch_stream_instance(const CUtensorMap& mw, const CUtensorMap& mx, const CUtensorMap& mg, const Bf16StreamParams& sp,
                                   uint32_t grid, cudaStream_t stream)
{
    auto kernel = gemm_bf16_stream_kernel<NT, GATED>;
    constexpr size_t smem = 1024 + BsRing<NT>::kStages * BsRing<NT>::kStageBytes + 256;
    static bool configured[64] = {}; // per instantiation and device
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
    return launch_chained(kernel, dim3(grid), kBsThreads, smem, stream, mw, mx, mg, sp);
}

} // namespace

bool bf16_one_tile_per_cta(uint32_t routes, uint32_t experts, uint32_t hidden, uint32_t inter)
{
    // Few experts give the streaming kernel fewer units than SMs, each of 256 weight rows with the epilogue of a whole
    // token tile at its end and, up to kGatherRows rows, gather4 loads that HBM no longer hides. Tiles of 128 x 128, two CTAs
    // per SM, are shorter; beyond about a round of them, and for few rows, where the weights decide, streaming wins.
    // Routed experts alone (hidden, experts top-k, intermediate; tokens: streaming / one tile per CTA, us):
    //   2048, 8 top-2, 512     100: 38 / 32, 150: 46 / 32, 1000: 61 / 46, 2500: 97 / 87, 4000: 109 / 106
    //   2048, 8 top-2, 1024    100: 43 / 47, 150: 52 / 45, 1000: 70 / 56, 2500: 121 / 120
    //   1024, 4 top-1, 512     64: 26 / 26, 150: 33 / 26, 1000: 46 / 28, 4000: 53 / 40
    //   2048, 16 top-4, 768    150: 51 / 55, 300: 73 / 56, 1000: 103 / 94, 1500: 121 / 121, 4000: 219 / 245
    //   2048, 32 top-4, 512    300: 61 / 70, 600: 81 / 71, 1500: 105 / 108
    // With a short k that epilogue does not hide behind the k loop of the next unit either, once an expert has the rows for
    // whole tiles:
    //   1024, 64 top-6, 512    600: 69 / 79, 1500: 111 / 113, 2500: 138 / 131, 6000: 269 / 255
    //   512, 256 top-8, 512    1000: 100 / 150, 2000: 144 / 155, 2500: 165 / 160, 6000: 296 / 270
    //   512, 64 top-8, 256     300: 36 / 36, 600: 50 / 37, 4000: 132 / 107
    //   256, 128 top-8, 128    300: 28 / 32, 600: 34 / 32, 1500: 48 / 35
    const uint64_t rows = (routes + experts - 1) / experts;
    const uint64_t ctas = (rows + kTileM - 1) / kTileM * experts * ((inter + 63) / 64);
    if (hidden <= 1024 && rows >= 16 + hidden * hidden / 5400)
        return true;
    return rows > 16 && 10 * ctas <= 26 * kSmCount && (rows - 16) * 2 * kSmCount >= 36 * ctas;
}

uint32_t bf16_tile_rows(uint32_t routes, uint32_t experts, uint32_t hidden, uint32_t inter)
{
    if (bf16_one_tile_per_cta(routes, experts, hidden, inter))
        return static_cast<uint32_t>(kTileM);
    // Token bytes per weight byte grow with the tile, weight passes with the tiles of an expert. Layer times, 128
    // experts top-8: 8 routes per expert 0.239 ms with 32-row against 0.243 with 64-row tiles, 32 routes of a skewed
    // router 0.229 against 0.203; 64 routes 0.287 with 64-row against 0.291 with 128-row tiles, 128 routes 0.380
    // against 0.367.
    return routes <= 12u * experts ? 32u : routes <= 96u * experts ? 64u : static_cast<uint32_t>(kTileM);
}

bool bf16_stream_gemm_supported(const GemmProblem& g)
{
    const bool plain = !g.nvfp4 && g.k % 8 == 0 && (g.alpha == 0.0f || g.alpha == 1.0f) && g.beta == 0.0f
        && g.group_scale == nullptr && g.group_scale_up == nullptr && g.bias == nullptr
        && (reinterpret_cast<uintptr_t>(g.a) & 15u) == 0 && (reinterpret_cast<uintptr_t>(g.b) & 15u) == 0
        && g.a_pitch_bytes % 16 == 0 && g.b_pitch_bytes % 16 == 0;
    if (g.tile_expert == nullptr) {
        return plain && !g.gated && g.groups == 1 && g.epilogue == EPI_STORE_BF16 && g.a_rows <= 64
            && (g.n + 255) / 256 >= device_sm_count();
    }
    return plain && !g.one_tile_per_cta && (g.tile_rows == 32 || g.tile_rows == 64 || g.tile_rows == 128)
        && (g.gated ? g.epilogue == EPI_SWIGLU_BF16 : g.epilogue == EPI_STORE_BF16);
}

cudaError_t launch_bf16_stream_gemm(const GemmProblem& g, cudaStream_t stream, const char** why)
{
    Bf16StreamParams sp {};
    sp.n = g.n;
    sp.k_blocks = (g.k + 63) / 64;
    sp.b_rows = g.gated ? 2 * g.n : g.n;
    sp.half = 128;
    if (g.tile_expert == nullptr) {
        // One row tile: the rounds of the CTAs are few, so the weight rows of a unit are chosen for a full last round
        // (151936 features: 594 units of 256 on 148 SMs leave two units to a fifth round; 208 fill five).
        uint32_t best = ~0u;
        for (uint32_t half = 128; half >= 64; half -= 8) {
            const uint32_t units = (g.n + 2 * half - 1) / (2 * half);
            const uint32_t cost = (units + device_sm_count() - 1) / device_sm_count() * (2 * half + 8);
            if (cost < best) {
                best = cost;
                sp.half = half;
            }
        }
    }
    sp.units_per_tile = (g.n + (g.gated ? 1 : 2) * sp.half - 1) / ((g.gated ? 1 : 2) * sp.half);
    sp.tile_expert = g.tile_expert;
    sp.tile_row0 = g.tile_row0;
    sp.tile_nrows = g.tile_nrows;
    sp.total_tiles = g.total_tiles;
    sp.dense_rows = static_cast<uint32_t>(g.a_rows);
    sp.tables_ready = g.tables_ready;
    sp.row_tokens = g.row_tokens;
    sp.indptr = g.indptr;
    sp.pad_indptr = g.pad_indptr;
    sp.gathered = g.gathered != nullptr;
    sp.out = static_cast<__nv_bfloat16*>(g.out);
    sp.out_pitch = g.out_pitch_elems;
    sp.err = device_error_word();
    const uint32_t nt = g.tile_expert != nullptr ? g.tile_rows : g.a_rows <= 32 ? 32u : 64u;
    CUtensorMap mw, mx, mg;
    const uint64_t w_rows = static_cast<uint64_t>(g.groups) * sp.b_rows;
    const bool copy = g.row_tokens != nullptr && g.gathered != nullptr; // (as many rows as the tables have room for)
    const bool ok = make_operand_map(&mw, false, g.b, g.k, w_rows, g.b_pitch_bytes, sp.half)
        && make_operand_map(&mx, false, g.a, g.k, g.a_rows, g.a_pitch_bytes, 1)
        && make_operand_map(&mg, false, copy ? g.gathered : g.a, g.k, copy ? static_cast<uint64_t>(g.max_tiles) * g.tile_rows : g.a_rows,
                            copy ? g.k * 2ull : g.a_pitch_bytes, kBsBox);
    if (!ok) {
        if (why != nullptr)
            *why = "cuTensorMapEncodeTiled failed";
        return cudaErrorInvalidValue;
    }
    const uint32_t grid = static_cast<uint32_t>(
        std::min<uint64_t>((g.tile_expert != nullptr ? g.max_tiles : (g.a_rows + nt - 1) / nt) * static_cast<uint64_t>(sp.units_per_tile), device_sm_count()));
    switch (nt) {
    case 32:
        return g.gated ? launch_stream_instance<32, true>(mw, mx, mg, sp, grid, stream)
                       : launch_stream_instance<32, false>(mw, mx, mg, sp, grid, stream);
    case 64:
        return g.gated ? launch_stream_instance<64, true>(mw, mx, mg, sp, grid, stream)
                       : launch_stream_instance<64, false>(mw, mx, mg, sp, grid, stream);
    default:
        return g.gated ? launch_stream_instance<128, true>(mw, mx, mg, sp, grid, stream)
                       : launch_stream_instance<128, false>(mw, mx, mg, sp, grid, stream);
    }
}

} // namespace qs3
