// NVFP4 grouped GEMMs for experts with few rows (decode batches, chunks of a prefill): weight streaming.
//
// With token rows as the M = 128 side of the MMA most of every instruction multiplies padding. Here the operands are
// swapped: the 128 WEIGHT rows of a feature block are M, the expert's token tile of NT (32 or 64) padded rows is N,
// and the kernel runs at the speed the weights arrive from HBM.
//
//   grid   persistent, one CTA per SM; the (token tile, feature block) units are cut into equal contiguous ranges
//          (the CTA-per-tile grid of an earlier version lost a load latency per CTA and its last wave)
//   smem   token panel (all of k: k/256 tiles of NT x 128 B), its scale tiles, weight ring: stages x (128 x 128 B
//          codes + 4 scale tiles); gated: f32 exchange buffer of 32 tokens x (64 gate + 64 up) values
//   TMEM   2 or 4 accumulators of NT columns (lane = weight row, column = token) | 16 columns of weight scales per ring
//          stage | 2 x token scales of all of k (alternating per tile)
//   warps  0-3 epilogue, 4 weight producer (TMA), 5 and 11 MMA issuers, 6 scale copier, 7-10 panel loaders
//
// The panel loaders fetch the token rows themselves, through the routing tables when the rows are still in token
// order (no gather pass), and hold the next tile's rows in registers while the current tile is multiplied, so that a
// change of tile costs the MMA thread only their shared-memory stores; the ring covers those. The scale copies
// (tcgen05.cp) come from a warp of their own: from the MMA thread each costs ~50 cycles.
//
// A shared expert of the same intermediate size is one more group whose rows are all tokens in order, with weights of
// its own: as GEMMs of their own on a side stream its two launches and the fork and join cost a single-token layer
// more host time than the GPU work they overlapped.
//
// Gated epilogue: gate rows are lanes 0-63, up rows lanes 64-127. The values go through shared memory so that one
// thread holds one 16-feature block of one token: SwiGLU, block maximum and quantisation without shuffles, and the
// time does not grow with the rows of the tile.
//
// Scale tiles are the library's tiled layout (include/qs3_moe.h): 512 bytes per (128-row block, 64-element k group),
// byte = (row % 32) * 16 + (row / 32 % 4) * 4 + k / 16 % 4, which tcgen05.cp.32x128b.warpx4 turns into four TMEM
// columns, one per group of 32 rows. The loaders lay the token tile's scale words down as groups 0 (and 1) of such
// tiles, so that the MMA reads them from a 4-column aligned tensor-memory address like any other scale operand.
//
// Bound by HBM: hit experts * weight bytes. 128 tokens, 512 experts top-10 (471 hit): gate_up 0.112 -> 0.092 ms
// (6.0 TB/s), down 0.055 -> 0.050; 1021 tokens: gate_up 0.150 -> 0.110, down 0.110 -> 0.058 ms against 128-row tiles. Since
// then, by shorter panel loaders and issue from elected lanes, replayed from a graph in turn on one board (others take up to 4 %
// longer): layer of 128 tokens 0.177 -> 0.162, of 1021 0.222 -> 0.206.
#include "common.cuh"
#include "nvfp4.cuh"
#include "tcgen05.cuh"

#include <algorithm>

namespace qs3 {
namespace {

using namespace tc;

constexpr int kSwThreads = 384;
constexpr uint32_t kSwLoaders = 128;               // threads of the panel loaders
constexpr uint32_t kSwStageBytes = kTileBytes + kSfBytes;
constexpr uint32_t kSwMaxStages = 9;
constexpr uint32_t kSwMaxAcc = 4;
constexpr uint32_t kSwMaxKBlocks = 8;              // k <= 2048
constexpr uint32_t kSwMiscBytes = 512;
constexpr uint32_t kSwExPitch = 68;                // floats per token row of the exchange buffer (no bank conflicts)
constexpr uint32_t kSwExBytes = 2 * 32 * kSwExPitch * 4;
constexpr uint32_t kSwBatch = 16;                  // 16-byte vectors a loader thread keeps in registers

enum : uint32_t {
    ERR_SW_PANEL_WAIT = 0x54000001u,
    ERR_SW_FULL_WAIT = 0x54000002u,
    ERR_SW_EMPTY_WAIT = 0x54000003u,
    ERR_SW_ACC_FULL_WAIT = 0x54000004u,
    ERR_SW_ACC_EMPTY_WAIT = 0x54000005u,
    ERR_SW_PANEL_FREE_WAIT = 0x54000006u,
    ERR_SW_SF_WAIT = 0x54000007u,
};

struct SwapParams {
    uint32_t n;          // output features per group (gated: intermediate size)
    uint32_t k_blocks;   // k / 256
    uint32_t kgroups;    // k / 64
    uint32_t b_rows;     // weight rows per group (gated: 2 n)
    uint32_t num_fb;     // feature blocks: n / 128 (gated: n / 64)
    uint32_t stages;
    uint32_t acc_mask;   // accumulators - 1 (2 or 4 of them)
    const uint8_t* x;    // token codes [rows, k / 2]
    const uint8_t* x_sf; // their scales, tiled by row (x_sf_linear: row-major)
    int x_sf_linear;
    const int32_t* row_tokens; // NULL: x rows are the padded rows; else dense row -> x row
    const int32_t* indptr;     // with row_tokens: segment starts, dense and padded
    const int32_t* pad_indptr;
    const uint8_t* w_sf; // weight scales, tiled per group
    uint64_t w_sf_group_stride;
    const int32_t* tile_expert;
    const int32_t* tile_row0;
    const int32_t* tile_nrows;
    const int32_t* total_tiles;
    void* out;           // gated: e2m1 codes [rows, n / 2]; else bf16 [rows, n]
    uint8_t* out_sf;     // gated: tiled scales of the output rows
    float alpha;
    const float* group_scale;
    const float* group_scale_up;
    float out_global;
    int tables_ready;        // the tile tables were complete before the predecessor in the stream started
    int shared_group;        // group number of a shared expert with weights of its own (map_ws, ...), -1: none
    const uint8_t* shared_w_sf;
    const float* shared_scale;
    const float* shared_scale_up;
    uint32_t* err;
};

template <int NT, bool GATED>
__global__ void __launch_bounds__(kSwThreads, 1)
gemm_nvfp4_swap_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_ws,
                       const SwapParams p)
{
    constexpr uint32_t kFeat = GATED ? 64 : 128; // output features per feature block
    constexpr uint32_t kPanelTile = NT * 128;    // one k block of the token panel

    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    uint8_t* panel = smem;                                        // k_blocks x NT x 128 B
    uint8_t* ring = panel + p.k_blocks * kPanelTile;
    uint8_t* panel_sf = ring + p.stages * kSwStageBytes;          // kgroups x 512 B
    float* s_ex = reinterpret_cast<float*>(panel_sf + p.kgroups * 512); // gated: [2][32][kSwExPitch]
    uint8_t* misc = panel_sf + p.kgroups * 512 + (GATED ? kSwExBytes : 0);
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(misc);
    uint64_t* empty_bar = full_bar + kSwMaxStages;
    uint64_t* sf_ready = empty_bar + kSwMaxStages;
    uint64_t* acc_full = sf_ready + kSwMaxStages;
    uint64_t* acc_empty = acc_full + kSwMaxAcc;
    uint64_t* panel_full = acc_empty + kSwMaxAcc;  // loaders -> MMA: the tile's codes are in the panel
    uint64_t* panel_free = panel_full + 1; // MMA -> loaders: the tile's MMAs are done
    uint64_t* psf_full = panel_free + 1;   // loaders -> copier: the tile's scale words are in panel_sf
    uint64_t* psf_free = psf_full + 1;     // copier -> loaders: they are in tensor memory
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(psf_free + 1);
    volatile uint32_t* abort_flag = tmem_slot + 1;

    const uint32_t warp = threadIdx.x >> 5;
    const uint32_t lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < p.stages; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 2); // the MMAs of one issuer, and the other issuer has seen the stage
            mbar_init(&sf_ready[s], 1);
        }
        for (uint32_t b = 0; b < kSwMaxAcc; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], 4); // one arrival per epilogue warp
        }
        mbar_init(panel_full, 1);
        mbar_init(panel_free, 2); // one arrival per MMA issuer
        mbar_init(psf_full, 1);
        mbar_init(psf_free, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 5) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(512u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t tmem_wsf = tmem_base + (p.acc_mask + 1) * NT; // 16 columns per ring stage
    const uint32_t tmem_xsf = tmem_wsf + 16 * p.stages;          // 2 x 4 columns per k group
    const uint32_t xsf_cols = 4 * p.kgroups;

    // The tables of the down projection are older than its predecessor (the gate_up GEMM, whose start means that the
    // sort is complete), and weights are older still: its producer fills the ring before it waits, its panel loaders look up
    // their first tile. Every other role touches what the predecessor wrote.
    const bool early = p.tables_ready && (warp == 4 || (warp >= 7 && warp <= 10));
    if (!early)
        chain_begin();

    // this CTA's units: feature blocks [u0, u1) of the tiles in order
    const uint64_t total = static_cast<uint64_t>(__ldcg(p.total_tiles)) * p.num_fb;
    const uint32_t u0 = static_cast<uint32_t>(total * blockIdx.x / gridDim.x);
    const uint32_t u1 = static_cast<uint32_t>(total * (blockIdx.x + 1) / gridDim.x);
    const uint32_t tile_first = u0 / p.num_fb, fb_first = u0 % p.num_fb;
    const uint32_t acc_shift = p.acc_mask == 3 ? 2 : 1;

    if (warp == 4) {
        // ------------------------------------------------------------ producer --
        if (elect_one()) {
            uint32_t s = 0, ph = 0;
            bool ok = true;
            uint32_t tile = tile_first, fb = fb_first;
            for (uint32_t u = u0; u < u1 && ok; ++u) {
                const int expert = __ldcg(p.tile_expert + tile);
                const bool shared = expert == p.shared_group;
                const CUtensorMap* map = shared ? &map_ws : &map_w;
                const int w_row = (shared ? 0 : expert * static_cast<int>(p.b_rows)) + static_cast<int>(fb * kFeat);
                const uint8_t* sf_src = (shared ? p.shared_w_sf : p.w_sf + static_cast<uint64_t>(expert) * p.w_sf_group_stride)
                    + (static_cast<uint64_t>(fb) * p.kgroups) * 512;
                for (uint32_t kb = 0; kb < p.k_blocks; ++kb) {
                    if (!mbar_wait<true>(&empty_bar[s], ph ^ 1, abort_flag, p.err, ERR_SW_EMPTY_WAIT)) {
                        ok = false;
                        break;
                    }
                    uint8_t* sb = ring + s * kSwStageBytes;
                    mbar_expect_tx(&full_bar[s], kSwStageBytes);
                    if (GATED) { // 64 gate rows, then the 64 up rows of the same features
                        tma_load_2d(sb, map, &full_bar[s], static_cast<int>(kb * 128), w_row);
                        tma_load_2d(sb + kTileBytes / 2, map, &full_bar[s], static_cast<int>(kb * 128),
                                    w_row + static_cast<int>(p.n));
                    } else {
                        tma_load_2d(sb, map, &full_bar[s], static_cast<int>(kb * 128), w_row);
                    }
                    bulk_load(sb + kTileBytes, sf_src + static_cast<uint64_t>(kb) * kSfBytes, kSfBytes, &full_bar[s]);
                    if (++s == p.stages) {
                        s = 0;
                        ph ^= 1;
                    }
                }
                if (++fb == p.num_fb) {
                    fb = 0;
                    ++tile;
                }
            }
        }
    } else if (warp == 5 || warp == 11) {
        // --------------------------------------------------------- MMA issuers --
        // Alternate feature blocks: one thread's instructions, waits and commits take longer than the weights of a
        // feature block with a short k (down of a 128-token batch: one issuer 0.056 ms, two 0.050).
        if (elect_one()) {
            // M = 128 weight rows, N = NT tokens, e2m1 x e2m1 with e4m3 block scales, f32 accumulate
            constexpr uint32_t kIdesc
                = (1u << 7) | (1u << 10) | ((static_cast<uint32_t>(NT) >> 3) << 17) | ((kBM >> 4) << 24);
            const uint32_t mine = warp == 5 ? 0 : 1; // parity of this issuer's feature blocks
            uint32_t s = 0, ph = 0, fb = fb_first, i = 0; // i: tiles this CTA has started
            bool ok = true;
            for (uint32_t u = u0; u < u1 && ok; ++u) {
                const bool first = u == u0 || fb == 0;
                if (++fb == p.num_fb)
                    fb = 0;
                const bool last = u + 1 == u1 || fb == 0;
                const uint32_t buf = (u - u0) & p.acc_mask;
                if (first) {
                    ok = mbar_wait<true>(panel_full, i & 1, abort_flag, p.err, ERR_SW_PANEL_WAIT);
                    ++i;
                }
                if (ok && ((u - u0) & 1) != mine) {
                    // the other issuer's: its stages are waited for all the same, because a parity tells two
                    // successive uses of a stage apart and no more, and no stage is refilled before both have
                    for (uint32_t kb = 0; kb < p.k_blocks && ok; ++kb) {
                        ok = mbar_wait<true>(&sf_ready[s], ph, abort_flag, p.err, ERR_SW_SF_WAIT);
                        if (ok)
                            mbar_arrive(&empty_bar[s]);
                        if (++s == p.stages) {
                            s = 0;
                            ph ^= 1;
                        }
                    }
                    if (ok && last)
                        tc_commit(panel_free);
                    continue;
                }
                if (!ok
                    || !mbar_wait<true>(&acc_empty[buf], (((u - u0) >> acc_shift) & 1) ^ 1, abort_flag, p.err,
                                        ERR_SW_ACC_EMPTY_WAIT)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t d = tmem_base + buf * NT;
                const uint32_t xsf = tmem_xsf + xsf_cols * ((i - 1) & 1);
                for (uint32_t kb = 0; kb < p.k_blocks; ++kb) {
                    // the stage's scales are in tensor memory (the copier waited for the stage's loads)
                    if (!mbar_wait<true>(&sf_ready[s], ph, abort_flag, p.err, ERR_SW_SF_WAIT)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint64_t da = operand_desc(smem_u32(ring + s * kSwStageBytes));
                    const uint64_t db = operand_desc(smem_u32(panel + kb * kPanelTile));
#pragma unroll
                    for (uint32_t j = 0; j < 4; ++j)
                        tc_mma_nvfp4(d, da + 2 * j, db + 2 * j, kIdesc, (kb > 0 || j > 0) ? 1u : 0u,
                                     tmem_wsf + 16 * s + 4 * j, xsf + 16 * kb + 4 * j);
                    tc_commit(&empty_bar[s]);
                    if (++s == p.stages) {
                        s = 0;
                        ph ^= 1;
                    }
                }
                if (ok) {
                    tc_commit(&acc_full[buf]);
                    if (last)
                        tc_commit(panel_free);
                }
            }
        }
    } else if (warp == 6) {
        // -------------------------------------------------------- scale copier --
        if (elect_one()) {
            uint32_t s = 0, ph = 0, fb = fb_first, i = 0;
            bool ok = true;
            for (uint32_t u = u0; u < u1 && ok; ++u) {
                if (u == u0 || fb == 0) {
                    // the tile's token scales, into the columns of the tile before last: its MMAs are done, because
                    // the loaders waited for that before they filled the panel of the tile in between
                    ok = mbar_wait<true>(psf_full, i & 1, abort_flag, p.err, ERR_SW_PANEL_WAIT);
                    if (!ok)
                        break;
                    tc_fence_after();
                    for (uint32_t g = 0; g < p.kgroups; ++g)
                        tc_cp_scales(tmem_xsf + xsf_cols * (i & 1) + 4 * g, scale_desc(smem_u32(panel_sf) + g * 512));
                    tc_commit(psf_free);
                    ++i;
                }
                if (++fb == p.num_fb)
                    fb = 0;
                for (uint32_t kb = 0; kb < p.k_blocks; ++kb) {
                    // the stage was refilled, so the MMAs that read its scale columns last time round are done
                    if (!mbar_wait<true>(&full_bar[s], ph, abort_flag, p.err, ERR_SW_FULL_WAIT)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t sf = smem_u32(ring + s * kSwStageBytes) + kTileBytes;
#pragma unroll
                    for (uint32_t j = 0; j < 4; ++j)
                        tc_cp_scales(tmem_wsf + 16 * s + 4 * j, scale_desc(sf + j * 512));
                    tc_commit(&sf_ready[s]);
                    if (++s == p.stages) {
                        s = 0;
                        ph ^= 1;
                    }
                }
            }
        }
    } else if (warp >= 7 && warp <= 10) {
        // ------------------------------------------------------- panel loaders --
        // A warp takes every fourth row, a lane one or two vectors of it; scale words by (row, k group), each thread the same
        // row throughout. Few instructions: a warp of its own per scheduler runs them one after the other, and with
        // divisions per vector the first tile took 4 us to ask for and 2 to store, with the ring full and HBM idle
        // (first MMA 8.9 -> 4.0 us after the predecessor's end in the down kernel of 128 tokens).
        const uint32_t t = threadIdx.x - 7 * 32, lw = t >> 5;
        const uint32_t vecs = p.k_blocks * 8;      // 16-byte vectors per row
        const uint32_t halves = vecs > 32 ? 2 : 1; // vectors of a row per lane
        const uint32_t sj = t % NT, kg0 = t / NT;  // this thread's scale words: row, first k group
        constexpr uint32_t kKgStep = kSwLoaders / NT;
        uint32_t i = 0;
        bool ok = true, waited = !early;
        for (uint32_t u = u0; u < u1 && ok; u = (u / p.num_fb + 1) * p.num_fb, ++i) {
            const uint32_t tile = u / p.num_fb;
            const uint32_t row0 = static_cast<uint32_t>(p.tile_row0[tile]);
            const uint32_t nrows = static_cast<uint32_t>(p.tile_nrows[tile]);
            const int32_t* rows = nullptr;
            uint32_t first = row0; // source row of the tile's first row when they are consecutive
            if (p.row_tokens != nullptr) {
                const int expert = p.tile_expert[tile];
                first = row0 - static_cast<uint32_t>(p.pad_indptr[expert]); // a shared expert takes the tokens in order
                if (expert != p.shared_group)
                    rows = p.row_tokens + p.indptr[expert] + first;
            }
            // source rows of the tile's rows lane and lane + 32
            uint32_t src[NT / 32];
#pragma unroll
            for (uint32_t h = 0; h < NT / 32; ++h) {
                const uint32_t j = lane + 32 * h;
                src[h] = j >= nrows ? 0u : rows != nullptr ? static_cast<uint32_t>(rows[j]) : first + j;
            }
            if (!waited)
                chain_begin();
            waited = true;
            // the tile's codes (the first kSwBatch vectors a thread) and scale words travel together
            const uint32_t items = (nrows + 3) / 4 * halves; // of a warp
            uint4 v[kSwBatch];
            const auto load_codes = [&](uint32_t c0) {
#pragma unroll
                for (uint32_t q = 0; q < kSwBatch; ++q) {
                    const uint32_t c = c0 + q, j = lw + 4 * (halves == 2 ? c >> 1 : c), vec = lane + (halves == 2 ? (c & 1) * 32 : 0);
                    const uint32_t r = __shfl_sync(0xffffffffu, NT == 64 && j >= 32 ? src[NT / 32 - 1] : src[0], j & 31);
                    if (j < nrows && vec < vecs)
                        v[q] = *reinterpret_cast<const uint4*>(p.x + static_cast<uint64_t>(r) * (vecs * 16) + vec * 16);
                }
            };
            const auto store_codes = [&](uint32_t c0) {
#pragma unroll
                for (uint32_t q = 0; q < kSwBatch; ++q) {
                    const uint32_t c = c0 + q, j = lw + 4 * (halves == 2 ? c >> 1 : c), vec = lane + (halves == 2 ? (c & 1) * 32 : 0);
                    if (j < nrows && vec < vecs)
                        *reinterpret_cast<uint4*>(panel + (vec >> 3) * kPanelTile + j * 128 + (((vec & 7) ^ (j & 7)) << 4)) = v[q];
                }
            };
            load_codes(0);
            const uint64_t sr = NT == 64 && (lw & 1) ? src[NT / 32 - 1] : src[0]; // of row sj
            const uint8_t* sf = p.x_sf + (p.x_sf_linear ? sr * (p.kgroups * 4) : tiled_scale_offset(sr, 0, p.kgroups));
            const uint32_t sf_step = p.x_sf_linear ? 4 : 512; // bytes between k groups
            for (uint32_t k0 = kg0; k0 < p.kgroups; k0 += 8 * kKgStep) {
                uint32_t w[8];
#pragma unroll
                for (uint32_t q = 0; q < 8; ++q) {
                    const uint32_t kg = k0 + q * kKgStep;
                    w[q] = kg < p.kgroups && sj < nrows ? *reinterpret_cast<const uint32_t*>(sf + kg * sf_step) : 0u;
                }
                if (k0 == kg0 && i >= 1)
                    ok = mbar_wait(psf_free, (i - 1) & 1, abort_flag, p.err, ERR_SW_PANEL_FREE_WAIT);
#pragma unroll
                for (uint32_t q = 0; q < 8; ++q) {
                    const uint32_t kg = k0 + q * kKgStep;
                    if (kg < p.kgroups && ok)
                        *reinterpret_cast<uint32_t*>(panel_sf + kg * 512 + (sj & 31) * 16 + (sj >> 5) * 4) = w[q];
                }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); // tcgen05.cp reads through the async proxy
            ok = group_all(2, kSwLoaders, ok);
            if (!ok)
                break;
            if (t == 0)
                mbar_arrive(psf_full);
            if (i >= 1)
                ok = mbar_wait(panel_free, (i - 1) & 1, abort_flag, p.err, ERR_SW_PANEL_FREE_WAIT);
            // (every lane of a warp shuffles in load_codes: whether the wait gave up is decided for the warp)
            ok = __all_sync(0xffffffffu, ok);
            for (uint32_t c0 = 0; c0 < items && ok; c0 += kSwBatch) {
                if (c0 != 0)
                    load_codes(c0);
                store_codes(c0);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            ok = group_all(2, kSwLoaders, ok);
            if (ok && t == 0)
                mbar_arrive(panel_full);
        }
        if (!waited)
            chain_begin();
    } else {
        // ------------------------------------------------------------ epilogue --
        const uint32_t lane_base = (warp * 32) << 16;
        uint32_t tile = tile_first, fb_next = fb_first, row0 = 0, nrows = 0;
        float scale = 1.0f, scale_up = 1.0f;
        for (uint32_t u = u0; u < u1; ++u) {
            const uint32_t buf = (u - u0) & p.acc_mask;
            const uint32_t fb = fb_next;
            if (u == u0 || fb == 0) { // another tile
                const int expert = p.tile_expert[tile];
                row0 = static_cast<uint32_t>(p.tile_row0[tile]);
                nrows = static_cast<uint32_t>(p.tile_nrows[tile]);
                scale = p.alpha == 0.0f ? 1.0f : p.alpha;
                scale_up = scale;
                const bool shared = expert == p.shared_group;
                const float* gs = shared ? p.shared_scale : p.group_scale != nullptr ? p.group_scale + expert : nullptr;
                const float* gs_up = shared ? p.shared_scale_up : p.group_scale_up != nullptr ? p.group_scale_up + expert : nullptr;
                if (gs != nullptr)
                    scale *= *gs;
                scale_up *= gs_up != nullptr ? *gs_up : (gs != nullptr ? *gs : 1.0f);
            }
            if (++fb_next == p.num_fb) {
                fb_next = 0;
                ++tile;
            }
            bool ready = __all_sync(0xffffffffu, mbar_wait(&acc_full[buf], ((u - u0) >> acc_shift) & 1, abort_flag, p.err,
                                                           ERR_SW_ACC_FULL_WAIT));
            if constexpr (GATED)
                ready = group_all(1, 128, ready); // the four warps meet at barrier 1 below: stop together
            if (!ready)
                break;
            tc_fence_after();
#pragma unroll
            for (uint32_t hh = 0; hh < NT / 32; ++hh) {
                const bool any = hh * 32 < nrows; // uniform over the block
                uint32_t v[32];
                if (any) {
                    tc_ld16(tmem_base + lane_base + buf * NT + hh * 32, v);
                    tc_ld16(tmem_base + lane_base + buf * NT + hh * 32 + 16, v + 16);
                    tc_ld_wait();
                }
                if (hh + 1 == NT / 32) { // the accumulator has been read
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0)
                        mbar_arrive(&acc_empty[buf]);
                }
                if (!any)
                    continue;
                if constexpr (GATED) {
                    float* dst = s_ex + (warp >> 1) * 32 * kSwExPitch + (warp & 1) * 32 + lane;
                    const float sc = warp >= 2 ? scale_up : scale;
#pragma unroll
                    for (uint32_t t = 0; t < 32; ++t)
                        dst[t * kSwExPitch] = __uint_as_float(v[t]) * sc;
                    asm volatile("bar.sync 1, 128;" ::: "memory");
                    // thread = (16-feature block `warp`, token `lane`)
                    const uint32_t j = hh * 32 + lane;
                    if (j < nrows) {
                        const float4* g4 = reinterpret_cast<const float4*>(s_ex + lane * kSwExPitch + warp * 16);
                        const float4* u4 = reinterpret_cast<const float4*>(s_ex + (32 + lane) * kSwExPitch + warp * 16);
                        float a[16];
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            const float4 g = g4[q], up = u4[q];
                            a[4 * q] = __fdividef(g.x, 1.0f + __expf(-g.x)) * up.x;
                            a[4 * q + 1] = __fdividef(g.y, 1.0f + __expf(-g.y)) * up.y;
                            a[4 * q + 2] = __fdividef(g.z, 1.0f + __expf(-g.z)) * up.z;
                            a[4 * q + 3] = __fdividef(g.w, 1.0f + __expf(-g.w)) * up.w;
                        }
                        uint32_t lo, hi;
                        const uint8_t code = quantize_block16(a, p.out_global, &lo, &hi);
                        const uint64_t prow = static_cast<uint64_t>(row0) + j;
                        *reinterpret_cast<uint2*>(static_cast<uint8_t*>(p.out) + prow * (p.n / 2) + fb * 32 + warp * 8)
                            = make_uint2(lo, hi);
                        p.out_sf[tiled_scale_offset(prow, fb * 4 + warp, p.n / 64)] = code;
                    }
                    asm volatile("bar.sync 1, 128;" ::: "memory"); // the exchange buffer is reused
                } else {
                    const uint32_t f = fb * 128 + warp * 32 + lane;
                    __nv_bfloat16* out = static_cast<__nv_bfloat16*>(p.out) + (static_cast<uint64_t>(row0) + hh * 32) * p.n + f;
#pragma unroll
                    for (uint32_t t = 0; t < 32; ++t)
                        if (hh * 32 + t < nrows)
                            out[static_cast<uint64_t>(t) * p.n] = __float2bfloat16(__uint_as_float(v[t]) * scale);
                }
            }
        }
    }

    // ---- teardown ----
    if (p.tables_ready && warp == 4)
        chain_begin();
    tc_fence_before();
    __syncthreads();
    if (warp == 5) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
    }
}

template <int NT, bool GATED>
cudaError_t launch_swap_instance(const CUtensorMap& mw, const CUtensorMap& mws, const SwapParams& sp, uint32_t grid, size_t smem,
                                 cudaStream_t stream)
{
    auto kernel = gemm_nvfp4_swap_kernel<NT, GATED>;
    static bool configured[64] = {}; // per instantiation and device
    int dev = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err != cudaSuccess)
        return err;
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
        if (err != cudaSuccess)
            return err;
        if (dev >= 0 && dev < 64)
            configured[dev] = true;
    }
    return launch_chained(kernel, dim3(grid), kSwThreads, smem, stream, mw, mws, sp);
}

} // namespace

uint32_t nvfp4_tile_rows(uint32_t routes, uint32_t experts, uint32_t hidden, uint32_t inter)
{
    const bool fits = hidden % 256 == 0 && inter % 256 == 0 && hidden / 256 <= kSwMaxKBlocks
        && inter / 256 <= kSwMaxKBlocks;
    if (!fits)
        return static_cast<uint32_t>(kTileM);
    // 32-row tiles while nearly every expert fits one, 64-row tiles while they win whatever the skew (512 experts top-10:
    // 1021 tokens of a skewed router 0.180 against 0.188 ms with 128-row tiles of CTA pairs, even routing 0.23 against 0.35)
    return routes <= 8 * experts ? 32u : routes <= 22 * experts ? 64u : static_cast<uint32_t>(kTileM);
}

uint32_t nvfp4_alt_tile_rows(uint32_t routes, uint32_t experts, uint32_t hidden, uint32_t inter)
{
    // Beyond that it depends on the skew, which only the sort sees, by the cost of a tile of either kind (routing.cu: both
    // measured at 512 experts of 2048 x 512). From 80 routes per expert on (kAltMaxRoutes) evenly routed experts have one
    // 128-row tile for two of 64 or two for three, and those come out ahead.
    return nvfp4_tile_rows(22 * experts, experts, hidden, inter) == 64 && routes > 22 * experts
            && route_sort_can_choose(routes, experts)
        ? 64u
        : 0u;
}

cudaError_t launch_nvfp4_swap_gemm(const GemmProblem& g, cudaStream_t stream, const char** why)
{
    const auto fail = [&](const char* msg) {
        if (why != nullptr)
            *why = msg;
        return cudaErrorNotSupported;
    };
    const bool gated = g.gated != 0;
    if (g.tile_expert == nullptr || (g.tile_rows != 32 && g.tile_rows != 64))
        return fail("the decode NVFP4 GEMM takes grouped problems with 32- or 64-row token tiles");
    if (g.k % 256 != 0 || g.k / 256 > kSwMaxKBlocks || g.n % 128 != 0 || g.n == 0)
        return fail("the decode NVFP4 GEMM needs k divisible by 256 (<= 2048) and n divisible by 128");
    if (gated ? g.epilogue != EPI_SWIGLU_NVFP4 : g.epilogue != EPI_STORE_BF16)
        return fail("the decode NVFP4 GEMM writes NVFP4 SwiGLU rows (gated) or bf16 rows");
    if (g.beta != 0.0f || g.bias != nullptr)
        return fail("the decode NVFP4 GEMM has no beta / bias epilogue");
    if ((reinterpret_cast<uintptr_t>(g.a) & 15u) != 0 || (reinterpret_cast<uintptr_t>(g.b) & 15u) != 0
        || g.a_pitch_bytes != g.k / 2 || g.b_pitch_bytes != g.k / 2)
        return fail("the decode NVFP4 GEMM operands must be contiguous and 16-byte aligned");
    if (g.max_tiles == 0 || g.max_tiles > 65535)
        return fail("the decode NVFP4 GEMM launch grid is too large");

    SwapParams sp {};
    sp.n = g.n;
    sp.k_blocks = g.k / 256;
    sp.kgroups = g.k / 64;
    sp.b_rows = gated ? 2 * g.n : g.n;
    sp.num_fb = gated ? g.n / 64 : g.n / 128;
    sp.x = static_cast<const uint8_t*>(g.a);
    sp.x_sf = g.a_scale_tiled;
    sp.x_sf_linear = g.a_scale_linear;
    sp.row_tokens = g.row_tokens;
    sp.indptr = g.indptr;
    sp.pad_indptr = g.pad_indptr;
    sp.w_sf = g.b_scale_tiled;
    sp.w_sf_group_stride = qs3_nvfp4_tiled_scale_bytes(sp.b_rows, g.k);
    sp.tile_expert = g.tile_expert;
    sp.tile_row0 = g.tile_row0;
    sp.tile_nrows = g.tile_nrows;
    sp.total_tiles = g.total_tiles;
    sp.out = g.out;
    sp.out_sf = g.out_scale_tiled;
    sp.alpha = g.alpha;
    sp.group_scale = g.group_scale;
    sp.group_scale_up = g.group_scale_up;
    sp.out_global = g.out_global_scale == 0.0f ? 1.0f : g.out_global_scale;
    sp.tables_ready = g.tables_ready;
    sp.shared_group = g.shared_b != nullptr ? static_cast<int>(g.groups) : -1;
    sp.shared_w_sf = g.shared_b_scale_tiled;
    sp.shared_scale = g.shared_scale;
    sp.shared_scale_up = g.shared_scale_up;
    sp.err = device_error_word();

    const size_t fixed = 1024 + static_cast<size_t>(sp.k_blocks) * g.tile_rows * 128 + static_cast<size_t>(sp.kgroups) * 512
        + (gated ? kSwExBytes : 0) + kSwMiscBytes;
    // tensor memory: accumulators, 16 scale columns per stage, 2 x 4 token-scale columns per k group. Four accumulators
    // where they fit: handing one over takes longer than the MMAs of a feature block with a short k (down of a
    // 128-token batch 0.061 ms with two, 0.056 with four).
    sp.stages = static_cast<uint32_t>(std::min<size_t>(kSwMaxStages, (227 * 1024 - fixed) / kSwStageBytes));
    sp.acc_mask = 4 * g.tile_rows + 16 * sp.stages + 8 * sp.kgroups <= 512 ? 3 : 1;
    sp.stages = std::min(sp.stages, (512 - (sp.acc_mask + 1) * g.tile_rows - 8 * sp.kgroups) / 16);
    const size_t smem = fixed + static_cast<size_t>(sp.stages) * kSwStageBytes;
    const uint32_t grid = static_cast<uint32_t>(
        std::min<uint64_t>(static_cast<uint64_t>(g.max_tiles) * sp.num_fb, device_sm_count()));

    CUtensorMap mw, mws;
    bool mapped = make_operand_map(&mw, true, g.b, g.k / 2, static_cast<uint64_t>(g.groups) * sp.b_rows, g.k / 2,
                                   gated ? 64 : 128);
    mws = mw;
    if (mapped && g.shared_b != nullptr)
        mapped = make_operand_map(&mws, true, g.shared_b, g.k / 2, sp.b_rows, g.k / 2, gated ? 64 : 128);
    if (!mapped) {
        if (why != nullptr)
            *why = "cuTensorMapEncodeTiled failed";
        return cudaErrorInvalidValue;
    }
    if (g.tile_rows == 32)
        return gated ? launch_swap_instance<32, true>(mw, mws, sp, grid, smem, stream)
                     : launch_swap_instance<32, false>(mw, mws, sp, grid, smem, stream);
    return gated ? launch_swap_instance<64, true>(mw, mws, sp, grid, smem, stream)
                 : launch_swap_instance<64, false>(mw, mws, sp, grid, smem, stream);
}

} // namespace qs3
