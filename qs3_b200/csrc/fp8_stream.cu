// FP8 block-scaled grouped GEMM of experts with few rows: weight streaming with the operands swapped (weight rows are
// the M side of the MMA, the expert's token tile of up to 64 rows the N side).
//
//   unit   one token tile x 256 weight rows of its expert: gated: 128 gate rows and the 128 up rows of the same
//          features; plain: 256 features
//   grid   persistent, one CTA per SM, every gridDim.x-th unit: the CTAs of a round hold neighbouring units, so a
//          token tile and the weights of an expert with several tiles are read by several SMs at about the same time
//   smem   ring of stages: two weight tiles 128 x 128 B (32 KB) + token tile NT x 128 B, whose rows lie together or are
//          found through the routing tables (gather4); notes of the coming units (rows, scales)
//   TMEM   kFsBufs buffers of two NT-column accumulators (lane = weight row, column = token), one per k block: the
//          block scales are promoted outside the tensor core, acc += w_scale * x_scale * partial, in f32
//   warps  0-7 promotion and epilogue (lane quadrant warp % 4, token half warp / 4; both accumulators, so SwiGLU
//          needs no exchange), 8 producer (TMA), 9 MMA issuer, 10-11 note writers: they follow the tables and fetch
//          the scales of the units to come, two to four ahead. With HBM busy a dependent load takes over a
//          microsecond; the promotion warps doing this between two units lost 5 us of every 12.
//
// Bound by HBM while experts have few rows: hit experts * weight bytes. A k block's 32 KB of weights take an SM about
// 1400 cycles, its promotion (2 x 128 x 64 elements) about 400. 128 experts top-8 (hidden 2048, intermediate 768): 64
// tokens gate_up 0.071 ms (5.7 TB/s), down 0.034; layer of 1 token 0.041 -> 0.033, 64 tokens of a skewed router 0.091 ->
// 0.070, 256 tokens 0.183 -> 0.136 against a kernel of 16-row tiles with two CTAs per SM; 512 tokens 0.166 -> 0.149
// against 128-row tiles. Tiles of 32 rows are no faster at any size (64 tokens 0.123 against 0.123 ms, 400: 0.141
// against 0.144) and slower above.
#include "tcgen05.cuh"

#include <algorithm>

namespace qs3 {
namespace {

using namespace tc;

constexpr uint32_t NT = 64; // token rows per tile
constexpr int kFsThreads = 384;
constexpr uint32_t kFsBufs = 4;
constexpr uint32_t kFsStages = 5;
constexpr uint32_t kFsMaxKBlocks = 32; // k <= 4096: one weight scale of a 128-feature block per lane
constexpr uint32_t kFsBox = 32;         // rows of one copy where the token rows lie together
constexpr uint32_t kFsMaxNotes = 4;    // as many as the scales have room for: 4 up to 16 k blocks, 2 at 32

enum : uint32_t {
    ERR_FS_FULL_WAIT = 0x5b000001u,
    ERR_FS_EMPTY_WAIT = 0x5b000002u,
    ERR_FS_ACC_FULL_WAIT = 0x5b000003u,
    ERR_FS_ACC_EMPTY_WAIT = 0x5b000004u,
    ERR_FS_NOTE_FULL_WAIT = 0x5b000005u,
    ERR_FS_NOTE_EMPTY_WAIT = 0x5b000006u,
};

struct Fp8StreamParams {
    uint32_t n;              // output features per group (gated: intermediate size); multiple of 128
    uint32_t k_blocks;       // k / 128
    uint32_t b_rows;         // weight rows per group (gated: 2 n)
    uint32_t units_per_tile; // gated: n / 128; plain: ceil(n / 256)
    uint32_t num_fb;         // n / 128
    const float* x_scale;    // [rows of x, k_blocks]
    const float* w_scale;    // [groups, b_rows / 128, k_blocks]
    const int32_t* tile_expert;
    const int32_t* tile_row0;
    const int32_t* tile_nrows;
    const int32_t* total_tiles;
    const int32_t* row_tokens; // NULL: x rows are the padded rows; else dense row -> x row
    const int32_t* indptr;     // with row_tokens: segment starts, dense and padded
    const int32_t* pad_indptr;
    int gathered;              // rows of experts with more than kGatherRows rows are in map_g, padded
    int tables_ready;        // the tables were complete before the predecessor in the stream started
    void* out;               // gated: e4m3 codes [rows, n]; else bf16 [rows, n]
    float* out_scale;        // gated: f32 [rows, n / 128]
    uint32_t* err;
};

// What the other warps need to know about a unit.
struct FsNote {
    int row0, nrows, w_row, w_row2, boxes; // boxes: the token rows lie together (in map_g)
    int row[NT];                 // x row of each row of the tile (the last one's past the end)
    float ws[2][kFsMaxKBlocks];  // block scales of the two weight tiles
};

struct FsSmem {
    static constexpr uint32_t kStageBytes = 2 * kTileBytes + NT * 128;
    static constexpr uint32_t kScales = kFsStages * kStageBytes;                // [notes][k blocks][NT] f32
    static constexpr uint32_t kAmax = kScales + 2 * kFsMaxKBlocks * NT * 4;     // [4][NT] f32
    static constexpr uint32_t kNotes = kAmax + 4 * NT * 4;
    static constexpr uint32_t kBars = kNotes + kFsMaxNotes * static_cast<uint32_t>(sizeof(FsNote));
    static constexpr uint32_t kBytes = kBars + (2 * kFsStages + 2 * kFsBufs + 2 * kFsMaxNotes) * 8 + 16;
};

template <bool GATED>
__global__ void __launch_bounds__(kFsThreads, 1)
gemm_fp8_stream_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                       const __grid_constant__ CUtensorMap map_g, // boxes of padded rows
                       const Fp8StreamParams p)
{
    using S = FsSmem;
    constexpr uint32_t kBufCols = 2 * NT;
    constexpr uint32_t kTmemCols = kFsBufs * kBufCols;
    constexpr uint32_t HT = NT / 2; // tokens of one warp
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    float* s_xs = reinterpret_cast<float*>(smem + S::kScales);
    float* s_amax = reinterpret_cast<float*>(smem + S::kAmax);
    FsNote* s_note = reinterpret_cast<FsNote*>(smem + S::kNotes);
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + S::kBars);
    uint64_t* empty_bar = full_bar + kFsStages;
    uint64_t* acc_full = empty_bar + kFsStages;
    uint64_t* acc_empty = acc_full + kFsBufs;
    uint64_t* note_full = acc_empty + kFsBufs;
    uint64_t* note_empty = note_full + kFsMaxNotes;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(note_empty + kFsMaxNotes);
    volatile uint32_t* abort_flag = tmem_slot + 1;

    const uint32_t warp = threadIdx.x >> 5;
    const uint32_t lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < kFsStages; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        for (uint32_t b = 0; b < kFsBufs; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], 8); // one arrival per promotion warp
        }
        for (uint32_t b = 0; b < kFsMaxNotes; ++b) {
            mbar_init(&note_full[b], 2);   // the two writers
            mbar_init(&note_empty[b], 10); // promotion warps, producer, issuer
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 9) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const bool early = p.tables_ready && (warp == 8 || warp >= 10); // weights and tables are complete: no need to wait for them
    if (!early)
        chain_begin();

    const uint32_t total = static_cast<uint32_t>(*p.total_tiles) * p.units_per_tile;
    const uint32_t notes = min(kFsMaxNotes, 2 * kFsMaxKBlocks / p.k_blocks);
    // note of the next unit in turn; every reader takes each one and gives it back
    uint32_t nt = 0, nph = 0;
    const auto next_note = [&] {
        if (++nt == notes) {
            nt = 0;
            nph ^= 1;
        }
    };

    if (warp >= 10) {
        // -------------------------------------------------------- note writers --
        const uint32_t i = threadIdx.x - 320;
        bool waited = !early;
        for (uint32_t u = blockIdx.x; u < total; u += gridDim.x, next_note()) {
            const uint32_t tile = u / p.units_per_tile, nb = u % p.units_per_tile;
            const int row0 = p.tile_row0[tile], nrows = p.tile_nrows[tile], expert = p.tile_expert[tile];
            const uint32_t fb = GATED ? nb : 2 * nb;
            // (the last plain unit of an odd feature-block count takes its own tile twice and drops the second result)
            const uint32_t fb2 = GATED ? p.num_fb + nb : min(2 * nb + 1, p.num_fb - 1);
            const int j = min(static_cast<int>(i % NT), nrows - 1);
            int row = row0 + j;
            bool boxes = true;
            if (p.row_tokens != nullptr) {
                const int dense = p.indptr[expert];
                row = p.row_tokens[dense + row - p.pad_indptr[expert]];
                boxes = p.gathered && p.indptr[expert + 1] - dense > static_cast<int>(kGatherRows);
            }
            if (!waited)
                chain_begin();
            waited = true;
            if (!__all_sync(0xffffffffu, mbar_wait(&note_empty[nt], nph ^ 1, abort_flag, p.err, ERR_FS_NOTE_EMPTY_WAIT)))
                break;
            FsNote& note = s_note[nt];
            const float* xs = p.x_scale + static_cast<size_t>(row) * p.k_blocks;
            for (uint32_t kb = i / NT; kb < p.k_blocks; kb += 64 / NT)
                cp_async4(s_xs + (nt * p.k_blocks + kb) * NT + i % NT, xs + kb);
            if (lane < p.k_blocks)
                cp_async4(&note.ws[warp - 10][lane], p.w_scale
                              + (static_cast<size_t>(expert) * (p.b_rows / 128) + (warp == 10 ? fb : fb2)) * p.k_blocks + lane);
            if (i < NT)
                note.row[i] = row;
            if (i == 0) {
                note.row0 = row0;
                note.nrows = nrows;
                note.boxes = boxes;
                note.w_row = expert * static_cast<int>(p.b_rows) + static_cast<int>(fb * 128);
                note.w_row2 = expert * static_cast<int>(p.b_rows) + static_cast<int>(fb2 * 128);
            }
            cp_async_wait();
            __syncwarp();
            if (lane == 0)
                mbar_arrive(&note_full[nt]);
        }
        if (!waited)
            chain_begin();
    } else if (warp == 8) {
        // ------------------------------------------------------------ producer --
        // Lane 0 loads the weight tiles, lane j rows 4 j .. 4 j + 3 of the token tile; rows past its last are not moved.
        // A gather4 takes the copy engine about 80 cycles, so rows that lie together come in boxes.
        uint32_t s = 0, ph = 0;
        bool ok = true;
        uint32_t ahead = 0; // k blocks of the first unit whose weights are on their way already
        if (early) {
            if (blockIdx.x < total && elect_one()) {
                const uint32_t tile = blockIdx.x / p.units_per_tile, nb = blockIdx.x % p.units_per_tile;
                const uint32_t fb = GATED ? nb : 2 * nb, fb2 = GATED ? p.num_fb + nb : min(2 * nb + 1, p.num_fb - 1);
                const int w0 = p.tile_expert[tile] * static_cast<int>(p.b_rows);
                for (; ahead < min(kFsStages, p.k_blocks); ++ahead) {
                    uint8_t* sw = smem + ahead * S::kStageBytes;
                    mbar_expect_tx_only(&full_bar[ahead], 2 * kTileBytes);
                    tma_load_2d(sw, &map_w, &full_bar[ahead], static_cast<int>(ahead) * 128, w0 + static_cast<int>(fb * 128));
                    tma_load_2d(sw + kTileBytes, &map_w, &full_bar[ahead], static_cast<int>(ahead) * 128, w0 + static_cast<int>(fb2 * 128));
                }
            }
            __syncwarp();
            chain_begin();
        }
        for (uint32_t u = blockIdx.x; u < total && ok; u += gridDim.x, next_note(), ahead = 0) {
            ok = __all_sync(0xffffffffu, mbar_wait<true>(&note_full[nt], nph, abort_flag, p.err, ERR_FS_NOTE_FULL_WAIT));
            if (!ok)
                break;
            const FsNote& note = s_note[nt];
            const int nrows = note.nrows, w_row = note.w_row, w_row2 = note.w_row2, row0 = note.row0;
            const bool boxes = note.boxes;
            const uint32_t part_rows = boxes ? kFsBox : 4u, parts = (static_cast<uint32_t>(nrows) + part_rows - 1) / part_rows;
            int row[4];
#pragma unroll
            for (int q = 0; q < 4; ++q)
                row[q] = note.row[min(lane * 4 + q, NT - 1)];
            __syncwarp();
            if (lane == 0)
                mbar_arrive(&note_empty[nt]);
            for (uint32_t kb = 0; kb < p.k_blocks; ++kb) {
                ok = __all_sync(0xffffffffu, mbar_wait<true>(&empty_bar[s], ph ^ 1, abort_flag, p.err, ERR_FS_EMPTY_WAIT));
                if (!ok)
                    break;
                uint8_t* sw = smem + s * S::kStageBytes;
                const int c0 = static_cast<int>(kb) * 128;
                if (elect_one()) {
                    mbar_expect_tx(&full_bar[s], (kb < ahead ? 0 : 2 * kTileBytes) + parts * part_rows * 128);
                    if (kb >= ahead) {
                        tma_load_2d(sw, &map_w, &full_bar[s], c0, w_row);
                        tma_load_2d(sw + kTileBytes, &map_w, &full_bar[s], c0, w_row2);
                    }
                }
                __syncwarp();
                if (lane < parts) {
                    uint8_t* dst = sw + 2 * kTileBytes + lane * part_rows * 128;
                    if (boxes)
                        tma_load_2d(dst, &map_g, &full_bar[s], c0, row0 + static_cast<int>(lane * kFsBox));
                    else
                        tma_gather4(dst, &map_x, &full_bar[s], c0, row);
                }
                if (++s == kFsStages) {
                    s = 0;
                    ph ^= 1;
                }
            }
        }
    } else if (warp == 9) {
        // ---------------------------------------------------------- MMA issuer --
        if (elect_one()) {
            uint32_t s = 0, ph = 0, b = 0, bph = 0;
            bool ok = true;
            for (uint32_t u = blockIdx.x; u < total && ok; u += gridDim.x, next_note()) {
                if (!mbar_wait<true>(&note_full[nt], nph, abort_flag, p.err, ERR_FS_NOTE_FULL_WAIT))
                    break;
                // M = 128 weight rows, N = the tile's rows (a multiple of 16), e4m3 x e4m3 -> f32, both K-major
                const uint32_t cols = (static_cast<uint32_t>(s_note[nt].nrows) + 15u) & ~15u;
                mbar_arrive(&note_empty[nt]);
                const uint32_t idesc = (1u << 4) | ((cols >> 3) << 17) | ((kBM >> 4) << 24);
                for (uint32_t kb = 0; kb < p.k_blocks; ++kb) {
                    if (!mbar_wait<true>(&acc_empty[b], bph ^ 1, abort_flag, p.err, ERR_FS_ACC_EMPTY_WAIT)
                        || !mbar_wait<true>(&full_bar[s], ph, abort_flag, p.err, ERR_FS_FULL_WAIT)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t sw = smem_u32(smem + s * S::kStageBytes);
                    const uint64_t dw = operand_desc(sw), dw2 = operand_desc(sw + kTileBytes);
                    const uint64_t dx = operand_desc(sw + 2 * kTileBytes);
                    const uint32_t d = tmem_base + b * kBufCols;
#pragma unroll
                    for (uint32_t j = 0; j < 4; ++j) {
                        tc_mma_f8(d, dw + 2 * j, dx + 2 * j, idesc, j > 0 ? 1u : 0u);
                        tc_mma_f8(d + NT, dw2 + 2 * j, dx + 2 * j, idesc, j > 0 ? 1u : 0u);
                    }
                    tc_commit(&empty_bar[s]);
                    tc_commit(&acc_full[b]);
                    if (++s == kFsStages) {
                        s = 0;
                        ph ^= 1;
                    }
                    if (++b == kFsBufs) {
                        b = 0;
                        bph ^= 1;
                    }
                }
            }
        }
    } else {
        // ------------------------------------------------- promotion, epilogue --
        const uint32_t quad = warp & 3, half = warp >> 2;
        const uint32_t lane_base = (quad * 32) << 16;
        const uint32_t r = quad * 32 + lane; // feature within a tile = TMEM lane
        const int t0 = static_cast<int>(half * HT);
        uint32_t b = 0, bph = 0;
        for (uint32_t u = blockIdx.x; u < total; u += gridDim.x, next_note()) {
            bool ok = __all_sync(0xffffffffu, mbar_wait(&note_full[nt], nph, abort_flag, p.err, ERR_FS_NOTE_FULL_WAIT));
            const FsNote& note = s_note[nt];
            const int nrows = note.nrows;
            const uint32_t row0 = static_cast<uint32_t>(note.row0), nb = u % p.units_per_tile;
            float acc[2][HT];
#pragma unroll
            for (uint32_t t = 0; t < HT; ++t)
                acc[0][t] = acc[1][t] = 0.0f;
            for (uint32_t kb = 0; kb < p.k_blocks && ok; ++kb) {
                ok = __all_sync(0xffffffffu, mbar_wait(&acc_full[b], bph, abort_flag, p.err, ERR_FS_ACC_FULL_WAIT));
                if (!ok)
                    break;
                tc_fence_after();
                const float s0 = note.ws[0][kb], s1 = note.ws[1][kb];
                const float4* xs = reinterpret_cast<const float4*>(s_xs + (nt * p.k_blocks + kb) * NT + t0);
#pragma unroll
                for (uint32_t c = 0; c < HT / 16; ++c) {
                    if (t0 + static_cast<int>(c) * 16 < nrows) { // uniform
                        const uint32_t src = tmem_base + lane_base + b * kBufCols + t0 + c * 16;
                        uint32_t va[16], vb[16];
                        tc_ld16(src, va);
                        tc_ld16(src + NT, vb);
                        tc_ld_wait();
#pragma unroll
                        for (uint32_t q = 0; q < 4; ++q) {
                            const float4 x = xs[c * 4 + q];
                            const float xv[4] = { x.x, x.y, x.z, x.w };
#pragma unroll
                            for (uint32_t j = 0; j < 4; ++j) {
                                const uint32_t t = c * 16 + q * 4 + j;
                                acc[0][t] = fmaf(__uint_as_float(va[q * 4 + j]), s0 * xv[j], acc[0][t]);
                                acc[1][t] = fmaf(__uint_as_float(vb[q * 4 + j]), s1 * xv[j], acc[1][t]);
                            }
                        }
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0)
                    mbar_arrive(&acc_empty[b]);
                if (++b == kFsBufs) {
                    b = 0;
                    bph ^= 1;
                }
            }
            __syncwarp();
            if (lane == 0)
                mbar_arrive(&note_empty[nt]);
            // (the unrolled steps below are kept short: their instructions are fetched with HBM busy)
            const int live = nrows - t0;
            if constexpr (GATED) {
                // SwiGLU, then one e4m3 scale per token and 128 features: the four lane quadrants exchange their maxima
#pragma unroll
                for (uint32_t t = 0; t < HT; ++t) {
                    if (static_cast<int>(t) >= live)
                        break;
                    const float g = acc[0][t];
                    acc[0][t] = __fdividef(g, 1.0f + __expf(-g)) * acc[1][t];
                    const uint32_t m = __reduce_max_sync(0xffffffffu, __float_as_uint(fabsf(acc[0][t])));
                    if (lane == 0)
                        s_amax[quad * NT + t0 + t] = __uint_as_float(m);
                }
                ok = group_all(1 + half, 128, ok); // the half's four warps stop together
                if (!ok)
                    break;
                if (r < HT && static_cast<int>(r) < live) {
                    float* a = s_amax + t0 + r;
                    const float sc = fmaxf(__fdiv_rn(fmaxf(fmaxf(a[0], a[NT]), fmaxf(a[2 * NT], a[3 * NT])), 448.0f), 1.0e-30f);
                    a[0] = __fdiv_rn(1.0f, sc);
                    p.out_scale[static_cast<size_t>(row0 + t0 + r) * p.num_fb + nb] = sc;
                }
                asm volatile("bar.sync %0, 128;" ::"r"(1 + half) : "memory");
                uint8_t* out = static_cast<uint8_t*>(p.out) + static_cast<size_t>(row0 + t0) * p.n + nb * 128 + r;
#pragma unroll
                for (uint32_t t = 0; t < HT; ++t) {
                    if (static_cast<int>(t) >= live)
                        break;
                    *out = f32_to_e4m3_sat(__fmul_rn(acc[0][t], s_amax[t0 + t]));
                    out += p.n;
                }
                asm volatile("bar.sync %0, 128;" ::"r"(1 + half) : "memory"); // all have read: the next unit may write
            } else {
                if (!ok)
                    break;
                const uint32_t f = nb * 256 + r;
                const bool second = f + 128 < p.n;
                __nv_bfloat16* out = static_cast<__nv_bfloat16*>(p.out) + static_cast<size_t>(row0 + t0) * p.n + f;
#pragma unroll
                for (uint32_t t = 0; t < HT; ++t) {
                    if (static_cast<int>(t) >= live)
                        break;
                    *out = __float2bfloat16(acc[0][t]);
                    if (second)
                        out[128] = __float2bfloat16(acc[1][t]);
                    out += p.n;
                }
            }
        }
    }

    // ---- teardown ----
    tc_fence_before();
    __syncthreads();
    if (warp == 9) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols)
                     : "memory");
    }
}

template <bool GATED>
cudaError_t launch_stream_instance(const CUtensorMap& mw, const CUtensorMap& mx, const CUtensorMap& mg,
                                   const Fp8StreamParams& fp, uint32_t grid, cudaStream_t stream)
{
    auto kernel = gemm_fp8_stream_kernel<GATED>;
    constexpr size_t smem = 1024 + FsSmem::kBytes;
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
    return launch_chained(kernel, dim3(grid), kFsThreads, smem, stream, mw, mx, mg, fp);
}

} // namespace

cudaError_t launch_fp8_stream_gemm(const Fp8Gemm& g, cudaStream_t stream, const char** why)
{
    Fp8StreamParams fp {};
    fp.n = g.n;
    fp.k_blocks = g.k / 128;
    fp.b_rows = g.gated ? 2 * g.n : g.n;
    fp.num_fb = g.n / 128;
    fp.units_per_tile = g.gated ? g.n / 128 : (g.n + 255) / 256;
    fp.x_scale = g.x_scale;
    fp.w_scale = g.w_scale;
    fp.tile_expert = g.tile_expert;
    fp.tile_row0 = g.tile_row0;
    fp.tile_nrows = g.tile_nrows;
    fp.total_tiles = g.total_tiles;
    fp.row_tokens = g.row_tokens;
    fp.indptr = g.indptr;
    fp.pad_indptr = g.pad_indptr;
    fp.gathered = g.gathered != nullptr;
    fp.tables_ready = g.tables_ready;
    fp.out = g.out;
    fp.out_scale = g.out_scale;
    fp.err = device_error_word();
    CUtensorMap mw, mx, mg;
    bool ok = make_operand_map(&mw, true, g.w, g.k, static_cast<uint64_t>(g.groups) * fp.b_rows, g.k, 128);
    if (g.row_tokens == nullptr) {
        ok = ok && make_operand_map(&mg, true, g.x, g.k, g.x_rows, g.k, kFsBox);
        mx = mg;
    } else {
        ok = ok && make_operand_map(&mx, true, g.x, g.k, g.x_rows, g.k, 1);
        mg = mx;
        if (g.gathered != nullptr)
            ok = ok && make_operand_map(&mg, true, g.gathered, g.k, g.out_rows, g.k, kFsBox);
    }
    if (!ok) {
        if (why != nullptr)
            *why = "cuTensorMapEncodeTiled failed";
        return cudaErrorInvalidValue;
    }
    const uint32_t grid = static_cast<uint32_t>(
        std::min<uint64_t>(static_cast<uint64_t>(g.max_tiles) * fp.units_per_tile, device_sm_count()));
    return g.gated ? launch_stream_instance<true>(mw, mx, mg, fp, grid, stream)
                   : launch_stream_instance<false>(mw, mx, mg, fp, grid, stream);
}

} // namespace qs3
