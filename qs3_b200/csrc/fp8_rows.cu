// FP8 block-scaled grouped GEMM for experts with more rows than a decode batch gives them (fp8_stream.cu has the kernel
// for those): token rows are the M side of the MMA again.
//
// A 128 x 256 output tile per unit: 128 token rows of one expert x 256 weight rows (gated: 128 gate rows and the
// 128 up rows of the same features). The block scales are promoted outside the tensor core as in the streaming
// kernel, but with tokens in the tensor-memory lanes a lane needs ONE factor per k block and 128-feature block
// (x_scale[token] * w_scale[block]), so promoting an element is a single FMA without any shared-memory operand.
//
//   persistent  one CTA per SM, every gridDim.x-th (token tile, feature block) unit: the CTAs of a round hold
//               neighbouring units, so a token tile and the weights of an expert with several tiles are read by
//               several SMs at about the same time (contiguous ranges: gate_up 0.231, down 0.106 ms of the case below)
//   smem        ring of stages: A 128 x 128 B, B 256 x 128 B; plain: + four 16-KB boxes staging the bf16 tile for
//               TMA stores
//   TMEM        two 256-column buffers: k block i + 1 is multiplied while k block i is promoted
//   warps       0-15 promotion and epilogue (lane quadrant warp % 4, column quarter warp / 4), 16 producer, 17 MMA, 18-19
//               note writers: they follow the tables and fetch the scales of the next unit
//
// Bound by the hand-over of the two buffers: products, commit, the promotion's wait and the way back take a buffer 1.3 us,
// 0.65 a k block, of which the four MMAs are 0.35 (690 cycles). 4096 tokens, gate_up and down: 164 and 90 us; without the
// loads (48 KB a k block) 157 and 82, without the promotion 148 and 86, without both still 136 and 68. With few rows an expert
// the weights bound it: 1024 tokens 91 and 51, without the loads 72 and 38. 4096 tokens x 128 experts top-8 (hidden 2048, intermediate 768): gate_up 0.800 -> 0.156 ms, down 0.238
// -> 0.087 ms against the decode kernel on 32-row tiles, which streamed every weight through shared memory once per 32
// rows. With the scales and tables fetched between the units by the promotion warps, and whole token tiles moved for a
// few rows: layer of 1024 tokens 0.200 -> 0.177 ms, 2048 0.257 -> 0.222 (4096: 0.377 -> 0.366). Eight promotion warps
// with one tensor-memory read in flight each and an FMA per element took as long as the operands; four warps per
// scheduler, two elements per FMA and the buffer given back as soon as it is read: 1024 tokens 0.180 -> 0.174 ms, 2048
// 0.218 -> 0.211, 4096 0.380 -> 0.374. (Pairs of CTAs with half of B each, 32 KB a k block, were slower, 0.341 -> 0.389 ms:
// a buffer's way to the other CTA and back takes longer than the two buffers cover.)
#include "tcgen05.cuh"

#include <algorithm>

namespace qs3 {
namespace {

using namespace tc;

constexpr uint32_t kFrAdders = 16;                    // promotion warps
constexpr int kFrThreads = (kFrAdders + 4) * 32;
constexpr uint32_t kFrN = 256;                        // weight rows per unit = MMA N
constexpr uint32_t kFrStageBytes = 3 * kTileBytes;    // A tile + two B tiles
constexpr uint32_t kFrMaxStages = 4;
constexpr uint32_t kFrTmemCols = 512;
constexpr uint32_t kFrMaxKBlocks = 32;                // k <= 4096
constexpr uint32_t kFrMaxNotes = 2;
constexpr uint32_t kFrBox = 32;                       // token rows of one copy

enum : uint32_t {
    ERR_FR_FULL_WAIT = 0x58000001u,
    ERR_FR_EMPTY_WAIT = 0x58000002u,
    ERR_FR_ACC_FULL_WAIT = 0x58000003u,
    ERR_FR_ACC_EMPTY_WAIT = 0x58000004u,
    ERR_FR_NOTE_FULL_WAIT = 0x58000005u,
    ERR_FR_NOTE_EMPTY_WAIT = 0x58000006u,
};

struct Fp8RowsParams {
    uint32_t n;            // output features per group (gated: intermediate size); multiple of 128
    uint32_t k_blocks;     // k / 128
    uint32_t b_rows;       // weight rows per group (gated: 2 n)
    uint32_t units_per_tile; // gated: n / 128; plain: ceil(n / 256)
    uint32_t num_fb;       // n / 128
    const float* x_scale;  // [rows, k_blocks]
    const float* w_scale;  // [groups, b_rows / 128, k_blocks]
    const int32_t* tile_expert;
    const int32_t* tile_row0;
    const int32_t* tile_nrows;
    const int32_t* total_tiles;
    const int32_t* row_tokens; // NULL: scales by padded row; else dense row -> row of x_scale
    const int32_t* indptr;     // with row_tokens: segment starts, dense and padded
    const int32_t* pad_indptr;
    void* out;             // gated: e4m3 codes [rows, n]; plain: written through map_o
    float* out_scale;      // gated: f32 [rows, n / 128]
    uint32_t* err;
};

// What the other warps need to know about a unit.
struct FrNote {
    int row0, nrows, b_row, b_row2;
    float ws[2][kFrMaxKBlocks];  // block scales of the two B tiles
};

template <bool GATED> struct FrSmem {
    static constexpr uint32_t kStages = GATED ? kFrMaxStages : kFrMaxStages - 1;
    static constexpr uint32_t kScaleRows = GATED ? 48 : 32; // k blocks of activation scales held, over all notes
    static constexpr uint32_t kStaging = kStages * kFrStageBytes;               // plain: four 16-KB boxes
    static constexpr uint32_t kScales = kStaging + (GATED ? 0 : 4 * kTileBytes); // [notes][k blocks][128] f32
    static constexpr uint32_t kNotes = kScales + kScaleRows * 128 * 4;
    static constexpr uint32_t kAmax = kNotes + kFrMaxNotes * static_cast<uint32_t>(sizeof(FrNote)); // gated: [4][128] f32
    static constexpr uint32_t kBars = kAmax + (GATED ? 2048 : 0);
    static constexpr uint32_t kBytes = kBars + (2 * kFrMaxStages + 4 + 2 * kFrMaxNotes) * 8 + 16;
};

// a * b + c of two values, each as fmaf
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c)
{
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ uint64_t pack2(uint32_t a, uint32_t b) { return static_cast<uint64_t>(b) << 32 | a; }
__device__ __forceinline__ float part2(uint64_t v, uint32_t i) { return __uint_as_float(static_cast<uint32_t>(v >> (32 * i))); }

template <bool GATED>
__global__ void __launch_bounds__(kFrThreads, 1)
gemm_fp8_rows_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w,
                     const __grid_constant__ CUtensorMap map_o, const Fp8RowsParams p)
{
    using S = FrSmem<GATED>;
    constexpr uint32_t kStages = S::kStages;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    uint8_t* staging = smem + S::kStaging;
    float* s_xs = reinterpret_cast<float*>(smem + S::kScales);
    FrNote* s_note = reinterpret_cast<FrNote*>(smem + S::kNotes);
    float* s_amax = reinterpret_cast<float*>(smem + S::kAmax);
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + S::kBars);
    uint64_t* empty_bar = full_bar + kFrMaxStages;
    uint64_t* acc_full = empty_bar + kFrMaxStages;
    uint64_t* acc_empty = acc_full + 2;
    uint64_t* note_full = acc_empty + 2;
    uint64_t* note_empty = note_full + kFrMaxNotes;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(note_empty + kFrMaxNotes);
    volatile uint32_t* abort_flag = tmem_slot + 1;

    const uint32_t warp = threadIdx.x >> 5;
    const uint32_t lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < kStages; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], kFrAdders); // one arrival per promotion warp
        }
        for (uint32_t b = 0; b < kFrMaxNotes; ++b) {
            mbar_init(&note_full[b], 2);              // the two writers
            mbar_init(&note_empty[b], kFrAdders + 1); // promotion warps, producer
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == kFrAdders + 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(kFrTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    // weights and tables (the predecessor is the gather or the gate_up GEMM) are complete: who reads only them need not wait
    const bool early = warp == kFrAdders || warp >= kFrAdders + 2;
    if (!early)
        chain_begin();

    // units of this CTA: every gridDim.x-th one. The CTAs of a round hold neighbouring units, so that a token tile
    // and the weights of an expert with several tiles are read by several SMs at about the same time
    const uint32_t total = static_cast<uint32_t>(*p.total_tiles) * p.units_per_tile;
    const uint32_t notes = max(1u, min(kFrMaxNotes, S::kScaleRows / p.k_blocks));
    // note of the next unit in turn; every reader takes each one and gives it back
    uint32_t nt = 0, nph = 0;
    const auto next_note = [&] {
        if (++nt == notes) {
            nt = 0;
            nph ^= 1;
        }
    };
    // the B tiles of a unit, as 128-row blocks of the expert: gate and up rows of the same features, or two successive
    // blocks (the last unit of an odd count takes its own twice and drops the second result)
    const auto b_block = [&](uint32_t nb) { return GATED ? nb : 2 * nb; };
    const auto b_block2 = [&](uint32_t nb) { return GATED ? p.num_fb + nb : min(2 * nb + 1, p.num_fb - 1); };

    if (warp >= kFrAdders + 2) {
        // -------------------------------------------------------- note writers --
        const uint32_t i = threadIdx.x - (kFrAdders + 2) * 32, w = i / 32;
        bool waited = false;
        for (uint32_t u = blockIdx.x; u < total; u += gridDim.x, next_note()) {
            const uint32_t tile = u / p.units_per_tile, nb = u % p.units_per_tile;
            const int row0 = p.tile_row0[tile], nrows = p.tile_nrows[tile], expert = p.tile_expert[tile];
            int row[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                row[h] = row0 + min(static_cast<int>(i) + 64 * h, nrows - 1);
                if (p.row_tokens != nullptr)
                    row[h] = p.row_tokens[p.indptr[expert] + row[h] - p.pad_indptr[expert]];
            }
            if (!waited)
                chain_begin();
            waited = true;
            if (!__all_sync(0xffffffffu, mbar_wait(&note_empty[nt], nph ^ 1, abort_flag, p.err, ERR_FR_NOTE_EMPTY_WAIT)))
                break;
            FrNote& note = s_note[nt];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float* xs = p.x_scale + static_cast<size_t>(row[h]) * p.k_blocks;
                for (uint32_t kb = 0; kb < p.k_blocks; ++kb)
                    cp_async4(s_xs + (nt * p.k_blocks + kb) * 128 + i + 64 * h, xs + kb);
            }
            const uint32_t fb = w == 0 ? b_block(nb) : b_block2(nb);
            if (lane < p.k_blocks)
                cp_async4(&note.ws[w][lane],
                          p.w_scale + (static_cast<size_t>(expert) * (p.b_rows / 128) + fb) * p.k_blocks + lane);
            if (i == 0) {
                note.row0 = row0;
                note.nrows = nrows;
                note.b_row = expert * static_cast<int>(p.b_rows) + static_cast<int>(b_block(nb) * 128);
                note.b_row2 = expert * static_cast<int>(p.b_rows) + static_cast<int>(b_block2(nb) * 128);
            }
            cp_async_wait();
            __syncwarp();
            if (lane == 0)
                mbar_arrive(&note_full[nt]);
        }
        if (!waited)
            chain_begin();
    } else if (warp == kFrAdders) {
        // ------------------------------------------------------------ producer --
        // Lane 0 loads the weight tiles, lane j box j of the token tile: boxes past its last row are not moved.
        uint32_t s = 0, ph = 0;
        bool ok = true;
        uint32_t ahead = 0; // k blocks of the first unit whose weights are on their way already
        if (blockIdx.x < total && lane == 0) {
            const uint32_t tile = blockIdx.x / p.units_per_tile, nb = blockIdx.x % p.units_per_tile;
            const int b0 = p.tile_expert[tile] * static_cast<int>(p.b_rows);
            for (; ahead < min(kStages, p.k_blocks); ++ahead) {
                uint8_t* sa = smem + ahead * kFrStageBytes;
                const int c0 = static_cast<int>(ahead * 128);
                mbar_expect_tx_only(&full_bar[ahead], 2 * kTileBytes);
                tma_load_2d(sa + kTileBytes, &map_w, &full_bar[ahead], c0, b0 + static_cast<int>(b_block(nb) * 128));
                tma_load_2d(sa + 2 * kTileBytes, &map_w, &full_bar[ahead], c0, b0 + static_cast<int>(b_block2(nb) * 128));
            }
        }
        __syncwarp();
        chain_begin();
        for (uint32_t u = blockIdx.x; u < total && ok; u += gridDim.x, next_note(), ahead = 0) {
            ok = __all_sync(0xffffffffu, mbar_wait<true>(&note_full[nt], nph, abort_flag, p.err, ERR_FR_NOTE_FULL_WAIT));
            if (!ok)
                break;
            const FrNote& note = s_note[nt];
            const int nrows = note.nrows, b_row = note.b_row, b_row2 = note.b_row2, row0 = note.row0;
            const uint32_t boxes = (static_cast<uint32_t>(nrows) + kFrBox - 1) / kFrBox;
            __syncwarp();
            if (lane == 0)
                mbar_arrive(&note_empty[nt]);
            for (uint32_t kb = 0; kb < p.k_blocks; ++kb) {
                ok = __all_sync(0xffffffffu, mbar_wait<true>(&empty_bar[s], ph ^ 1, abort_flag, p.err, ERR_FR_EMPTY_WAIT));
                if (!ok)
                    break;
                uint8_t* sa = smem + s * kFrStageBytes;
                const int c0 = static_cast<int>(kb * 128);
                if (lane == 0) {
                    mbar_expect_tx(&full_bar[s], (kb < ahead ? 0 : 2 * kTileBytes) + boxes * kFrBox * 128);
                    if (kb >= ahead) {
                        tma_load_2d(sa + kTileBytes, &map_w, &full_bar[s], c0, b_row);
                        tma_load_2d(sa + 2 * kTileBytes, &map_w, &full_bar[s], c0, b_row2);
                    }
                }
                __syncwarp();
                if (lane < boxes)
                    tma_load_2d(sa + lane * kFrBox * 128, &map_x, &full_bar[s], c0, row0 + static_cast<int>(lane * kFrBox));
                if (++s == kStages) {
                    s = 0;
                    ph ^= 1;
                }
            }
        }
    } else if (warp == kFrAdders + 1) {
        // ---------------------------------------------------------- MMA issuer --
        if (lane == 0) {
            // M = 128 tokens, N = 256 weight rows, e4m3 x e4m3 -> f32, both operands K-major
            constexpr uint32_t kIdesc = (1u << 4) | ((kFrN >> 3) << 17) | ((kBM >> 4) << 24);
            uint32_t s = 0, ph = 0, b = 0, bph = 0;
            bool ok = true;
            for (uint32_t u = blockIdx.x; u < total && ok; u += gridDim.x) {
                for (uint32_t kb = 0; kb < p.k_blocks; ++kb) {
                    if (!mbar_wait<true>(&acc_empty[b], bph ^ 1, abort_flag, p.err, ERR_FR_ACC_EMPTY_WAIT)
                        || !mbar_wait<true>(&full_bar[s], ph, abort_flag, p.err, ERR_FR_FULL_WAIT)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t sa = smem_u32(smem + s * kFrStageBytes);
                    const uint64_t da = operand_desc(sa);
                    const uint64_t db = operand_desc(sa + kTileBytes); // 256 rows: two tiles back to back
#pragma unroll
                    for (uint32_t j = 0; j < 4; ++j)
                        tc_mma_f8(tmem_base + b * kFrN, da + 2 * j, db + 2 * j, kIdesc, j > 0 ? 1u : 0u);
                    tc_commit(&empty_bar[s]);
                    tc_commit(&acc_full[b]);
                    if (++s == kStages) {
                        s = 0;
                        ph ^= 1;
                    }
                    b ^= 1;
                    bph ^= b == 0;
                }
            }
        }
    } else {
        // ------------------------------------------------- promotion, epilogue --
        const uint32_t quad = warp & 3, part = warp >> 2;
        const uint32_t r = quad * 32 + lane; // token row of the tile = TMEM lane
        // columns of this warp: gated 32 gate columns and the 32 up columns of the same features; plain 64 columns
        const uint32_t col0 = (quad * 32) << 16 | part * (GATED ? 32 : 64);
        constexpr uint32_t kSecond = GATED ? 128 : 32; // distance of the second 32 columns
        uint32_t b = 0, bph = 0;
        bool ok = true;
        for (uint32_t u = blockIdx.x; u < total; u += gridDim.x, next_note()) {
            ok = __all_sync(0xffffffffu, mbar_wait(&note_full[nt], nph, abort_flag, p.err, ERR_FR_NOTE_FULL_WAIT));
            const FrNote& note = s_note[nt];
            const uint32_t nb = u % p.units_per_tile;
            const uint32_t row0 = static_cast<uint32_t>(note.row0);
            const int nrows = note.nrows;
            const bool live = static_cast<int>(quad * 32) < nrows; // whole warps without a valid row only count along
            const float* xs = s_xs + nt * p.k_blocks * 128 + r;
            const float* ws = note.ws[GATED ? 0 : part / 2];
            uint64_t acc[2][16]; // two neighbouring columns each
#pragma unroll
            for (int i = 0; i < 16; ++i)
                acc[0][i] = acc[1][i] = 0;
            for (uint32_t kb = 0; kb < p.k_blocks && ok; ++kb) {
                const uint32_t x = __float_as_uint(xs[kb * 128]);
                const uint32_t f0 = __float_as_uint(ws[kb] * __uint_as_float(x));
                const uint32_t f1 = GATED ? __float_as_uint(note.ws[1][kb] * __uint_as_float(x)) : f0;
                ok = __all_sync(0xffffffffu, mbar_wait(&acc_full[b], bph, abort_flag, p.err, ERR_FR_ACC_FULL_WAIT));
                if (!ok)
                    break;
                tc_fence_after();
                if (live) {
                    const uint32_t src = tmem_base + b * kFrN + col0;
#pragma unroll
                    for (uint32_t c = 0; c < 4; ++c) {
                        uint32_t v[16];
                        tc_ld16(src + (c >> 1) * kSecond + (c & 1) * 16, v);
                        tc_ld_wait();
                        if (c == 3) { // the buffer has been read: the next k block may be multiplied into it
                            tc_fence_before();
                            __syncwarp();
                            if (lane == 0)
                                mbar_arrive(&acc_empty[b]);
                        }
                        const uint64_t f = (c >> 1) ? pack2(f1, f1) : pack2(f0, f0);
#pragma unroll
                        for (int i = 0; i < 8; ++i)
                            acc[c >> 1][(c & 1) * 8 + i]
                                = fma2(pack2(v[2 * i], v[2 * i + 1]), f, acc[c >> 1][(c & 1) * 8 + i]);
                    }
                } else if (lane == 0) {
                    mbar_arrive(&acc_empty[b]);
                }
                b ^= 1;
                bph ^= b == 0;
            }
            __syncwarp();
            if (lane == 0)
                mbar_arrive(&note_empty[nt]);
            if constexpr (GATED) {
                // SwiGLU, then one e4m3 scale per token and 128 features: the four quarters of a row are in the four
                // warps of a lane quadrant, which exchange their maxima
                float act[32];
                float amax = 0.0f;
#pragma unroll
                for (int i = 0; i < 32; ++i) {
                    const float g = part2(acc[0][i / 2], i % 2);
                    act[i] = __fdividef(g, 1.0f + __expf(-g)) * part2(acc[1][i / 2], i % 2);
                    amax = fmaxf(amax, fabsf(act[i]));
                }
                s_amax[part * 128 + r] = amax;
                ok = group_all(1 + quad, 128, ok); // the four warps stop together
                if (!ok)
                    break;
#pragma unroll
                for (uint32_t q = 0; q < 4; ++q)
                    amax = fmaxf(amax, s_amax[q * 128 + r]);
                asm volatile("bar.sync %0, 128;" ::"r"(1 + quad) : "memory"); // all have read: the next unit may write
                if (static_cast<int>(r) < nrows) {
                    const float sc = fmaxf(__fdiv_rn(amax, 448.0f), 1.0e-30f);
                    const float inv = __fdiv_rn(1.0f, sc);
                    uint8_t* out = static_cast<uint8_t*>(p.out) + static_cast<size_t>(row0 + r) * p.n + nb * 128 + part * 32;
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        uint32_t w[4];
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            w[j] = 0;
#pragma unroll
                            for (int q = 0; q < 4; ++q)
                                w[j] |= static_cast<uint32_t>(f32_to_e4m3_sat(__fmul_rn(act[16 * i + 4 * j + q], inv)))
                                    << (8 * q);
                        }
                        reinterpret_cast<uint4*>(out)[i] = make_uint4(w[0], w[1], w[2], w[3]);
                    }
                    if (part == 0)
                        p.out_scale[static_cast<size_t>(row0 + r) * p.num_fb + nb] = sc;
                }
            } else {
                // bf16 rows through shared memory and TMA stores (a 64-column box for the four warps of a part). Every
                // row of the tile is written: rows past the segment end are padding rows of the same expert.
                ok = group_all(1 + part, 128, ok);
                if (!ok)
                    break;
                const bool issuer = quad == 0 && lane == 0;
                if (issuer) // the part's previous box has left the staging
                    asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                asm volatile("bar.sync %0, 128;" ::"r"(1 + part) : "memory");
                uint8_t* row_smem = staging + part * kTileBytes + r * 128;
#pragma unroll
                for (uint32_t q = 0; q < 8; ++q) {
                    uint32_t w[4];
#pragma unroll
                    for (uint32_t i = 0; i < 4; ++i) {
                        const uint64_t v = acc[q / 4][(q % 4) * 4 + i];
                        w[i] = pack_bf16x2(part2(v, 0), part2(v, 1));
                    }
                    *reinterpret_cast<uint4*>(row_smem + ((q ^ (r & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                asm volatile("bar.sync %0, 128;" ::"r"(1 + part) : "memory");
                if (issuer) {
                    const uint32_t n0 = nb * kFrN + part * 64;
                    if (n0 < p.n)
                        asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(
                                         reinterpret_cast<uint64_t>(&map_o)),
                                     "r"(smem_u32(staging + part * kTileBytes)), "r"(static_cast<int>(n0)),
                                     "r"(static_cast<int>(row0))
                                     : "memory");
                    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                }
            }
        }
        if (!GATED && quad == 0 && lane == 0)
            asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); // stores done before smem goes away
    }

    // ---- teardown ----
    tc_fence_before();
    __syncthreads();
    if (warp == kFrAdders + 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kFrTmemCols)
                     : "memory");
    }
}

template <bool GATED>
cudaError_t launch_rows_instance(const CUtensorMap& mx, const CUtensorMap& mw, const CUtensorMap& mo,
                                 const Fp8RowsParams& fp, uint32_t grid, cudaStream_t stream)
{
    auto kernel = gemm_fp8_rows_kernel<GATED>;
    constexpr size_t smem = 1024 + FrSmem<GATED>::kBytes;
    static_assert(smem <= 227 * 1024);
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
    return launch_chained(kernel, dim3(grid), kFrThreads, smem, stream, mx, mw, mo, fp);
}

} // namespace

cudaError_t launch_fp8_rows_gemm(const Fp8Gemm& g, cudaStream_t stream, const char** why)
{
    Fp8RowsParams fp {};
    fp.n = g.n;
    fp.k_blocks = g.k / 128;
    fp.b_rows = g.gated ? 2 * g.n : g.n;
    fp.num_fb = g.n / 128;
    fp.units_per_tile = g.gated ? g.n / 128 : (g.n + kFrN - 1) / kFrN;
    fp.x_scale = g.x_scale;
    fp.w_scale = g.w_scale;
    fp.tile_expert = g.tile_expert;
    fp.tile_row0 = g.tile_row0;
    fp.tile_nrows = g.tile_nrows;
    fp.total_tiles = g.total_tiles;
    fp.row_tokens = g.row_tokens;
    fp.indptr = g.indptr;
    fp.pad_indptr = g.pad_indptr;
    fp.out = g.out;
    fp.out_scale = g.out_scale;
    fp.err = device_error_word();
    if (!g.tables_ready) {
        if (why != nullptr)
            *why = "the FP8 GEMM of 128-row tiles reads its tables before its predecessor ends";
        return cudaErrorNotSupported;
    }
    CUtensorMap mx, mw, mo;
    bool ok = make_operand_map(&mx, true, g.row_tokens != nullptr ? g.gathered : g.x, g.k, g.out_rows, g.k, kFrBox)
        && make_operand_map(&mw, true, g.w, g.k, static_cast<uint64_t>(g.groups) * fp.b_rows, g.k, 128);
    mo = mx;
    if (ok && !g.gated)
        ok = make_operand_map(&mo, false, g.out, g.n, g.out_rows, static_cast<uint64_t>(g.n) * 2, 128);
    if (!ok) {
        if (why != nullptr)
            *why = "cuTensorMapEncodeTiled failed";
        return cudaErrorInvalidValue;
    }
    const uint32_t grid = static_cast<uint32_t>(
        std::min<uint64_t>(static_cast<uint64_t>(g.max_tiles) * fp.units_per_tile, device_sm_count()));
    return g.gated ? launch_rows_instance<true>(mx, mw, mo, fp, grid, stream)
                   : launch_rows_instance<false>(mx, mw, mo, fp, grid, stream);
}

} // namespace qs3
