// Route permutation (histogram, scan, stable placement), token gather and the
// weighted combine. Replaces upstream count_routes / prefix_sum / fill_route_rows /
// scatter_hidden / finalize (qsfi_moe.cu:327-409,465-492).
#include "common.cuh"
#include "route_sort.cuh"
#include "topk.cuh"
#include "fp8.cuh"
#include "nvfp4.cuh"

#include <algorithm>
#include <cstdlib>

#include <mutex>

namespace qs3 {

namespace {

constexpr int kSortWarps = 8;              // warps per block of the counting sort
constexpr int kSortRounds = 4;              // 32-route rounds per warp
constexpr int kSortChunk = kSortWarps * kSortRounds * 32; // routes per block (1024)

// Per-warp histogram of the block's routes into s_hist[warp][expert] (u16: a warp
// sees at most kSortRounds * 32 routes). Each warp owns a contiguous run of routes,
// which is what makes the later placement stable.
__device__ __forceinline__ void
warp_histogram(const int32_t* ids, uint32_t routes, uint32_t local_offset, uint32_t experts,
               uint16_t* s_hist, uint32_t chunk)
{
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (uint32_t i = threadIdx.x; i < kSortWarps * experts; i += blockDim.x)
        s_hist[i] = 0;
    __syncthreads();
    uint16_t* mine = s_hist + static_cast<size_t>(warp) * experts;
    const uint32_t base = chunk * kSortChunk + warp * (kSortRounds * 32);
#pragma unroll
    for (int r = 0; r < kSortRounds; ++r) {
        const int e = local_expert(ids, base + r * 32 + lane, routes, local_offset, experts);
        const uint32_t peers = __match_any_sync(0xffffffffu, e);
        if (e >= 0 && lane == static_cast<uint32_t>(__ffs(peers) - 1))
            mine[e] += static_cast<uint16_t>(__popc(peers));
        __syncwarp();
    }
    __syncthreads();
}

__device__ __forceinline__ void route_hist_body(const int32_t* __restrict__ ids, uint32_t routes,
                                                uint32_t local_offset, uint32_t experts,
                                                int32_t* __restrict__ block_hist, uint16_t* s_hist, uint32_t chunk)
{
    warp_histogram(ids, routes, local_offset, experts, s_hist, chunk);
    for (uint32_t e = threadIdx.x; e < experts; e += blockDim.x) {
        int total = 0;
#pragma unroll
        for (int w = 0; w < kSortWarps; ++w)
            total += s_hist[static_cast<size_t>(w) * experts + e];
        block_hist[static_cast<size_t>(chunk) * experts + e] = total;
    }
}

__global__ void __launch_bounds__(kSortWarps * 32)
route_hist_kernel(const int32_t* __restrict__ ids, uint32_t routes, uint32_t local_offset,
                  uint32_t experts, int32_t* __restrict__ block_hist)
{
    extern __shared__ uint16_t s_hist[];
    chain_begin();
    route_hist_body(ids, routes, local_offset, experts, block_hist, s_hist, blockIdx.x);
}

// Where the tables may have one of two tile heights: the time of a tile of either kind. NVFP4 layer, 512 experts top-10,
// 64- against 128-row tiles: even routing, 1399 tokens (512 tiles of either kind) 0.25 against 0.345 ms, 2200 tokens 0.284
// against 0.361; skewed routing, 2048 tokens 0.247 against 0.216.
constexpr int kAltTileCost = 5, kTileCost = 7;

// Single block: per expert, exclusive scan of the block histograms (column scan),
// then exclusive scans over experts of the counts, of the counts padded to the
// tile height, and of the tile counts; finally the tile table.
__device__ __forceinline__ void route_scan_body(int32_t* __restrict__ block_hist, uint32_t num_blocks,
                                                uint32_t experts, const RouteTables& rt)
{
    constexpr int kScans = 5; // counts, padded counts, tiles, full pair tiles, single tiles
    __shared__ int s_warp[kScans][32];
    __shared__ int s_carry[kScans];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    bool use_alt = false;
    if (threadIdx.x < kScans)
        s_carry[threadIdx.x] = 0;
    __syncthreads();
    for (uint32_t e0 = 0; e0 < experts; e0 += blockDim.x) {
        const uint32_t e = e0 + threadIdx.x;
        int count = 0;
        if (e < experts) {
            // loads are issued in independent batches so that their latencies overlap
            constexpr uint32_t kBatch = 16;
            for (uint32_t b0 = 0; b0 < num_blocks; b0 += kBatch) {
                int v[kBatch];
#pragma unroll
                for (uint32_t j = 0; j < kBatch; ++j)
                    v[j] = b0 + j < num_blocks
                        ? block_hist[static_cast<size_t>(b0 + j) * experts + e]
                        : 0;
#pragma unroll
                for (uint32_t j = 0; j < kBatch; ++j) {
                    if (b0 + j < num_blocks)
                        block_hist[static_cast<size_t>(b0 + j) * experts + e] = count;
                    count += v[j];
                }
            }
            rt.counts[e] = count;
        }
        int tile_rows = static_cast<int>(rt.tile_rows);
        if (rt.alt_total_tiles != nullptr) { // (one pass over the experts: they fit the block)
            const int tr = static_cast<int>(rt.tile_rows), ar = static_cast<int>(rt.alt_tile_rows);
            const int t = __reduce_add_sync(0xffffffffu, (count + tr - 1) / tr), a = __reduce_add_sync(0xffffffffu, (count + ar - 1) / ar);
            if (lane == 0) {
                s_warp[0][warp] = t;
                s_warp[1][warp] = a;
            }
            __syncthreads();
            int total = 0, alt = 0;
            for (uint32_t w = 0; w < blockDim.x / 32; ++w) {
                total += s_warp[0][w];
                alt += s_warp[1][w];
            }
            __syncthreads(); // the slots are used again below
            use_alt = alt * kAltTileCost < total * kTileCost;
            if (use_alt)
                tile_rows = ar;
        }
        const int tiles = (count + tile_rows - 1) / tile_rows;
        const bool pairing = rt.pair_expert != nullptr && !use_alt;
        int v[kScans] = { count, tiles * tile_rows, tiles, pairing ? tiles >> 1 : 0, pairing ? tiles & 1 : 0 };
        int incl[kScans];
#pragma unroll
        for (int j = 0; j < kScans; ++j) {
            int x = v[j];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= static_cast<uint32_t>(o))
                    x += y;
            }
            incl[j] = x;
            if (lane == 31)
                s_warp[j][warp] = x;
            if (threadIdx.x < 32 && threadIdx.x >= blockDim.x / 32)
                s_warp[j][threadIdx.x] = 0; // slots of warps this block does not have
        }
        __syncthreads();
        if (warp == 0) {
#pragma unroll
            for (int j = 0; j < kScans; ++j) {
                int x = s_warp[j][lane];
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int y = __shfl_up_sync(0xffffffffu, x, o);
                    if (lane >= static_cast<uint32_t>(o))
                        x += y;
                }
                s_warp[j][lane] = x; // inclusive over warps
            }
        }
        __syncthreads();
        int excl[kScans];
#pragma unroll
        for (int j = 0; j < kScans; ++j)
            excl[j] = s_carry[j] + (warp > 0 ? s_warp[j][warp - 1] : 0) + incl[j] - v[j];
        if (e < experts) {
            rt.indptr[e] = excl[0];
            rt.pad_indptr[e] = excl[1];
            for (int m = 0; m < tiles; ++m) {
                rt.tile_expert[excl[2] + m] = static_cast<int32_t>(e);
                rt.tile_row0[excl[2] + m] = excl[1] + m * tile_rows;
                rt.tile_nrows[excl[2] + m] = min(tile_rows, count - m * tile_rows);
            }
            if (pairing) {
                for (int m = 0; m < (tiles >> 1); ++m) {
                    rt.pair_expert[excl[3] + m] = static_cast<int32_t>(e);
                    rt.pair_row0[excl[3] + m] = excl[1] + m * 2 * tile_rows;
                    rt.pair_nrows[excl[3] + m] = min(2 * tile_rows, count - m * 2 * tile_rows);
                }
                if (tiles & 1) {
                    const int at = static_cast<int>(rt.max_tiles) - 1 - excl[4];
                    rt.pair_expert[at] = static_cast<int32_t>(e);
                    rt.pair_row0[at] = excl[1] + (tiles - 1) * tile_rows;
                    rt.pair_nrows[at] = count - (tiles - 1) * tile_rows;
                }
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) {
#pragma unroll
            for (int j = 0; j < kScans; ++j)
                s_carry[j] += s_warp[j][31];
        }
        __syncthreads();
    }
    append_shared_tiles(rt, experts, static_cast<uint32_t>(s_carry[2]));
    if (threadIdx.x == 0) {
        rt.indptr[experts] = s_carry[0];
        rt.pad_indptr[experts] = s_carry[1];
        *rt.total_tiles = use_alt ? 0 : s_carry[2] + static_cast<int>((rt.shared_rows + rt.tile_rows - 1) / rt.tile_rows);
        if (rt.alt_total_tiles != nullptr)
            *rt.alt_total_tiles = use_alt ? s_carry[2] : 0;
        if (rt.pair_counts != nullptr) {
            rt.pair_counts[0] = s_carry[3];
            rt.pair_counts[1] = s_carry[4];
        }
    }
}

__global__ void __launch_bounds__(1024)
route_scan_kernel(int32_t* __restrict__ block_hist, uint32_t num_blocks, uint32_t experts,
                  RouteTables rt)
{
    chain_begin();
    route_scan_body(block_hist, num_blocks, experts, rt);
}

// Placement: row of a route = segment start + routes of the same expert in earlier
// blocks + in earlier warps of this block + earlier in this warp. Stable in route
// index, so the permutation is reproducible (upstream's is atomics-ordered).
// `s_hist` holds the per-warp histograms of this block (warp_histogram).
__device__ __forceinline__ void route_place_body(const int32_t* __restrict__ ids,
                                                 const float* __restrict__ weights, uint32_t routes,
                                                 uint32_t top_k, uint32_t local_offset, uint32_t experts,
                                                 const RouteTables& rt, uint16_t* s_hist, uint32_t chunk)
{
    // exclusive prefix over the warps of the block, per expert
    for (uint32_t e = threadIdx.x; e < experts; e += blockDim.x) {
        int run = 0;
#pragma unroll
        for (int w = 0; w < kSortWarps; ++w) {
            const size_t i = static_cast<size_t>(w) * experts + e;
            const int v = s_hist[i];
            s_hist[i] = static_cast<uint16_t>(run);
            run += v;
        }
    }
    __syncthreads();
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint16_t* mine = s_hist + static_cast<size_t>(warp) * experts;
    const uint32_t base = chunk * kSortChunk + warp * (kSortRounds * 32);
    const int32_t* block_off = rt.block_hist + static_cast<size_t>(chunk) * experts;
#pragma unroll
    for (int r = 0; r < kSortRounds; ++r) {
        const uint32_t route = base + r * 32 + lane;
        const int e = local_expert(ids, route, routes, local_offset, experts);
        const uint32_t peers = __match_any_sync(0xffffffffu, e);
        int in_block = 0;
        if (e >= 0)
            in_block = mine[e] + __popc(peers & ((1u << lane) - 1u));
        __syncwarp();
        if (e >= 0 && lane == static_cast<uint32_t>(__ffs(peers) - 1))
            mine[e] += static_cast<uint16_t>(__popc(peers));
        __syncwarp();
        if (route < routes) {
            if (e >= 0) {
                const int off = block_off[e] + in_block;
                const int row = rt.indptr[e] + off;
                rt.route_rows[route] = row;
                rt.route_prows[route] = rt.pad_indptr[e] + off;
                rt.row_tokens[row] = static_cast<int32_t>(route / top_k);
                rt.row_scales[row] = weights[route];
            } else {
                rt.route_rows[route] = -1;
                rt.route_prows[route] = -1;
            }
        }
    }
}

__global__ void __launch_bounds__(kSortWarps * 32)
route_place_kernel(const int32_t* __restrict__ ids, const float* __restrict__ weights,
                   uint32_t routes, uint32_t top_k, uint32_t local_offset, uint32_t experts,
                   RouteTables rt)
{
    extern __shared__ uint16_t s_hist[];
    chain_begin();
    warp_histogram(ids, routes, local_offset, experts, s_hist, blockIdx.x);
    route_place_body(ids, weights, routes, top_k, local_offset, experts, rt, s_hist, blockIdx.x);
}

// ---- counting sort of a large batch in two launches -----------------------------------------------------------------
// The histograms of the chunks, then every block adds up all of them by itself, scans the experts and places its chunk: the
// single block that did the scans alone made the sort of 10210 routes over 512 experts 22.7 us, now 15.6 (81920: 23.4 / 15.2). The
// blocks' sums cost blocks * experts * 2 bytes of L2 reads each. Tables of the experts are written by the blocks in turn.
constexpr uint32_t kSpThreads = 512, kSpWarps = kSpThreads / 32;
constexpr uint32_t kSpRounds = kSortChunk / kSpThreads; // 32-route rounds per warp
constexpr uint32_t kSpMaxExperts = 2 * kSpThreads;      // two per thread
constexpr uint32_t kSpMaxChunks = 256;                  // the blocks' reads grow with the square of their number

__host__ __device__ constexpr uint32_t sp_pitch(uint32_t experts) { return (experts + 7) / 8 * 8; }

__global__ void __launch_bounds__(kSpThreads)
route_chunk_hist_kernel(const int32_t* __restrict__ ids, uint32_t routes, uint32_t local_offset, uint32_t experts,
                        uint16_t* __restrict__ hist)
{
    extern __shared__ __align__(16) uint8_t s_dyn[];
    uint32_t* s_count = reinterpret_cast<uint32_t*>(s_dyn); // [experts]
    for (uint32_t e = threadIdx.x; e < experts; e += kSpThreads)
        s_count[e] = 0;
    chain_begin();
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < static_cast<uint32_t>(kSortChunk); i += kSpThreads) {
        const int e = local_expert(ids, blockIdx.x * kSortChunk + i, routes, local_offset, experts);
        const uint32_t peers = __match_any_sync(0xffffffffu, e);
        if (e >= 0 && threadIdx.x % 32 == static_cast<uint32_t>(__ffs(static_cast<int>(peers)) - 1))
            atomicAdd(s_count + e, __popc(peers));
    }
    __syncthreads();
    uint16_t* row = hist + static_cast<size_t>(blockIdx.x) * sp_pitch(experts);
    for (uint32_t e = threadIdx.x; e < sp_pitch(experts); e += kSpThreads)
        row[e] = e < experts ? static_cast<uint16_t>(s_count[e]) : 0;
}

__global__ void __launch_bounds__(kSpThreads)
route_scan_place_kernel(const int32_t* __restrict__ ids, const float* __restrict__ weights, uint32_t routes, uint32_t top_k,
                        uint32_t local_offset, uint32_t experts, const uint16_t* __restrict__ hist, RouteTables rt)
{
    extern __shared__ __align__(16) uint8_t s_dyn[];
    const uint32_t pitch = sp_pitch(experts);
    uint32_t* s_total = reinterpret_cast<uint32_t*>(s_dyn); // [pitch] routes of the expert; then its first dense row here
    uint32_t* s_before = s_total + pitch;                   // [pitch] those of earlier chunks
    uint32_t* s_pad = s_before + pitch;                     // [pitch] first padded row here
    uint16_t* s_hist = reinterpret_cast<uint16_t*>(s_pad + pitch); // [kSpWarps][experts]
    __shared__ uint32_t s_warp[4][kSpWarps];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (uint32_t e = threadIdx.x; e < pitch; e += kSpThreads)
        s_total[e] = s_before[e] = 0;
    for (uint32_t i = threadIdx.x; i < kSpWarps * experts; i += kSpThreads)
        s_hist[i] = 0;
    chain_begin();
    __syncthreads();

    // this chunk's routes, each warp a run of them, and the other chunks' histograms, eight experts at a time
    uint16_t* mine = s_hist + static_cast<size_t>(warp) * experts;
    const uint32_t base = blockIdx.x * kSortChunk + warp * (kSpRounds * 32);
    int expert[kSpRounds];
    uint32_t peers[kSpRounds];
#pragma unroll
    for (uint32_t r = 0; r < kSpRounds; ++r)
        expert[r] = local_expert(ids, base + r * 32 + lane, routes, local_offset, experts);
    const uint32_t vecs = pitch / 8, slices = max(1u, kSpThreads / vecs);
    if (threadIdx.x < vecs * slices) {
        const uint32_t v = threadIdx.x % vecs;
        uint32_t total[8] = {}, before[8] = {};
        const uint4* src = reinterpret_cast<const uint4*>(hist) + v;
#pragma unroll 4
        for (uint32_t b = threadIdx.x / vecs; b < gridDim.x; b += slices) {
            const uint4 h = src[static_cast<size_t>(b) * vecs];
            const uint32_t w[4] = { h.x, h.y, h.z, h.w };
            const bool earlier = b < blockIdx.x;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const uint32_t n = w[i / 2] >> (16 * (i % 2)) & 0xffffu;
                total[i] += n;
                before[i] += earlier ? n : 0u;
            }
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            if (total[i] != 0)
                atomicAdd(s_total + v * 8 + i, total[i]);
            if (before[i] != 0)
                atomicAdd(s_before + v * 8 + i, before[i]);
        }
    }
#pragma unroll
    for (uint32_t r = 0; r < kSpRounds; ++r) {
        peers[r] = __match_any_sync(0xffffffffu, expert[r]);
        if (expert[r] >= 0 && lane == static_cast<uint32_t>(__ffs(static_cast<int>(peers[r])) - 1))
            mine[expert[r]] += static_cast<uint16_t>(__popc(peers[r]));
        __syncwarp();
    }
    __syncthreads();

    // scans over the experts, a thread owns two neighbouring ones
    uint32_t count[2];
#pragma unroll
    for (uint32_t j = 0; j < 2; ++j)
        count[j] = 2 * threadIdx.x + j < experts ? s_total[2 * threadIdx.x + j] : 0u;
    uint32_t tile_rows = rt.tile_rows;
    bool use_alt = false;
    const auto tiles_of = [](uint32_t n, uint32_t rows) { return (n + rows - 1) / rows; };
    if (rt.alt_total_tiles != nullptr) {
        const uint32_t t = __reduce_add_sync(0xffffffffu, tiles_of(count[0], tile_rows) + tiles_of(count[1], tile_rows));
        const uint32_t a = __reduce_add_sync(0xffffffffu, tiles_of(count[0], rt.alt_tile_rows) + tiles_of(count[1], rt.alt_tile_rows));
        if (lane == 0) {
            s_warp[0][warp] = t;
            s_warp[1][warp] = a;
        }
        __syncthreads();
        uint32_t total = 0, alt = 0;
#pragma unroll
        for (uint32_t w = 0; w < kSpWarps; ++w) {
            total += s_warp[0][w];
            alt += s_warp[1][w];
        }
        __syncthreads(); // the slots are used again below
        use_alt = alt * kAltTileCost < total * kTileCost;
        if (use_alt)
            tile_rows = rt.alt_tile_rows;
    }
    const bool pairing = rt.pair_expert != nullptr && !use_alt;
    uint32_t tiles[2] = { tiles_of(count[0], tile_rows), tiles_of(count[1], tile_rows) };
    // routes, tiles, full pairs, single tiles
    const uint32_t v[4] = { count[0] + count[1], tiles[0] + tiles[1], pairing ? tiles[0] / 2 + tiles[1] / 2 : 0u,
                            pairing ? tiles[0] % 2 + tiles[1] % 2 : 0u };
    uint32_t ex[4], all[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        uint32_t x = v[q];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= static_cast<uint32_t>(o))
                x += y;
        }
        if (lane == 31)
            s_warp[q][warp] = x;
        ex[q] = x - v[q];
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        all[q] = 0;
#pragma unroll
        for (uint32_t w = 0; w < kSpWarps; ++w) {
            if (w == warp)
                ex[q] += all[q];
            all[q] += s_warp[q][w];
        }
    }
#pragma unroll
    for (uint32_t j = 0; j < 2; ++j) {
        const uint32_t e = 2 * threadIdx.x + j;
        if (e >= experts)
            break;
        const uint32_t n = count[j], pad = ex[1] * tile_rows;
        s_total[e] = ex[0] + s_before[e];
        s_pad[e] = pad + s_before[e];
        if (e % gridDim.x == blockIdx.x) { // this block's share of the tables
            rt.counts[e] = static_cast<int32_t>(n);
            rt.indptr[e] = static_cast<int32_t>(ex[0]);
            rt.pad_indptr[e] = static_cast<int32_t>(pad);
            for (uint32_t m = 0; m < tiles[j]; ++m) {
                rt.tile_expert[ex[1] + m] = static_cast<int32_t>(e);
                rt.tile_row0[ex[1] + m] = static_cast<int32_t>(pad + m * tile_rows);
                rt.tile_nrows[ex[1] + m] = static_cast<int32_t>(min(tile_rows, n - m * tile_rows));
            }
            if (pairing) {
                for (uint32_t m = 0; m < tiles[j] / 2; ++m) {
                    rt.pair_expert[ex[2] + m] = static_cast<int32_t>(e);
                    rt.pair_row0[ex[2] + m] = static_cast<int32_t>(pad + m * 2 * tile_rows);
                    rt.pair_nrows[ex[2] + m] = static_cast<int32_t>(min(2 * tile_rows, n - m * 2 * tile_rows));
                }
                if (tiles[j] % 2 != 0) {
                    const uint32_t at = rt.max_tiles - 1 - ex[3];
                    rt.pair_expert[at] = static_cast<int32_t>(e);
                    rt.pair_row0[at] = static_cast<int32_t>(pad + (tiles[j] - 1) * tile_rows);
                    rt.pair_nrows[at] = static_cast<int32_t>(n - (tiles[j] - 1) * tile_rows);
                }
            }
        }
        ex[0] += n;
        ex[1] += tiles[j];
        ex[2] += tiles[j] / 2;
        ex[3] += tiles[j] % 2;
    }
    if (blockIdx.x == 0) {
        append_shared_tiles(rt, experts, all[1]);
        if (threadIdx.x == 0) {
            rt.indptr[experts] = static_cast<int32_t>(all[0]);
            rt.pad_indptr[experts] = static_cast<int32_t>(all[1] * tile_rows);
            *rt.total_tiles = use_alt ? 0 : static_cast<int32_t>(all[1] + (rt.shared_rows + rt.tile_rows - 1) / rt.tile_rows);
            if (rt.alt_total_tiles != nullptr)
                *rt.alt_total_tiles = use_alt ? static_cast<int32_t>(all[1]) : 0;
            if (rt.pair_counts != nullptr) {
                rt.pair_counts[0] = static_cast<int32_t>(all[2]);
                rt.pair_counts[1] = static_cast<int32_t>(all[3]);
            }
        }
    }

    // placement: earlier chunks, earlier warps of this one, earlier routes of the warp
    for (uint32_t e = threadIdx.x; e < experts; e += kSpThreads) {
        uint32_t run = 0;
#pragma unroll
        for (uint32_t w = 0; w < kSpWarps; ++w) {
            const uint32_t n = s_hist[w * experts + e];
            s_hist[w * experts + e] = static_cast<uint16_t>(run);
            run += n;
        }
    }
    __syncthreads();
#pragma unroll
    for (uint32_t r = 0; r < kSpRounds; ++r) {
        const uint32_t route = base + r * 32 + lane;
        const int e = expert[r];
        uint32_t off = 0;
        if (e >= 0)
            off = mine[e] + __popc(peers[r] & ((1u << lane) - 1u));
        __syncwarp();
        if (e >= 0 && lane == static_cast<uint32_t>(__ffs(static_cast<int>(peers[r])) - 1))
            mine[e] += static_cast<uint16_t>(__popc(peers[r]));
        __syncwarp();
        if (route < routes) {
            if (e >= 0) {
                const uint32_t row = s_total[e] + off;
                rt.route_rows[route] = static_cast<int32_t>(row);
                rt.route_prows[route] = static_cast<int32_t>(s_pad[e] + off);
                rt.row_tokens[row] = static_cast<int32_t>(route / top_k);
                rt.row_scales[row] = weights[route];
            } else {
                rt.route_rows[route] = -1;
                rt.route_prows[route] = -1;
            }
        }
    }
}

__device__ __forceinline__ void quantize_beside(const TokenQuant& q, uint64_t warp)
{
    if (q.fp8_scale != nullptr)
        fp8_quantize_groups(q.x, q.rows, q.k, q.packed, q.fp8_scale, warp);
    else
        quantize_row_chunk(q.x, q.rows, q.k, q.global_scale, q.packed, q.scale_tiled, warp);
}

// All three steps in one block for a decode batch's routes: 1280 routes over 512 experts 0.0129 ->
// 0.0078 ms, 10 routes 0.0058 -> 0.0042 against 256 threads with global histograms.
__global__ void __launch_bounds__(kBlockSortThreads)
route_sort_block_kernel(const int32_t* __restrict__ ids, const float* __restrict__ weights, uint32_t routes,
                        uint32_t top_k, uint32_t local_offset, uint32_t experts, RouteTables rt, TokenQuant quant)
{
    chain_begin();
    if (blockIdx.x > 0) { // the other blocks quantise the tokens meanwhile
        quantize_beside(quant, static_cast<uint64_t>(blockIdx.x - 1) * kBlockSortWarps + (threadIdx.x >> 5));
        return;
    }
    extern __shared__ __align__(16) uint8_t s_dyn[];
    const BlockSortSmem s = block_sort_carve(s_dyn, experts);
    for (uint32_t i = threadIdx.x; i < routes; i += kBlockSortThreads)
        s.ids[i] = static_cast<int16_t>(local_expert(ids, i, routes, local_offset, experts));
    block_sort(s, weights, routes, top_k, experts, rt); // (starts with a barrier)
}

// The same after the top-k of up to kBlockSortWarps tokens, a warp per token, in the same launch (as launches of their own:
// layer of 16 tokens over 8 experts 0.0278 ms instead of 0.0240, 1 token over 512 experts 0.0369 instead of 0.0360).
template <int ITEMS>
__global__ void __launch_bounds__(kBlockSortThreads)
router_sort_block_kernel(RouterParams r, uint32_t top_k, uint32_t local_offset, uint32_t experts, RouteTables rt, TokenQuant quant)
{
    chain_begin();
    if (blockIdx.x > 0) {
        quantize_beside(quant, static_cast<uint64_t>(blockIdx.x - 1) * kBlockSortWarps + (threadIdx.x >> 5));
        return;
    }
    extern __shared__ __align__(16) uint8_t s_dyn[];
    __shared__ uint32_t s_cand[kBlockSortWarps][64];
    const BlockSortSmem s = block_sort_carve(s_dyn, experts);
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp < r.num_tokens) {
        int id;
        float weight;
        topk_row<float, ITEMS>(r.logits + static_cast<size_t>(warp) * r.num_experts, r.bias, r.num_experts, top_k,
                               r.sigmoid_score, r.renormalize, r.scaling, s_cand[warp], &id, &weight);
        if (lane < top_k) {
            const uint32_t route = warp * top_k + lane;
            const int local = id - static_cast<int>(local_offset);
            r.ids[route] = id;
            r.weights[route] = weight;
            s.ids[route] = static_cast<int16_t>(local < 0 || local >= static_cast<int>(experts) ? -1 : local);
        }
    }
    block_sort(s, r.weights, r.num_tokens * top_k, top_k, experts, rt); // (starts with a barrier)
}

// dst[padded row] = src[token] for the tiles of experts with more than `min_rows` rows; a block per 32 rows of a tile (8 where
// those blocks fit the device at once), a warp per row, four 16-byte vectors per lane in flight. Bound by HBM and L2: rows *
// row bytes, read and written; where few experts are heavy, by the blocks that find nothing to do (8 rows per block: 2048
// tokens, 512 experts 0.008 ms).

__global__ void __launch_bounds__(256)
gather_rows_kernel(const uint4* __restrict__ src, uint32_t vec_per_row, RouteTables rt, int min_rows, uint4* __restrict__ dst)
{
    chain_begin();
    const uint32_t tile = blockIdx.y, lane = threadIdx.x & 31;
    if (static_cast<int>(tile) >= *rt.total_tiles)
        return;
    const int expert = rt.tile_expert[tile], row0 = rt.tile_row0[tile], nrows = rt.tile_nrows[tile], dense0 = rt.indptr[expert];
    if (rt.indptr[expert + 1] - dense0 <= min_rows)
        return;
    const int32_t* tokens = rt.row_tokens + dense0 + row0 - rt.pad_indptr[expert];
    const uint32_t block_rows = rt.tile_rows / gridDim.x;
    const int end = min(nrows, static_cast<int>((blockIdx.x + 1) * block_rows));
    for (int j = static_cast<int>(blockIdx.x * block_rows + (threadIdx.x >> 5)); j < end; j += 8) {
        const uint4* s = src + static_cast<size_t>(tokens[j]) * vec_per_row;
        uint4* d = dst + static_cast<size_t>(row0 + j) * vec_per_row;
        for (uint32_t i0 = lane; i0 < vec_per_row; i0 += 128) {
            uint4 v[4];
#pragma unroll
            for (uint32_t q = 0; q < 4; ++q)
                if (i0 + 32 * q < vec_per_row)
                    v[q] = s[i0 + 32 * q];
#pragma unroll
            for (uint32_t q = 0; q < 4; ++q)
                if (i0 + 32 * q < vec_per_row)
                    d[i0 + 32 * q] = v[q];
        }
    }
}

// out[t, :] = bf16(sum_k w[t,k] * f32(Y2[prow(t,k), :])) (+ shared-expert term).
// TOKENS tokens per block, GROUP threads per token; a thread owns CHUNKS 8-element chunks of the row per step and
// issues the loads of up to BATCH routes for all of them together. k ascending and f32 accumulation as upstream
// finalize_kernel (qsfi_moe.cu:465-492); the shape of the block does not change a sum.
//   prefill  4 tokens x 64 threads, two chunks, four routes: bound by HBM (R * H * 2 bytes in), eight 16-byte loads in
//            flight per thread, so that tokens with one or two local routes (expert parallelism) still keep the memory
//            system busy
//   decode   one token x 256 threads, all routes of a chunk in one round: bound by latency, and 128 tokens in blocks of
//            four left 116 SMs idle and took three rounds per chunk (128 tokens with the fused norm 0.0149 -> 0.0072 ms,
//            1 token 0.0074 -> 0.0039)
constexpr uint32_t kCombineThreads = 256;

__device__ __forceinline__ void accumulate_row(float* acc, const uint4& v, float w)
{
    const uint32_t vs[4] = { v.x, v.y, v.z, v.w };
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        acc[2 * j] += w * bf16_bits_to_f32(vs[j] & 0xffffu);
        acc[2 * j + 1] += w * bf16_bits_to_f32(vs[j] >> 16);
    }
}

// acc[c] = sum over the token's valid routes, in order, of weight * the route's row at chunk i0 + c * GROUP.
template <uint32_t CHUNKS, uint32_t BATCH, uint32_t GROUP>
__device__ __forceinline__ void sum_routes(const CombineParams& p, const int* rows, const float* weights,
                                           uint32_t n_valid, uint32_t i0, uint32_t vec_per_row, float (*acc)[8])
{
    const uint4* y2 = reinterpret_cast<const uint4*>(p.expert_out);
#pragma unroll
    for (uint32_t c = 0; c < CHUNKS; ++c)
#pragma unroll
        for (int j = 0; j < 8; ++j)
            acc[c][j] = 0.0f;
    for (uint32_t k0 = 0; k0 < n_valid; k0 += BATCH) {
        uint4 v[CHUNKS][BATCH];
        float w[BATCH];
        int row[BATCH];
#pragma unroll
        for (uint32_t q = 0; q < BATCH; ++q) {
            row[q] = k0 + q < n_valid ? rows[k0 + q] : -1;
            w[q] = row[q] >= 0 ? weights[k0 + q] : 0.0f;
            const uint4* src = y2 + static_cast<size_t>(row[q] >= 0 ? row[q] : 0) * vec_per_row;
#pragma unroll
            for (uint32_t c = 0; c < CHUNKS; ++c)
                v[c][q] = (row[q] >= 0 && i0 + c * GROUP < vec_per_row) ? src[i0 + c * GROUP] : make_uint4(0, 0, 0, 0);
        }
#pragma unroll
        for (uint32_t q = 0; q < BATCH; ++q) {
            if (row[q] < 0)
                continue; // a skipped route adds nothing (not even a signed zero)
#pragma unroll
            for (uint32_t c = 0; c < CHUNKS; ++c)
                accumulate_row(acc[c], v[c][q], w[q]);
        }
    }
}

// acc += sigmoid gate * the shared expert's row at chunk i (the routed sum rounded to bf16 first for bf16 plans, as
// upstream does).
__device__ __forceinline__ void add_shared(const CombineParams& p, uint32_t token, uint32_t vec_per_row, uint32_t i,
                                           float gate, float* acc)
{
    const size_t row = (p.shared_row0 != nullptr ? static_cast<size_t>(*p.shared_row0) : 0) + token;
    const uint4 sv = reinterpret_cast<const uint4*>(p.shared_out)[row * vec_per_row + i];
    const uint32_t ss[4] = { sv.x, sv.y, sv.z, sv.w };
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        float a0 = acc[2 * j], a1 = acc[2 * j + 1];
        if (p.round_before_shared) {
            a0 = __bfloat162float(__float2bfloat16(a0));
            a1 = __bfloat162float(__float2bfloat16(a1));
        }
        acc[2 * j] = a0 + gate * bf16_bits_to_f32(ss[j] & 0xffffu);
        acc[2 * j + 1] = a1 + gate * bf16_bits_to_f32(ss[j] >> 16);
    }
}

template <uint32_t TOKENS, uint32_t CHUNKS, uint32_t BATCH>
__global__ void __launch_bounds__(kCombineThreads, TOKENS == 1 ? 2 : 4) combine_kernel(CombineParams p)
{
    constexpr uint32_t kGroup = kCombineThreads / TOKENS;
    __shared__ int s_row[TOKENS][32];
    __shared__ float s_w[TOKENS][32];
    __shared__ float s_dot[TOKENS][kGroup / 32];
    __shared__ int s_any[TOKENS];
    if (!p.early)
        chain_begin();
    const uint32_t group = threadIdx.x / kGroup, gl = threadIdx.x % kGroup;
    const uint32_t token = blockIdx.x * TOKENS + group;
    const bool live = token < p.num_tokens;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t vec_per_row = p.hidden_size / 8;

    if (gl < 32) {
        // the token's routes that have a row here, compacted in ascending k
        int row = -1;
        float wgt = 0.0f;
        if (live && gl < p.top_k) {
            row = p.route_prows[static_cast<size_t>(token) * p.top_k + gl];
            wgt = p.topk_weights[static_cast<size_t>(token) * p.top_k + gl];
        }
        const uint32_t valid = __ballot_sync(0xffffffffu, row >= 0);
        if (row >= 0) {
            const uint32_t slot = __popc(valid & ((1u << gl) - 1u));
            s_row[group][slot] = row;
            s_w[group][slot] = wgt;
        }
        if (gl == 0)
            s_any[group] = __popc(valid);
    }
    float dot = 0.0f;
    if (p.shared_out != nullptr) {
        // gate logit x . w_gate in f32 (upstream computes it as an N = 1 GEMM,
        // src/model.rs:2218-2226)
        if (live) {
            const uint4* x = reinterpret_cast<const uint4*>(p.hidden) + static_cast<size_t>(token) * vec_per_row;
            const uint4* w = reinterpret_cast<const uint4*>(p.gate_w);
            for (uint32_t i = gl; i < vec_per_row; i += kGroup) {
                const uint4 xv = x[i], wv = w[i];
                const uint32_t xs[4] = { xv.x, xv.y, xv.z, xv.w };
                const uint32_t ws[4] = { wv.x, wv.y, wv.z, wv.w };
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    dot += bf16_bits_to_f32(xs[j] & 0xffffu) * bf16_bits_to_f32(ws[j] & 0xffffu);
                    dot += bf16_bits_to_f32(xs[j] >> 16) * bf16_bits_to_f32(ws[j] >> 16);
                }
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            dot += __shfl_xor_sync(0xffffffffu, dot, o);
        if (lane == 0)
            s_dot[group][gl / 32] = dot;
    }
    if (p.early) // all of the above is older than the predecessor
        chain_begin();
    __syncthreads();
    if (!live || (p.skip_empty && !s_any[group]))
        return; // no local route: the row stays unwritten and is never read
    float gate = 0.0f;
    if (p.shared_out != nullptr) {
        dot = 0.0f;
#pragma unroll
        for (uint32_t w = 0; w < kGroup / 32; ++w) // fixed order: the same sum in every thread
            dot += s_dot[group][w];
        gate = sigmoid_fast(dot);
    }

    uint4* out = reinterpret_cast<uint4*>(p.out) + static_cast<size_t>(token) * vec_per_row;
    const uint32_t n_valid = static_cast<uint32_t>(s_any[group]);
    for (uint32_t i0 = gl; i0 < vec_per_row; i0 += CHUNKS * kGroup) {
        float acc[CHUNKS][8];
        sum_routes<CHUNKS, BATCH, kGroup>(p, s_row[group], s_w[group], n_valid, i0, vec_per_row, acc);
#pragma unroll
        for (uint32_t c = 0; c < CHUNKS; ++c) {
            const uint32_t i = i0 + c * kGroup;
            if (i >= vec_per_row)
                break;
            if (p.shared_out != nullptr)
                add_shared(p, token, vec_per_row, i, gate, acc[c]);
            uint32_t o[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const __nv_bfloat162 r = __floats2bfloat162_rn(acc[c][2 * j], acc[c][2 * j + 1]);
                o[j] = *reinterpret_cast<const uint32_t*>(&r);
            }
            out[i] = make_uint4(o[0], o[1], o[2], o[3]);
        }
    }
}

// The combine above followed by the block's post-MoE neighbours in the same pass:
//   x        = bf16(sum_k w_k * Y2[row_k] (+ shared term))        (what combine_kernel stores)
//   residual = bf16(f32(x) + f32(residual))                       (in place)
//   out      = bf16((f32(x) + f32(residual)) * rsqrt(mean(.^2) + eps) * norm_weight)
// i.e. qsfi_fused_add_rmsnorm applied to the MoE output without the round trip of [T, H]
// through HBM. A thread keeps its chunks of the row (256 in all, so rows are limited to 2048 elements) in registers
// across the row-wide reduction. One token or four per block, as above.
template <uint32_t TOKENS, uint32_t BATCH>
__global__ void __launch_bounds__(kCombineThreads, 2) combine_norm_kernel(CombineParams p)
{
    constexpr uint32_t kGroup = kCombineThreads / TOKENS;
    constexpr uint32_t kStep = TOKENS == 1 ? 1 : 2; // chunks per round of loads
    __shared__ int s_row[TOKENS][32];
    __shared__ float s_w[TOKENS][32];
    __shared__ float s_dot[TOKENS][kGroup / 32];
    __shared__ float s_sq[TOKENS][kGroup / 32];
    __shared__ int s_any[TOKENS];
    if (!p.early)
        chain_begin();
    const uint32_t group = threadIdx.x / kGroup, gl = threadIdx.x % kGroup;
    const uint32_t token = blockIdx.x * TOKENS + group;
    const bool live = token < p.num_tokens;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t vec_per_row = p.hidden_size / 8;

    if (gl < 32) {
        int row = -1;
        float wgt = 0.0f;
        if (live && gl < p.top_k) {
            row = p.route_prows[static_cast<size_t>(token) * p.top_k + gl];
            wgt = p.topk_weights[static_cast<size_t>(token) * p.top_k + gl];
        }
        const uint32_t valid = __ballot_sync(0xffffffffu, row >= 0);
        if (row >= 0) {
            const uint32_t slot = __popc(valid & ((1u << gl) - 1u));
            s_row[group][slot] = row;
            s_w[group][slot] = wgt;
        }
        if (gl == 0)
            s_any[group] = __popc(valid);
    }
    float dot = 0.0f;
    if (p.shared_out != nullptr) {
        if (live) {
            const uint4* x = reinterpret_cast<const uint4*>(p.hidden) + static_cast<size_t>(token) * vec_per_row;
            const uint4* w = reinterpret_cast<const uint4*>(p.gate_w);
            for (uint32_t i = gl; i < vec_per_row; i += kGroup) {
                const uint4 xv = x[i], wv = w[i];
                const uint32_t xs[4] = { xv.x, xv.y, xv.z, xv.w };
                const uint32_t ws[4] = { wv.x, wv.y, wv.z, wv.w };
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    dot += bf16_bits_to_f32(xs[j] & 0xffffu) * bf16_bits_to_f32(ws[j] & 0xffffu);
                    dot += bf16_bits_to_f32(xs[j] >> 16) * bf16_bits_to_f32(ws[j] >> 16);
                }
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            dot += __shfl_xor_sync(0xffffffffu, dot, o);
        if (lane == 0)
            s_dot[group][gl / 32] = dot;
    }
    const uint4* nw = reinterpret_cast<const uint4*>(p.norm_weight);
    uint4* res = reinterpret_cast<uint4*>(p.residual) + static_cast<size_t>(live ? token : 0) * vec_per_row;
    uint4 own_res = make_uint4(0, 0, 0, 0), own_nw = make_uint4(0, 0, 0, 0); // one token per block: a thread has one chunk
    if (TOKENS == 1 && live && gl < vec_per_row) {
        own_res = res[gl];
        own_nw = nw[gl];
    }
    if (p.early) // all of the above is older than the predecessor
        chain_begin();
    __syncthreads();
    float gate = 0.0f;
    if (p.shared_out != nullptr) {
        dot = 0.0f;
#pragma unroll
        for (uint32_t w = 0; w < kGroup / 32; ++w)
            dot += s_dot[group][w];
        gate = sigmoid_fast(dot);
    }

    const uint32_t n_valid = live ? static_cast<uint32_t>(s_any[group]) : 0u;
    float vals[TOKENS][8]; // chunks gl, gl + kGroup, ... of the row
    float sum_sq = 0.0f;
#pragma unroll
    for (uint32_t c0 = 0; c0 < TOKENS; c0 += kStep) {
        sum_routes<kStep, BATCH, kGroup>(p, s_row[group], s_w[group], n_valid, gl + c0 * kGroup, vec_per_row, vals + c0);
#pragma unroll
        for (uint32_t c = c0; c < c0 + kStep; ++c) {
            float* acc = vals[c];
            const uint32_t i = gl + c * kGroup;
            if (!live || i >= vec_per_row)
                continue;
            if (p.shared_out != nullptr)
                add_shared(p, token, vec_per_row, i, gate, acc);
            const uint4 rv = TOKENS == 1 ? own_res : res[i];
            const uint32_t rs[4] = { rv.x, rv.y, rv.z, rv.w };
            uint32_t o[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                // the MoE output as the unfused path would have stored it, plus the residual
                const float x0 = __bfloat162float(__float2bfloat16(acc[2 * j]));
                const float x1 = __bfloat162float(__float2bfloat16(acc[2 * j + 1]));
                acc[2 * j] = x0 + bf16_bits_to_f32(rs[j] & 0xffffu);
                acc[2 * j + 1] = x1 + bf16_bits_to_f32(rs[j] >> 16);
                sum_sq += acc[2 * j] * acc[2 * j] + acc[2 * j + 1] * acc[2 * j + 1];
                const __nv_bfloat162 r2 = __floats2bfloat162_rn(acc[2 * j], acc[2 * j + 1]);
                o[j] = *reinterpret_cast<const uint32_t*>(&r2);
            }
            res[i] = make_uint4(o[0], o[1], o[2], o[3]);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        sum_sq += __shfl_xor_sync(0xffffffffu, sum_sq, o);
    if (lane == 0)
        s_sq[group][gl / 32] = sum_sq;
    __syncthreads();
    if (!live)
        return;
    float total = 0.0f;
#pragma unroll
    for (uint32_t w = 0; w < kGroup / 32; ++w)
        total += s_sq[group][w];
    const float inv_rms = 1.0f / sqrtf(total / static_cast<float>(p.hidden_size) + p.norm_eps);
    uint4* out = reinterpret_cast<uint4*>(p.out) + static_cast<size_t>(token) * vec_per_row;
#pragma unroll
    for (uint32_t c = 0; c < TOKENS; ++c) {
        const uint32_t i = gl + c * kGroup;
        if (i >= vec_per_row)
            continue;
        const uint4 wv = TOKENS == 1 ? own_nw : nw[i];
        const uint32_t ws[4] = { wv.x, wv.y, wv.z, wv.w };
        uint32_t o[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const __nv_bfloat162 r2
                = __floats2bfloat162_rn(vals[c][2 * j] * inv_rms * bf16_bits_to_f32(ws[j] & 0xffffu),
                                        vals[c][2 * j + 1] * inv_rms * bf16_bits_to_f32(ws[j] >> 16));
            o[j] = *reinterpret_cast<const uint32_t*>(&r2);
        }
        out[i] = make_uint4(o[0], o[1], o[2], o[3]);
    }
}

// rows[t * ranks + r] = r * tokens + t, weights = 1: lets the combine kernel sum the
// per-rank partial rows of one token in ascending rank order.
__global__ void ep_rank_routes_kernel(int32_t* rows, float* weights, uint32_t tokens, uint32_t ranks)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= tokens * ranks)
        return;
    rows[i] = static_cast<int32_t>((i % ranks) * tokens + i / ranks);
    weights[i] = 1.0f;
}

// Per token: dispatch ids out[t, k] = map[ids[t, k]] (ids outside the map stay -1; without a map the
// ids themselves are the dispatch ids) and mask[t] = the set of ranks the token has a route to (bit r:
// some dispatch id lies in rank r's `per_rank` expert slots). The map turns the router's expert ids
// into the expert SLOTS of a placement in which every rank holds its own experts and replicas of hot ones.
__global__ void ep_route_targets_kernel(const int32_t* __restrict__ ids, const int32_t* __restrict__ map,
                                        uint32_t map_len, int32_t* __restrict__ out, uint32_t* __restrict__ mask,
                                        uint32_t tokens, uint32_t top_k, uint32_t per_rank, uint32_t ranks)
{
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= tokens)
        return;
    uint32_t m = 0;
    for (uint32_t k = 0; k < top_k; ++k) {
        int32_t id = ids[static_cast<size_t>(t) * top_k + k];
        if (map != nullptr) {
            id = (id >= 0 && static_cast<uint32_t>(id) < map_len) ? map[id] : -1;
            out[static_cast<size_t>(t) * top_k + k] = id;
        }
        if (id >= 0 && static_cast<uint32_t>(id) / per_rank < ranks)
            m |= 1u << (static_cast<uint32_t>(id) / per_rank);
    }
    if (mask != nullptr)
        mask[t] = m;
}

// Dispatch that pulls only what this rank needs: for every token of every rank, its dispatch ids
// and weights always (the route sort needs them to see that a row is not local), its NVFP4 codes and
// scales only when the token's rank mask says it has a route to an expert slot of this rank. A warp
// takes eight consecutive tokens of one peer: eight lanes fetch the masks, then the warp issues
// the loads of all wanted rows before storing any of them, so that the NVLink round trips overlap.
// Rows that are not pulled keep whatever an earlier step left there; nothing reads them, because
// none of their (fresh) ids is local. Plain peer loads; no load of this kernel is multicast.
__global__ void __launch_bounds__(256) ep_pull_routed_kernel(EpPullRoutedParams p)
{
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t groups_per_rank = (p.num_tokens + 7) / 8;
    const uint32_t group = blockIdx.x * 8 + warp;
    if (group >= groups_per_rank * p.num_ranks)
        return;
    const uint32_t r = group / groups_per_rank;
    const uint32_t t0 = (group % groups_per_rank) * 8;
    const uint8_t* peer = p.peer[r];
    const uint32_t nrows = min(8u, p.num_tokens - t0);
    uint32_t my_mask = 0;
    if (lane < nrows)
        my_mask = reinterpret_cast<const uint32_t*>(peer + p.off_mask)[t0 + lane];
    // ids and weights of the eight tokens: 8 * top_k words each, contiguous in the peer's block
    const uint32_t words = nrows * p.top_k;
    const uint32_t* ids_src = reinterpret_cast<const uint32_t*>(peer + p.off_ids) + static_cast<size_t>(t0) * p.top_k;
    const uint32_t* wts_src = reinterpret_cast<const uint32_t*>(peer + p.off_wts) + static_cast<size_t>(t0) * p.top_k;
    const size_t row0 = static_cast<size_t>(r) * p.num_tokens + t0;
    uint32_t* ids_dst = reinterpret_cast<uint32_t*>(p.dst_ids) + row0 * p.top_k;
    uint32_t* wts_dst = reinterpret_cast<uint32_t*>(p.dst_wts) + row0 * p.top_k;
    uint32_t iv[4], wv[4];
#pragma unroll
    for (uint32_t q = 0; q < 4; ++q) {
        const uint32_t i = lane + 32 * q;
        iv[q] = i < words ? ids_src[i] : 0;
        wv[q] = i < words ? wts_src[i] : 0;
    }
    uint32_t wanted = 0; // bit i: row t0 + i goes to this rank
#pragma unroll
    for (uint32_t i = 0; i < 8; ++i)
        wanted |= ((__shfl_sync(0xffffffffu, my_mask, i) >> p.my_rank) & 1u) << i;
    // codes: code_vecs 16-byte vectors per row (<= 64 per lane pair of loads), scales: scale_vecs (<= 32)
    const uint4* codes = reinterpret_cast<const uint4*>(peer + p.off_codes);
    const uint4* scales = reinterpret_cast<const uint4*>(peer + p.off_scales);
    uint4* codes_dst = reinterpret_cast<uint4*>(p.dst_codes);
    uint4* scales_dst = reinterpret_cast<uint4*>(p.dst_scales);
    for (uint32_t i0 = 0; i0 < 8; i0 += 4) {
        uint4 c[4][2], sc[4];
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j) {
            const uint32_t i = i0 + j;
            const bool on = (wanted >> i) & 1u;
            const size_t src_row = t0 + i;
#pragma unroll
            for (uint32_t h = 0; h < 2; ++h)
                if (on && lane + 32 * h < p.code_vecs)
                    c[j][h] = codes[src_row * p.code_vecs + lane + 32 * h];
            if (on && lane < p.scale_vecs)
                sc[j] = scales[src_row * p.scale_vecs + lane];
        }
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j) {
            const uint32_t i = i0 + j;
            if (!((wanted >> i) & 1u))
                continue;
            const size_t dst_row = row0 + i;
#pragma unroll
            for (uint32_t h = 0; h < 2; ++h)
                if (lane + 32 * h < p.code_vecs)
                    codes_dst[dst_row * p.code_vecs + lane + 32 * h] = c[j][h];
            if (lane < p.scale_vecs)
                scales_dst[dst_row * p.scale_vecs + lane] = sc[j];
        }
    }
#pragma unroll
    for (uint32_t q = 0; q < 4; ++q) {
        const uint32_t i = lane + 32 * q;
        if (i < words) {
            ids_dst[i] = iv[q];
            wts_dst[i] = wv[q];
        }
    }
}

template <typename T> T* carve(char* base, size_t& offset, size_t count)
{
    offset = align_up(offset, kWorkspaceAlign);
    T* p = base != nullptr ? reinterpret_cast<T*>(base + offset) : nullptr;
    offset += count * sizeof(T);
    return p;
}

// Expert-parallel combine that PULLS: out[t] = bf16(sum over ranks r, ascending, of
// f32(partial_r[my_rank * T + t]) + sigmoid(x . w_gate) * shared[t]), where partial_r is
// rank r's partial-sum buffer read in place over NVLink (plain peer loads). A rank is
// read only when one of the token's routes targets one of its experts, so pairs
// (token, rank) without a route cost no traffic. Same summation order and roundings as
// exchanging the partial sums first and then running combine_kernel on the copies.
// Four tokens per block, 64 threads (two warps) per token: the kernel is bound by the latency of its
// dependent loads (ids -> which ranks -> peer rows over NVLink), so what matters is how many tokens
// are in flight per SM; with a block per token 4096 tokens took 3.5 waves of ~8 us.
constexpr uint32_t kEpTokensPerBlock = 4;

__global__ void __launch_bounds__(64 * kEpTokensPerBlock, 3) ep_pull_combine_kernel(EpPullParams p)
{
    __shared__ uint32_t s_active[kEpTokensPerBlock];
    __shared__ float s_dot[kEpTokensPerBlock][2];
    const uint32_t slot = threadIdx.x >> 6;           // token of the block
    const uint32_t tid = threadIdx.x & 63;            // thread of the token
    const uint32_t lane = threadIdx.x & 31, half = tid >> 5;
    const uint32_t token = blockIdx.x * kEpTokensPerBlock + slot;
    const bool live = token < p.num_tokens;
    const uint32_t vec_per_row = p.hidden_size / 8;

    // which ranks hold a partial sum for this token
    if (live && half == 0) {
        uint32_t mine = 0;
        if (lane < p.top_k) {
            const int id = p.topk_ids[static_cast<size_t>(token) * p.top_k + lane];
            if (id >= 0 && static_cast<uint32_t>(id) / p.experts_per_rank < p.num_ranks)
                mine = 1u << (static_cast<uint32_t>(id) / p.experts_per_rank);
        }
        const uint32_t any = __reduce_or_sync(0xffffffffu, mine);
        if (lane == 0)
            s_active[slot] = any;
    }
    float dot = 0.0f;
    if (live && p.shared_out != nullptr) {
        // gate logit: the row's loads are issued together (four chunks per thread and pass)
        const uint4* x = reinterpret_cast<const uint4*>(p.hidden) + static_cast<size_t>(token) * vec_per_row;
        const uint4* w = reinterpret_cast<const uint4*>(p.gate_w);
        for (uint32_t i0 = tid; i0 < vec_per_row; i0 += 256) {
            uint4 xv[4], wv[4];
#pragma unroll
            for (uint32_t c = 0; c < 4; ++c) {
                const uint32_t i = i0 + 64 * c;
                xv[c] = i < vec_per_row ? x[i] : make_uint4(0, 0, 0, 0);
                wv[c] = i < vec_per_row ? w[i] : make_uint4(0, 0, 0, 0);
            }
#pragma unroll
            for (uint32_t c = 0; c < 4; ++c) {
                const uint32_t xs[4] = { xv[c].x, xv[c].y, xv[c].z, xv[c].w };
                const uint32_t ws[4] = { wv[c].x, wv[c].y, wv[c].z, wv[c].w };
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    dot += bf16_bits_to_f32(xs[j] & 0xffffu) * bf16_bits_to_f32(ws[j] & 0xffffu);
                    dot += bf16_bits_to_f32(xs[j] >> 16) * bf16_bits_to_f32(ws[j] >> 16);
                }
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            dot += __shfl_xor_sync(0xffffffffu, dot, o);
        if (lane == 0)
            s_dot[slot][half] = dot;
    }
    __syncthreads();
    if (!live)
        return;
    const uint32_t active = (p.dbg & 1u) ? (s_active[slot] & (1u << p.my_rank)) : s_active[slot];
    float gate = 0.0f;
    if (p.shared_out != nullptr)
        gate = sigmoid_fast(s_dot[slot][0] + s_dot[slot][1]);

    const size_t row = static_cast<size_t>(p.my_rank) * p.num_tokens + token;
    uint4* out = reinterpret_cast<uint4*>(p.out) + static_cast<size_t>(token) * vec_per_row;
    // A thread owns up to four 16-byte chunks of the row (hidden <= 2048) and keeps the loads of all of
    // them, for two ranks at a time, in flight together: what bounds this kernel is the latency of the
    // peer loads, so the number of dependent rounds (ranks / 2), not the bytes, sets its time. Ranks are
    // added in ascending order.
    constexpr uint32_t kChunks = 4;
    for (uint32_t i0 = tid; i0 < vec_per_row; i0 += 64 * kChunks) {
        float acc[kChunks][8];
#pragma unroll
        for (uint32_t c = 0; c < kChunks; ++c)
#pragma unroll
            for (int j = 0; j < 8; ++j)
                acc[c][j] = 0.0f;
        // the shared expert's rows travel with the first round of partial sums
        uint4 sh[kChunks];
#pragma unroll
        for (uint32_t c = 0; c < kChunks; ++c) {
            const uint32_t i = i0 + 64 * c;
            sh[c] = (p.shared_out != nullptr && i < vec_per_row)
                ? reinterpret_cast<const uint4*>(p.shared_out)[static_cast<size_t>(token) * vec_per_row + i]
                : make_uint4(0, 0, 0, 0);
        }
        uint32_t todo = active & (p.num_ranks >= 32 ? 0xffffffffu : (1u << p.num_ranks) - 1u);
        while (todo != 0) {
            const uint32_t ra = static_cast<uint32_t>(__ffs(static_cast<int>(todo))) - 1u;
            todo &= todo - 1u;
            const bool two = todo != 0;
            const uint32_t rb = two ? static_cast<uint32_t>(__ffs(static_cast<int>(todo))) - 1u : ra;
            todo &= todo - 1u; // no-op on zero
            const uint4* pa = reinterpret_cast<const uint4*>(p.peer[ra]) + row * vec_per_row;
            const uint4* pb = reinterpret_cast<const uint4*>(p.peer[rb]) + row * vec_per_row;
            uint4 va[kChunks], vb[kChunks];
#pragma unroll
            for (uint32_t c = 0; c < kChunks; ++c) {
                const uint32_t i = i0 + 64 * c;
                va[c] = i < vec_per_row ? pa[i] : make_uint4(0, 0, 0, 0);
                vb[c] = (two && i < vec_per_row) ? pb[i] : make_uint4(0, 0, 0, 0);
            }
#pragma unroll
            for (uint32_t c = 0; c < kChunks; ++c) {
                const uint32_t as[4] = { va[c].x, va[c].y, va[c].z, va[c].w };
                const uint32_t bs[4] = { vb[c].x, vb[c].y, vb[c].z, vb[c].w };
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    acc[c][2 * j] += bf16_bits_to_f32(as[j] & 0xffffu);
                    acc[c][2 * j + 1] += bf16_bits_to_f32(as[j] >> 16);
                }
                if (two) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        acc[c][2 * j] += bf16_bits_to_f32(bs[j] & 0xffffu);
                        acc[c][2 * j + 1] += bf16_bits_to_f32(bs[j] >> 16);
                    }
                }
            }
        }
#pragma unroll
        for (uint32_t c = 0; c < kChunks; ++c) {
            const uint32_t i = i0 + 64 * c;
            if (i >= vec_per_row)
                break;
            if (p.shared_out != nullptr) {
                const uint32_t ss[4] = { sh[c].x, sh[c].y, sh[c].z, sh[c].w };
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    acc[c][2 * j] += gate * bf16_bits_to_f32(ss[j] & 0xffffu);
                    acc[c][2 * j + 1] += gate * bf16_bits_to_f32(ss[j] >> 16);
                }
            }
            uint32_t o[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const __nv_bfloat162 r2 = __floats2bfloat162_rn(acc[c][2 * j], acc[c][2 * j + 1]);
                o[j] = *reinterpret_cast<const uint32_t*>(&r2);
            }
            out[i] = make_uint4(o[0], o[1], o[2], o[3]);
        }
    }
}

// dst_j[r * bytes_j ...] = peer block r, segment j: every rank copies the token blocks of all
// ranks (its own included) out of the ranks' symmetric buffers with plain 16-byte peer loads.
// Grid: (chunks, ranks, segments).
__global__ void __launch_bounds__(256) ep_pull_tokens_kernel(EpPullTokensParams p)
{
    const uint32_t r = blockIdx.y, seg = blockIdx.z;
    const uint64_t vecs = p.seg_bytes[seg] / 16;
    const uint4* src = reinterpret_cast<const uint4*>(p.peer[r] + p.seg_offset[seg]);
    uint4* dst = reinterpret_cast<uint4*>(p.dst[seg] + static_cast<uint64_t>(r) * p.seg_bytes[seg]);
    const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
    for (uint64_t i0 = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i0 < vecs; i0 += 4 * stride) {
        uint4 v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (i0 + q * stride < vecs)
                v[q] = src[i0 + q * stride];
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (i0 + q * stride < vecs)
                dst[i0 + q * stride] = v[q];
    }
}

} // namespace

cudaError_t launch_ep_pull_combine(const EpPullParams& params, cudaStream_t stream)
{
    if (params.num_tokens == 0)
        return cudaSuccess;
    EpPullParams p = params;
    static const uint32_t dbg = [] {
        const char* v = std::getenv("QS3_EP_FINISH_DBG");
        return v != nullptr ? static_cast<uint32_t>(std::atoi(v)) : 0u;
    }();
    p.dbg = dbg;
    ep_pull_combine_kernel<<<(p.num_tokens + kEpTokensPerBlock - 1) / kEpTokensPerBlock, 64 * kEpTokensPerBlock, 0,
                             stream>>>(p);
    note_launch();
    return cudaGetLastError();
}

cudaError_t launch_ep_pull_tokens(const EpPullTokensParams& p, cudaStream_t stream)
{
    if (p.num_ranks == 0 || p.num_segments == 0)
        return cudaSuccess;
    uint64_t largest = 0;
    for (uint32_t j = 0; j < p.num_segments; ++j)
        largest = std::max<uint64_t>(largest, p.seg_bytes[j]);
    const uint32_t chunks = static_cast<uint32_t>(std::min<uint64_t>(2 * 148, std::max<uint64_t>(1, largest / 16 / 1024)));
    ep_pull_tokens_kernel<<<dim3(chunks, p.num_ranks, p.num_segments), 256, 0, stream>>>(p);
    note_launch();
    return cudaGetLastError();
}

cudaError_t launch_ep_route_targets(const int32_t* ids, const int32_t* map, uint32_t map_len, int32_t* out,
                                    uint32_t* mask, uint32_t tokens, uint32_t top_k, uint32_t per_rank,
                                    uint32_t ranks, cudaStream_t stream)
{
    if (tokens == 0 || (map == nullptr && mask == nullptr))
        return cudaSuccess;
    ep_route_targets_kernel<<<(tokens + 255) / 256, 256, 0, stream>>>(ids, map, map_len, out, mask, tokens, top_k,
                                                                      per_rank, ranks);
    note_launch();
    return cudaGetLastError();
}

cudaError_t launch_ep_pull_routed(const EpPullRoutedParams& p, cudaStream_t stream)
{
    if (p.num_ranks == 0 || p.num_tokens == 0)
        return cudaSuccess;
    const uint32_t groups = (p.num_tokens + 7) / 8 * p.num_ranks;
    ep_pull_routed_kernel<<<(groups + 7) / 8, 256, 0, stream>>>(p);
    note_launch();
    return cudaGetLastError();
}

cudaError_t launch_ep_rank_routes(int32_t* rows, float* weights, uint32_t tokens, uint32_t ranks,
                                  cudaStream_t stream)
{
    const uint32_t total = tokens * ranks;
    ep_rank_routes_kernel<<<(total + 255) / 256, 256, 0, stream>>>(rows, weights, tokens, ranks);
    note_launch();
    return cudaGetLastError();
}

bool route_sort_can_choose(uint32_t routes, uint32_t experts)
{
    return (routes > kBlockSortRoutes || experts > kBlockSortExperts) && experts <= 1024;
}

namespace {

// Blocks of the one-block sorts beyond the first: a warp per 512 elements to quantise (FP8: 256).
uint32_t quant_blocks(const TokenQuant* quant)
{
    if (quant == nullptr)
        return 0;
    const uint64_t units = quant->fp8_scale != nullptr ? (static_cast<uint64_t>(quant->rows) * (quant->k / 128) + 1) / 2
                                                       : static_cast<uint64_t>(quant->rows) * ((quant->k + 511) / 512);
    return static_cast<uint32_t>((units + kBlockSortWarps - 1) / kBlockSortWarps);
}

} // namespace

bool router_sort_supported(uint32_t num_tokens, uint32_t num_experts, uint32_t top_k, uint32_t experts)
{
    // (16 tokens of 512 experts: the same time in a layer, 1 us more in a captured step)
    return num_tokens <= (num_experts <= 128 ? kBlockSortWarps : kBlockSortWarps / 2) && num_experts <= 512 && top_k <= 32 && num_tokens * top_k <= kBlockSortRoutes
        && experts <= kBlockSortExperts;
}

cudaError_t launch_router_sort(const float* logits, const float* bias, int32_t* ids, float* weights, uint32_t num_tokens,
                               uint32_t num_experts, uint32_t top_k, int sigmoid_score, int renormalize, float scaling,
                               uint32_t local_offset, uint32_t experts, const RouteTables& rt, cudaStream_t stream,
                               const TokenQuant* quant)
{
    const RouterParams r { logits, bias, ids, weights, num_tokens, num_experts, sigmoid_score, renormalize, scaling };
    const uint32_t per_lane = (num_experts + 31) / 32;
    const auto kernel = per_lane <= 1 ? router_sort_block_kernel<1>
        : per_lane <= 4               ? router_sort_block_kernel<4>
        : per_lane <= 8               ? router_sort_block_kernel<8>
                                      : router_sort_block_kernel<16>;
    return launch_chained(kernel, dim3(1 + quant_blocks(quant)), kBlockSortThreads, block_sort_smem(experts), stream, r, top_k,
                          local_offset, experts, rt, quant != nullptr ? *quant : TokenQuant {});
}

size_t route_tables_carve(char* base, uint32_t routes, uint32_t experts, RouteTables* out, uint32_t tile_rows,
                          uint32_t shared_rows, uint32_t alt_tile_rows)
{
    RouteTables rt {};
    size_t off = 0;
    const uint64_t seg = routes < experts ? routes : experts; // experts that can hold a row
    const uint64_t max_pad_rows = align_up(routes, tile_rows) + seg * tile_rows + align_up(shared_rows, tile_rows);
    rt.tile_rows = tile_rows;
    rt.shared_rows = shared_rows;
    rt.max_pad_rows = static_cast<uint32_t>(max_pad_rows);
    rt.max_tiles = static_cast<uint32_t>(max_pad_rows / tile_rows);
    uint32_t tiles = rt.max_tiles; // room in the tables
    // A plan keeps the room of the largest choice beyond it: a workspace for many tokens serves fewer as well.
    const bool alt = alt_tile_rows != 0 && routes <= kAltMaxRoutes * experts;
    if (alt_tile_rows != 0) {
        const uint32_t alt_routes = alt ? routes : kAltMaxRoutes * experts;
        const uint32_t alt_tiles = static_cast<uint32_t>(align_up(alt_routes, alt_tile_rows) / alt_tile_rows + seg);
        tiles = alt_tiles > tiles ? alt_tiles : tiles;
        if (alt) { // (no more padded rows than with the larger tiles)
            rt.alt_tile_rows = alt_tile_rows;
            rt.alt_max_tiles = alt_tiles;
        }
    }
    rt.route_blocks = (routes + kSortChunk - 1) / kSortChunk;
    rt.counts = carve<int32_t>(base, off, experts);
    rt.indptr = carve<int32_t>(base, off, experts + 1);
    rt.pad_indptr = carve<int32_t>(base, off, experts + 1);
    rt.route_rows = carve<int32_t>(base, off, routes);
    rt.route_prows = carve<int32_t>(base, off, routes);
    rt.row_tokens = carve<int32_t>(base, off, routes);
    rt.row_scales = carve<float>(base, off, routes);
    rt.tile_expert = carve<int32_t>(base, off, tiles);
    rt.tile_row0 = carve<int32_t>(base, off, tiles);
    rt.tile_nrows = carve<int32_t>(base, off, tiles);
    rt.total_tiles = carve<int32_t>(base, off, 1);
    if (alt_tile_rows != 0) {
        int32_t* const alt_total = carve<int32_t>(base, off, 1);
        rt.alt_total_tiles = alt ? alt_total : nullptr;
    }
    if (tile_rows == static_cast<uint32_t>(kTileM)) {
        rt.pair_expert = carve<int32_t>(base, off, rt.max_tiles);
        rt.pair_row0 = carve<int32_t>(base, off, rt.max_tiles);
        rt.pair_nrows = carve<int32_t>(base, off, rt.max_tiles);
        rt.pair_counts = carve<int32_t>(base, off, 2);
    }
    rt.block_hist = carve<int32_t>(base, off, static_cast<size_t>(rt.route_blocks) * experts);
    if (out != nullptr)
        *out = rt;
    return align_up(off, kWorkspaceAlign);
}

size_t route_tables_bytes(uint32_t routes, uint32_t experts)
{
    return route_tables_carve(nullptr, routes, experts, nullptr);
}

cudaError_t launch_route_sort(const int32_t* topk_ids, const float* topk_weights, uint32_t routes,
                              uint32_t top_k, uint32_t local_offset, uint32_t experts,
                              const RouteTables& rt, cudaStream_t stream, const TokenQuant* quant)
{
    if (routes <= kBlockSortRoutes && experts <= kBlockSortExperts) {
        return launch_chained(route_sort_block_kernel, dim3(1 + quant_blocks(quant)), kBlockSortThreads,
                              block_sort_smem(experts), stream, topk_ids, topk_weights, routes, top_k, local_offset, experts,
                              rt, quant != nullptr ? *quant : TokenQuant {});
    }
    if (quant != nullptr) {
        const cudaError_t err = quant->fp8_scale != nullptr
            ? launch_fp8_quantize_rows(quant->x, quant->rows, quant->k, quant->packed, quant->fp8_scale, stream)
            : launch_nvfp4_quantize_rows(quant->x, quant->rows, quant->k, quant->global_scale, quant->packed,
                                         quant->scale_tiled, stream);
        if (err != cudaSuccess)
            return err;
    }
    // (the histograms of fewer than eight experts, padded to eight, do not fit the room of the other kernels')
    if (experts >= 8 && experts <= kSpMaxExperts && rt.route_blocks <= kSpMaxChunks) {
        const size_t pitch = sp_pitch(experts);
        uint16_t* hist = reinterpret_cast<uint16_t*>(rt.block_hist);
        const cudaError_t err = launch_chained(route_chunk_hist_kernel, dim3(rt.route_blocks), kSpThreads, pitch * sizeof(uint32_t),
                                               stream, topk_ids, routes, local_offset, experts, hist);
        if (err != cudaSuccess)
            return err;
        return launch_chained(route_scan_place_kernel, dim3(rt.route_blocks), kSpThreads,
                              pitch * 3 * sizeof(uint32_t) + kSpWarps * static_cast<size_t>(experts) * sizeof(uint16_t), stream,
                              topk_ids, topk_weights, routes, top_k, local_offset, experts, static_cast<const uint16_t*>(hist), rt);
    }
    const size_t smem = static_cast<size_t>(kSortWarps) * experts * sizeof(uint16_t);
    if (smem > 200 * 1024)
        return cudaErrorInvalidValue;
    if (smem > 48 * 1024) {
        cudaError_t err = cudaFuncSetAttribute(route_hist_kernel,
                                               cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               static_cast<int>(smem));
        if (err == cudaSuccess)
            err = cudaFuncSetAttribute(route_place_kernel,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       static_cast<int>(smem));
        if (err != cudaSuccess)
            return err;
    }
    cudaError_t err = launch_chained(route_hist_kernel, dim3(rt.route_blocks), kSortWarps * 32, smem, stream, topk_ids,
                                     routes, local_offset, experts, rt.block_hist);
    if (err == cudaSuccess)
        err = launch_chained(route_scan_kernel, dim3(1), 1024, 0, stream, rt.block_hist, rt.route_blocks, experts, rt);
    if (err == cudaSuccess)
        err = launch_chained(route_place_kernel, dim3(rt.route_blocks), kSortWarps * 32, smem, stream, topk_ids,
                             topk_weights, routes, top_k, local_offset, experts, rt);
    return err;
}

cudaError_t launch_gather_rows(const void* src, uint32_t row_bytes, const RouteTables& rt, uint32_t min_rows, void* dst,
                               cudaStream_t stream)
{
    if (rt.max_tiles == 0)
        return cudaSuccess;
    const uint32_t block_rows = rt.max_tiles * (rt.tile_rows / 8) <= 8 * kSmCount ? 8 : 32;
    return launch_chained(gather_rows_kernel, dim3(rt.tile_rows / block_rows, rt.max_tiles), 256, 0, stream,
                          static_cast<const uint4*>(src), row_bytes / 16, rt, static_cast<int>(min_rows),
                          static_cast<uint4*>(dst));
}

cudaError_t launch_combine(const CombineParams& p, cudaStream_t stream)
{
    if (p.num_tokens == 0)
        return cudaSuccess;
    // one block per token while the blocks fit two waves of two per SM (600 tokens: 0.0137 against 0.0142 ms, 1021: 0.019
    // against 0.014)
    const bool spread = p.num_tokens <= 4 * device_sm_count();
    const uint32_t blocks = spread ? p.num_tokens : (p.num_tokens + 3) / 4;
    if (p.residual != nullptr) {
        if (p.hidden_size > kCombineThreads * 8 || p.skip_empty)
            return cudaErrorNotSupported;
        return launch_chained(spread ? combine_norm_kernel<1, 16> : combine_norm_kernel<4, 4>, dim3(blocks),
                              kCombineThreads, 0, stream, p);
    }
    return launch_chained(spread ? combine_kernel<1, 1, 16> : combine_kernel<4, 2, 4>, dim3(blocks), kCombineThreads, 0,
                          stream, p);
}

} // namespace qs3

// ---- route sort without any allocation ------------------------------------------------
//
// qs3_moe_route_sort_static runs the same three counting-sort kernels as the MoE
// execute calls, but takes its scratch (block histograms, padded segment starts, tile
// table) from the fixed array below instead of a caller workspace. It is meant for
// callers that cannot obtain device memory at the point where they need the routing
// tables: a serving process that handed its whole HBM budget to weight and cache pools
// at start-up and forbids later cudaMalloc, or code inside a latency-critical or
// stream-ordered section where cudaMalloc's implicit device-wide synchronisation is
// not acceptable. The price is a hard size limit and a buffer that every device
// loading this library keeps until the process exits.
namespace {

constexpr size_t kStaticScratchBytes = QS3_ROUTE_SORT_STATIC_SCRATCH_BYTES;

// Device-resident scratch. In HOST code this name is only a handle for the runtime's
// symbol table, not a device address: kernels must be given the pointer that
// cudaGetSymbolAddress returns (looked up once per device below).
static __device__ __align__(256) unsigned char g_route_sort_scratch[kStaticScratchBytes];

// Per-device address of g_route_sort_scratch, resolved with that device current.
cudaError_t static_scratch_base(unsigned char** out)
{
    static std::mutex mu;
    static unsigned char* base[64] = {};
    int dev = -1;
    cudaError_t err = cudaGetDevice(&dev);
    if (err != cudaSuccess)
        return err;
    if (dev < 0 || dev >= 64)
        return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lock(mu);
    if (base[dev] == nullptr) {
        unsigned char* ptr = nullptr;
        err = cudaGetSymbolAddress(reinterpret_cast<void**>(&ptr), g_route_sort_scratch);
        if (err != cudaSuccess)
            return err;
        if (ptr == nullptr)
            return cudaErrorInvalidSymbol;
        base[dev] = ptr;
    }
    *out = base[dev];
    return cudaSuccess;
}

template <typename T> T* static_take(unsigned char* base, size_t& offset, size_t count)
{
    offset = qs3::align_up(offset, qs3::kWorkspaceAlign);
    T* p = reinterpret_cast<T*>(base + offset);
    offset += count * sizeof(T);
    return p;
}

bool bad_out(const qsfi_tensor1& t, qsfi_dtype dtype, uint64_t count)
{
    return t.data == nullptr || t.dtype != dtype || t.stride[0] != 1 || t.shape[0] < 0
        || static_cast<uint64_t>(t.shape[0]) < count || (reinterpret_cast<uintptr_t>(t.data) & 3u) != 0;
}

} // namespace

extern "C" qsfi_status qs3_moe_route_sort_static(qsfi_context* ctx, const qs3_route_sort_static_desc* d)
{
    using namespace qs3;
    if (ctx == nullptr)
        return QSFI_STATUS_INVALID_ARGUMENT;
    clear_error(&ctx->last_error);
    qsfi_status status = activate_context(ctx);
    if (status != QSFI_STATUS_OK)
        return status;
    if (d == nullptr)
        return set_invalid_arg(ctx, "desc is null");
    if (d->num_tokens == 0 || d->top_k == 0 || d->local_num_experts == 0)
        return set_invalid_arg(ctx, "route sort dimensions must be non-zero");
    const uint64_t routes64 = static_cast<uint64_t>(d->num_tokens) * d->top_k;
    if (routes64 > QS3_ROUTE_SORT_STATIC_MAX_ROUTES || d->local_num_experts > QS3_ROUTE_SORT_STATIC_MAX_EXPERTS)
        return set_unsupported(
            ctx,
            "qs3_moe_route_sort_static handles at most %u routes and %u local experts (got %llu and %u); "
            "use an execute call with a caller workspace for larger problems",
            QS3_ROUTE_SORT_STATIC_MAX_ROUTES, QS3_ROUTE_SORT_STATIC_MAX_EXPERTS,
            static_cast<unsigned long long>(routes64), d->local_num_experts);
    const uint32_t routes = static_cast<uint32_t>(routes64);
    const uint32_t experts = d->local_num_experts;
    if (d->topk_ids.data == nullptr || d->topk_ids.dtype != QSFI_DTYPE_I32 || !contiguous2(d->topk_ids)
        || d->topk_ids.shape[0] != d->num_tokens || d->topk_ids.shape[1] != d->top_k)
        return set_invalid_arg(ctx, "topk_ids must be a contiguous i32 [num_tokens, top_k] tensor");
    if (d->topk_weights.data == nullptr || d->topk_weights.dtype != QSFI_DTYPE_F32
        || !contiguous2(d->topk_weights) || d->topk_weights.shape[0] != d->num_tokens
        || d->topk_weights.shape[1] != d->top_k)
        return set_invalid_arg(ctx, "topk_weights must be a contiguous f32 [num_tokens, top_k] tensor");
    if (bad_out(d->counts, QSFI_DTYPE_I32, experts) || bad_out(d->indptr, QSFI_DTYPE_I32, experts + 1ull)
        || bad_out(d->route_rows, QSFI_DTYPE_I32, routes) || bad_out(d->row_tokens, QSFI_DTYPE_I32, routes)
        || bad_out(d->row_scales, QSFI_DTYPE_F32, routes))
        return set_invalid_arg(ctx, "route sort outputs must be contiguous i32/f32 vectors of the documented length");

    unsigned char* base = nullptr;
    cudaError_t err = static_scratch_base(&base);
    if (err != cudaSuccess)
        return set_cuda_error(ctx, err, "cudaGetSymbolAddress(route sort scratch)");

    // caller-owned outputs + scratch-owned internals; every scratch word that a kernel
    // reads is written earlier in the same call, so nothing needs clearing between calls
    RouteTables rt {};
    size_t off = 0;
    const uint64_t seg = routes < experts ? routes : experts;
    rt.tile_rows = kTileM;
    rt.max_pad_rows = static_cast<uint32_t>(align_up(routes, kTileM) + seg * kTileM);
    rt.max_tiles = rt.max_pad_rows / kTileM;
    rt.route_blocks = (routes + kSortChunk - 1) / kSortChunk;
    rt.counts = static_cast<int32_t*>(d->counts.data);
    rt.indptr = static_cast<int32_t*>(d->indptr.data);
    rt.route_rows = static_cast<int32_t*>(d->route_rows.data);
    rt.row_tokens = static_cast<int32_t*>(d->row_tokens.data);
    rt.row_scales = static_cast<float*>(d->row_scales.data);
    rt.pad_indptr = static_take<int32_t>(base, off, experts + 1ull);
    rt.route_prows = static_take<int32_t>(base, off, routes);
    rt.tile_expert = static_take<int32_t>(base, off, rt.max_tiles);
    rt.tile_row0 = static_take<int32_t>(base, off, rt.max_tiles);
    rt.tile_nrows = static_take<int32_t>(base, off, rt.max_tiles);
    rt.total_tiles = static_take<int32_t>(base, off, 1);
    rt.block_hist = static_take<int32_t>(base, off, static_cast<size_t>(rt.route_blocks) * experts);
    if (off > kStaticScratchBytes)
        return set_unsupported(ctx, "route sort scratch need of %llu bytes exceeds the static %llu bytes",
                               static_cast<unsigned long long>(off),
                               static_cast<unsigned long long>(kStaticScratchBytes));
    err = launch_route_sort(static_cast<const int32_t*>(d->topk_ids.data),
                            static_cast<const float*>(d->topk_weights.data), routes, d->top_k,
                            d->local_expert_offset, experts, rt, ctx->stream);
    return set_cuda_error(ctx, err, "qs3_moe_route_sort_static");
}
