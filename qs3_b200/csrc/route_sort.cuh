// Counting sort of a decode batch's routes by one block (routing.cu, and beside the weights in gemv.cu).
#pragma once

#include "common.cuh"

namespace qs3 {

__device__ __forceinline__ int local_expert(const int32_t* ids, uint32_t route, uint32_t routes,
                                            uint32_t local_offset, uint32_t experts)
{
    if (route >= routes)
        return -1;
    const int local = ids[route] - static_cast<int>(local_offset);
    return (local < 0 || local >= static_cast<int>(experts)) ? -1 : local;
}

// Tiles of the shared expert (all tokens in order), after the experts' `tiles` tiles; called by a whole block.
__device__ __forceinline__ void append_shared_tiles(const RouteTables& rt, uint32_t experts, uint32_t tiles)
{
    for (uint32_t m = threadIdx.x; m * rt.tile_rows < rt.shared_rows; m += blockDim.x) {
        rt.tile_expert[tiles + m] = static_cast<int32_t>(experts);
        rt.tile_row0[tiles + m] = static_cast<int32_t>((tiles + m) * rt.tile_rows);
        rt.tile_nrows[tiles + m] = static_cast<int32_t>(min(rt.tile_rows, rt.shared_rows - m * rt.tile_rows));
    }
}

// ---- counting sort of up to kBlockSortRoutes routes by one block ------------------------------------------------
// Everything stays in shared memory between the routes' local expert ids (`ids`, -1: not local) and the tables: per-warp
// histograms by match_any, prefix over the warps, one packed block scan (routes in the low, tiles in the high
// half), stable placement. Stable in route index, like the sorts of larger batches in routing.cu, whose tables these are.
constexpr uint32_t kBlockSortThreads = 512;
constexpr uint32_t kBlockSortWarps = kBlockSortThreads / 32;
// 512 experts, one block against the two launches of a larger batch: 1280 routes 12.5 / 13.2 us, 2000 14.4 / 13.2, 2560 15.4 /
// 13.3; layers of 2048 routes and fewer are within 2 % either way, of 2560 up to 3 % longer (58.2 / 56.2).
constexpr uint32_t kBlockSortRoutes = 2560;
constexpr uint32_t kBlockSortExperts = 1024; // two per thread; the shared memory stays below 48 KB

inline size_t block_sort_smem(uint32_t experts)
{
    return kBlockSortRoutes * sizeof(int16_t) + (kBlockSortWarps * sizeof(uint16_t) + 2 * sizeof(int32_t)) * static_cast<size_t>(experts);
}

struct BlockSortSmem {
    int16_t* ids;    // [kBlockSortRoutes]
    uint16_t* hist;  // [kBlockSortWarps][experts]
    int32_t* start;  // [experts] dense segment starts
    int32_t* pad;    // [experts] padded segment starts
};

__device__ __forceinline__ BlockSortSmem block_sort_carve(uint8_t* smem, uint32_t experts)
{
    BlockSortSmem s;
    s.start = reinterpret_cast<int32_t*>(smem);
    s.pad = s.start + experts;
    s.ids = reinterpret_cast<int16_t*>(s.pad + experts);
    s.hist = reinterpret_cast<uint16_t*>(s.ids + kBlockSortRoutes);
    return s;
}

__device__ __forceinline__ void block_sort(const BlockSortSmem& s, const float* weights, uint32_t routes, uint32_t top_k,
                                           uint32_t experts, const RouteTables& rt)
{
    __shared__ uint32_t s_total[2][kBlockSortWarps];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rounds = (routes + kBlockSortThreads - 1) / kBlockSortThreads;
    uint16_t* mine = s.hist + static_cast<size_t>(warp) * experts;
    for (uint32_t i = threadIdx.x; i < kBlockSortWarps * experts; i += kBlockSortThreads)
        s.hist[i] = 0;
    __syncthreads();
    const uint32_t base = warp * rounds * 32; // a warp owns a contiguous run of routes
    for (uint32_t r = 0; r < rounds; ++r) {
        const uint32_t route = base + r * 32 + lane;
        const int e = route < routes ? s.ids[route] : -1;
        const uint32_t peers = __match_any_sync(0xffffffffu, e);
        if (e >= 0 && lane == static_cast<uint32_t>(__ffs(static_cast<int>(peers)) - 1))
            mine[e] += static_cast<uint16_t>(__popc(peers));
        __syncwarp();
    }
    __syncthreads();
    // a thread owns up to two neighbouring experts
    const uint32_t per = (experts + kBlockSortThreads - 1) / kBlockSortThreads;
    const uint32_t tile_rows = rt.tile_rows;
    const bool pairing = rt.pair_expert != nullptr;
    uint32_t count[2] = { 0, 0 };
    uint32_t sum0 = 0, sum1 = 0; // tiles << 16 | routes, pairs << 16 | singles
    for (uint32_t j = 0; j < per; ++j) {
        const uint32_t e = threadIdx.x * per + j;
        if (e < experts) {
            uint32_t run = 0;
#pragma unroll
            for (uint32_t w = 0; w < kBlockSortWarps; ++w) {
                const uint32_t v = s.hist[w * experts + e];
                s.hist[w * experts + e] = static_cast<uint16_t>(run);
                run += v;
            }
            count[j] = run;
            rt.counts[e] = static_cast<int32_t>(run);
            const uint32_t tiles = (run + tile_rows - 1) / tile_rows;
            sum0 += tiles << 16 | run;
            sum1 += (tiles >> 1) << 16 | (tiles & 1);
        }
    }
    uint32_t inc0 = sum0, inc1 = sum1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t a = __shfl_up_sync(0xffffffffu, inc0, o), b = __shfl_up_sync(0xffffffffu, inc1, o);
        if (lane >= static_cast<uint32_t>(o)) {
            inc0 += a;
            inc1 += b;
        }
    }
    if (lane == 31) {
        s_total[0][warp] = inc0;
        s_total[1][warp] = inc1;
    }
    __syncthreads();
    uint32_t ex0 = inc0 - sum0, ex1 = inc1 - sum1, all0 = 0, all1 = 0;
#pragma unroll
    for (uint32_t w = 0; w < kBlockSortWarps; ++w) {
        const uint32_t a = s_total[0][w], b = s_total[1][w];
        if (w < warp) {
            ex0 += a;
            ex1 += b;
        }
        all0 += a;
        all1 += b;
    }
    for (uint32_t j = 0; j < per; ++j) {
        const uint32_t e = threadIdx.x * per + j;
        if (e >= experts)
            break;
        const uint32_t n = count[j], tiles = (n + tile_rows - 1) / tile_rows;
        const uint32_t start = ex0 & 0xffffu, tile0 = ex0 >> 16, pad = tile0 * tile_rows;
        rt.indptr[e] = s.start[e] = static_cast<int32_t>(start);
        rt.pad_indptr[e] = s.pad[e] = static_cast<int32_t>(pad);
        for (uint32_t m = 0; m < tiles; ++m) {
            rt.tile_expert[tile0 + m] = static_cast<int32_t>(e);
            rt.tile_row0[tile0 + m] = static_cast<int32_t>(pad + m * tile_rows);
            rt.tile_nrows[tile0 + m] = static_cast<int32_t>(min(tile_rows, n - m * tile_rows));
        }
        if (pairing) {
            for (uint32_t m = 0; m < tiles >> 1; ++m) {
                const uint32_t at = (ex1 >> 16) + m;
                rt.pair_expert[at] = static_cast<int32_t>(e);
                rt.pair_row0[at] = static_cast<int32_t>(pad + m * 2 * tile_rows);
                rt.pair_nrows[at] = static_cast<int32_t>(min(2 * tile_rows, n - m * 2 * tile_rows));
            }
            if (tiles & 1) {
                const uint32_t at = rt.max_tiles - 1 - (ex1 & 0xffffu);
                rt.pair_expert[at] = static_cast<int32_t>(e);
                rt.pair_row0[at] = static_cast<int32_t>(pad + (tiles - 1) * tile_rows);
                rt.pair_nrows[at] = static_cast<int32_t>(n - (tiles - 1) * tile_rows);
            }
            ex1 += (tiles >> 1) << 16 | (tiles & 1);
        }
        ex0 += tiles << 16 | n;
    }
    append_shared_tiles(rt, experts, all0 >> 16);
    if (threadIdx.x == 0) {
        rt.indptr[experts] = static_cast<int32_t>(all0 & 0xffffu);
        rt.pad_indptr[experts] = static_cast<int32_t>((all0 >> 16) * tile_rows);
        *rt.total_tiles = static_cast<int32_t>((all0 >> 16) + (rt.shared_rows + tile_rows - 1) / tile_rows);
        if (rt.pair_counts != nullptr) {
            rt.pair_counts[0] = static_cast<int32_t>(all1 >> 16);
            rt.pair_counts[1] = static_cast<int32_t>(all1 & 0xffffu);
        }
    }
    __syncthreads();
    for (uint32_t r = 0; r < rounds; ++r) {
        const uint32_t route = base + r * 32 + lane;
        const int e = route < routes ? s.ids[route] : -1;
        const uint32_t peers = __match_any_sync(0xffffffffu, e);
        int off = 0;
        if (e >= 0)
            off = mine[e] + __popc(peers & ((1u << lane) - 1u));
        __syncwarp();
        if (e >= 0 && lane == static_cast<uint32_t>(__ffs(static_cast<int>(peers)) - 1))
            mine[e] += static_cast<uint16_t>(__popc(peers));
        __syncwarp();
        if (route < routes) {
            if (e >= 0) {
                const int row = s.start[e] + off;
                rt.route_rows[route] = row;
                rt.route_prows[route] = s.pad[e] + off;
                rt.row_tokens[row] = static_cast<int32_t>(route / top_k);
                rt.row_scales[row] = weights[route];
            } else {
                rt.route_rows[route] = -1;
                rt.route_prows[route] = -1;
            }
        }
    }
}

} // namespace qs3
