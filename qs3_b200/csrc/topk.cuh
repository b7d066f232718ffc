// Top-k of one token's router scores by one warp (router.cu, and fused with the sort of a small batch in routing.cu).
#pragma once

#include "common.cuh"

namespace qs3 {

constexpr float kRouterNegInf = -3.4028234663852886e38f; // upstream qscu.cu:31

// Order-preserving map float -> u32 for the values upstream's insertion accepts
// (score >= -FLT_MAX, not NaN); everything else maps to 0 and never wins. -0 is folded
// into +0 so that equal floats give equal keys.
__device__ __forceinline__ uint32_t score_key(float s)
{
    if (!(s >= kRouterNegInf))
        return 0u;
    const uint32_t b = __float_as_uint(s + 0.0f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

__device__ __forceinline__ float key_score(uint32_t k)
{
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

// Same routing as router_topk_kernel for num_experts <= 32 * ITEMS, with the token's
// scores held in registers (lane owns experts lane, lane + 32, ...). A round is a
// register arg-max per lane, one redux.sync max over the keys and one redux.sync min
// over the candidate ids (ties go to the lowest id, as upstream's insertion does).
// Called by a whole warp for one token; `s_cand` is 64 words of shared memory of the warp. Lane p returns slot p.
template <typename LogitT, int ITEMS>
__device__ __forceinline__ void topk_row(const LogitT* __restrict__ row, const float* __restrict__ bias,
                                         uint32_t num_experts, uint32_t top_k, int sigmoid_score, int renormalize,
                                         float scaling, uint32_t* s_cand, int* id_out, float* weight_out)
{
    const uint32_t lane = threadIdx.x & 31;
    float val[ITEMS];
    uint32_t key[ITEMS];
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
        const uint32_t e = lane + 32u * j;
        float l = __uint_as_float(0x7fc00000u); // padding: NaN, never selected, skipped below
        if (e < num_experts) {
            if constexpr (sizeof(LogitT) == 2)
                l = __bfloat162float(row[e]);
            else
                l = row[e];
            if (bias != nullptr)
                l += bias[e];
        }
        val[j] = l;
    }
    uint32_t kmax = 0;
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
        key[j] = score_key(val[j]);
        kmax = max(kmax, key[j]);
    }
    kmax = __reduce_max_sync(0xffffffffu, kmax);
    const float vmax = kmax != 0u ? key_score(kmax) : kRouterNegInf;

    float denom = 0.0f;
    if (!sigmoid_score) {
#pragma unroll
        for (int j = 0; j < ITEMS; ++j)
            if (lane + 32u * j < num_experts)
                denom += expf(val[j] - vmax);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            denom += __shfl_xor_sync(0xffffffffu, denom, o);
    } else {
#pragma unroll
        for (int j = 0; j < ITEMS; ++j)
            key[j] = lane + 32u * j < num_experts ? score_key(sigmoid_fast(val[j])) : 0u;
    }

    float my_weight = 0.0f;
    int my_id = 0;

    // Fast path. The arg-max rounds below cost ~3 * ITEMS integer instructions each, and the integer pipe,
    // not memory, bounds this kernel (ncu: 1800 instructions per token, ALU pipe 70 % busy). Most of that
    // work is spent on keys that cannot win: tau, the top_k-th largest of the 32 lane maxima, is a lower
    // bound of the top_k-th largest key (top_k different lanes hold a key >= tau), so every winner is
    // among the keys >= tau. Those are usually a dozen or two; they are compacted to one per lane and the
    // rounds run on them. Ties keep upstream's rule (equal keys: lowest id), because all keys equal to
    // the boundary value are candidates too. Falls back to the full rounds when fewer than top_k lanes
    // hold a valid key (tau == 0) or more than 32 keys reach tau. Both the lane maxima and the candidates are
    // ranked by counting the better ones (independent shuffles) instead of arg-max rounds, whose chain of
    // reductions decided the latency of a decode batch (1 token 0.0045 -> 0.0039 ms).
    bool fast = top_k <= 32;
    uint32_t tau = 0;
    if (fast) {
        uint32_t t = 0;
#pragma unroll
        for (int j = 0; j < ITEMS; ++j)
            t = max(t, key[j]);
        uint32_t rank = 0;
#pragma unroll
        for (uint32_t i = 0; i < 32; ++i) {
            const uint32_t o = __shfl_sync(0xffffffffu, t, i);
            rank += (o > t || (o == t && i < lane)) ? 1u : 0u; // equal maxima count once each
        }
        const uint32_t holder = __ballot_sync(0xffffffffu, rank == top_k - 1);
        tau = __shfl_sync(0xffffffffu, t, __ffs(static_cast<int>(holder)) - 1);
        fast = tau != 0u;
    }
    if (fast) {
        uint32_t cnt = 0;
#pragma unroll
        for (int j = 0; j < ITEMS; ++j)
            cnt += key[j] >= tau ? 1u : 0u;
        uint32_t incl = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= static_cast<uint32_t>(o))
                incl += v;
        }
        const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
        fast = total <= 32u;
        if (fast) {
            uint32_t at = incl - cnt;
#pragma unroll
            for (int j = 0; j < ITEMS; ++j)
                if (key[j] >= tau) {
                    s_cand[at] = key[j];
                    s_cand[32 + at] = lane + 32u * static_cast<uint32_t>(j);
                    ++at;
                }
            __syncwarp();
            const uint32_t ck = lane < total ? s_cand[lane] : 0u;
            const uint32_t cid = lane < total ? s_cand[32 + lane] : 0xffffffffu;
            uint32_t rank = 0;
            for (uint32_t i = 0; i < total; ++i) {
                const uint32_t ok = __shfl_sync(0xffffffffu, ck, i), oid = __shfl_sync(0xffffffffu, cid, i);
                rank += (ok > ck || (ok == ck && oid < cid)) ? 1u : 0u;
            }
            __syncwarp();
            if (lane < total && rank < top_k) { // total >= top_k: every slot is filled
                s_cand[rank] = ck;
                s_cand[32 + rank] = cid;
            }
            __syncwarp();
            if (lane < top_k) {
                const float sc = key_score(s_cand[lane]);
                my_id = static_cast<int>(s_cand[32 + lane]);
                my_weight = sigmoid_score ? sc : (denom > 0.0f ? expf(sc - vmax) / denom : 0.0f);
            }
        }
    }
    for (uint32_t pos = 0; !fast && pos < top_k; ++pos) {
        uint32_t best = 0;
        int bj = 0;
#pragma unroll
        for (int j = 0; j < ITEMS; ++j)
            if (key[j] > best) { // strict: the lowest id of equal keys stays
                best = key[j];
                bj = j;
            }
        const uint32_t top = __reduce_max_sync(0xffffffffu, best);
        float w = 0.0f;
        int id = static_cast<int>(pos); // unfilled slot (qscu.cu:945-949)
        if (top != 0u) {
            const uint32_t cand = best == top ? lane + 32u * static_cast<uint32_t>(bj) : 0xffffffffu;
            const uint32_t win = __reduce_min_sync(0xffffffffu, cand);
            id = static_cast<int>(win);
            const float s = key_score(top);
            w = sigmoid_score ? s : (denom > 0.0f ? expf(s - vmax) / denom : 0.0f);
            if (cand == win) {
#pragma unroll
                for (int j = 0; j < ITEMS; ++j)
                    if (j == bj)
                        key[j] = 0u;
            }
        }
        if (lane == pos) {
            my_weight = w;
            my_id = id;
        }
    }

    float sum = 0.0f;
    for (uint32_t pos = 0; pos < top_k; ++pos)
        sum += __shfl_sync(0xffffffffu, my_weight, pos);
    const float renorm = renormalize ? 1.0f / fmaxf(sum, 1.0e-20f) : 1.0f;
    *id_out = my_id;
    *weight_out = my_weight * renorm * scaling;
    __syncwarp(); // s_cand may be reused
}

} // namespace qs3
