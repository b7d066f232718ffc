// Internal declarations shared by the translation units of libqs3moe.so.
#pragma once

#include "../../include/qs3_moe.h"

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdarg>
#include <cstdint>
#include <cstdio>

// Context object behind the opaque qsfi_context handle. Field order follows
// upstream qsfi_internal.h:11-20 so that an object built against either
// definition reads the same device ordinal, stream and error record.
struct qsfi_context {
    int32_t device_ordinal;
    cudaStream_t stream;
    void* float_workspace;
    size_t float_workspace_bytes;
    size_t int_workspace_bytes;
    size_t host_int_workspace_bytes;
    uint64_t scratch_generation;
    qsfi_error_info last_error;
    // (after upstream's fields) Side streams of the whole-layer call, one for each stream that the context was on lately, latest
    // first: the token quantiser and the shared expert run there beside the router chain. Each context has its own, so that
    // calls of several contexts on one plan do not meet in an event; each stream has its own, so that a call on one neither
    // waits for what another stream has queued nor meets a capture that is open there.
    struct qs3_side_stream* side;
};

struct qs3_side_stream {
    int device;
    cudaStream_t beside; // of the context
    cudaStream_t stream;
    cudaEvent_t fork, quant, shared; // fork / join with the context's stream
    qs3_side_stream* next;
};

struct qsfi_moe_plan {
    qsfi_moe_plan_desc desc;
};

namespace qs3 {

constexpr size_t kWorkspaceAlign = 256;
constexpr int kTileM = 128; // rows of one tensor-core tile; expert segments are padded to it
constexpr uint32_t kSmCount = 148; // of the device, for rules that decide a workspace's layout: its size is asked for without one

// ---- error plumbing (upstream qsfi_context.cu:10-101) -------------------------
void clear_error(qsfi_error_info* err);
qsfi_status set_error(qsfi_context* ctx, qsfi_status status, qsfi_error_source source,
                      int32_t native_code, const char* fmt, ...);
qsfi_status set_invalid_arg(qsfi_context* ctx, const char* fmt, ...);
qsfi_status set_unsupported(qsfi_context* ctx, const char* fmt, ...);
qsfi_status set_cuda_error(qsfi_context* ctx, cudaError_t err, const char* op);
qsfi_status activate_context(qsfi_context* ctx);
qsfi_status status_from_cuda(cudaError_t err);

// The side stream beside the context's present stream, NULL when none can be had; given back with the context.
qs3_side_stream* side_stream(qsfi_context* ctx);

// SMs of the current device.
uint32_t device_sm_count();

// Device-side error word shared by the tensor-core kernels (one per device).
uint32_t* device_error_word();

#if QSFI_ENABLE_CHECKED_VALIDATION
// Checked builds only (upstream qsfi_native_common.h checked-validation flag): a device flag
// that validator kernels raise; `checked_flag_finish` copies it back (one stream sync) and
// returns true when it was raised. The flag lives in the library, nothing is allocated.
int* checked_flag_reset(cudaStream_t stream, cudaError_t* err);
bool checked_flag_finish(cudaStream_t stream, cudaError_t* err);
#endif

// Kernel-launch counter (all kernels of this library) and the optional per-stage
// event recorder behind qs3_moe_profile_begin / qs3_moe_profile_end.
void note_launch(uint32_t n = 1);
enum Stage {
    STAGE_END = 0, STAGE_ROUTER_GEMM = 1, STAGE_ROUTER_TOPK = 2, STAGE_ROUTE_SORT = 3,
    STAGE_GATHER = 4, STAGE_GATE_UP_GEMM = 5, STAGE_DOWN_GEMM = 6, STAGE_SHARED = 7, STAGE_COMBINE = 8
};
void stage_mark(cudaStream_t stream, int stage);
bool stage_recording();

inline size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

template <typename T> bool contiguous1(const T& t) { return t.stride[0] == 1; }
template <typename T> bool contiguous2(const T& t)
{
    return t.stride[1] == 1 && t.stride[0] == t.shape[1];
}
template <typename T> bool contiguous3(const T& t)
{
    return t.stride[2] == 1 && t.stride[1] == t.shape[2]
        && t.stride[0] == t.shape[1] * t.shape[2];
}

// ---- routing tables -------------------------------------------------------------
// Everything the routed path derives from topk_ids, laid out in the workspace.
struct RouteTables {
    int32_t* counts;       // [E] routes per local expert
    int32_t* indptr;       // [E+1] exclusive scan of counts
    int32_t* pad_indptr;   // [E+1] exclusive scan of counts rounded up to tile_rows
    int32_t* route_rows;   // [R] dense row of a route (-1: expert not local)
    int32_t* route_prows;  // [R] row in the padded layout (-1: expert not local)
    int32_t* row_tokens;   // [R] token of a dense row
    float* row_scales;     // [R] routing weight of a dense row
    int32_t* tile_expert;  // [max_tiles]
    int32_t* tile_row0;    // [max_tiles] first padded row of the tile
    int32_t* tile_nrows;   // [max_tiles] valid rows in the tile
    int32_t* total_tiles;  // [1]
    // Tables for either of two tile heights, chosen by the sort from the routes of each expert (NULL: `tile_rows` only):
    // *alt_total_tiles counts the tiles if they have alt_tile_rows rows, *total_tiles if they have tile_rows, and the other
    // one is 0, so that of two kernels launched one after the other one does the work.
    int32_t* alt_total_tiles; // [1]
    uint32_t alt_tile_rows, alt_max_tiles;
    // 256-row "pair tiles" for the CTA-pair GEMM (128-row plans only, NULL otherwise): an expert with t
    // row tiles gives t / 2 full pairs, listed from index 0 upwards, and t % 2 single (<= 128 rows),
    // listed from index max_tiles - 1 downwards; pair_counts = {full pairs, singles}
    int32_t* pair_expert;  // [max_tiles]
    int32_t* pair_row0;    // [max_tiles] first padded row
    int32_t* pair_nrows;   // [max_tiles] valid rows, 1..256
    int32_t* pair_counts;  // [2]
    int32_t* block_hist;   // [route_blocks * E] scratch of the counting sort
    uint32_t max_tiles;
    uint32_t max_pad_rows;
    uint32_t route_blocks;
    uint32_t tile_rows;    // rows of one tile: expert segments are padded to a multiple of it
    // > 0: a shared expert joins the grouped GEMMs as group number E. The sort appends tiles of these rows (all tokens,
    // in token order) after the experts' tiles; their padded rows start at pad_indptr[E].
    uint32_t shared_rows;
};

constexpr uint32_t kAltMaxRoutes = 80; // routes per expert up to which the sort chooses between tile heights
size_t route_tables_bytes(uint32_t routes, uint32_t experts);
// Carves the tables out of `base` (may be NULL for sizing); returns bytes used, never fewer for more routes.
size_t route_tables_carve(char* base, uint32_t routes, uint32_t experts, RouteTables* out,
                          uint32_t tile_rows = kTileM, uint32_t shared_rows = 0, uint32_t alt_tile_rows = 0);
// Tokens to quantise beside the sort: NVFP4, or FP8 with row-major scales.
struct TokenQuant {
    const __nv_bfloat16* x; // [rows, k]
    uint32_t rows, k;
    float global_scale;
    uint8_t* packed;
    uint8_t* scale_tiled;
    float* fp8_scale; // NULL: NVFP4
};
// Counting sort of the routes by local expert, stable in route index.
cudaError_t launch_route_sort(const int32_t* topk_ids, const float* topk_weights, uint32_t routes,
                              uint32_t top_k, uint32_t local_offset, uint32_t experts,
                              const RouteTables& rt, cudaStream_t stream, const TokenQuant* quant = nullptr);
// Router scores of a few tokens, for kernels that route them on the way.
struct RouterParams {
    const float* logits; // [num_tokens, num_experts]
    const float* bias;   // optional [num_experts]
    int32_t* ids;        // out [num_tokens, top_k]
    float* weights;
    uint32_t num_tokens, num_experts;
    int sigmoid_score, renormalize;
    float scaling;
};
// Top-k and sort of a small batch in one launch (f32 logits).
bool router_sort_supported(uint32_t num_tokens, uint32_t num_experts, uint32_t top_k, uint32_t experts);
cudaError_t launch_router_sort(const float* logits, const float* bias, int32_t* ids, float* weights, uint32_t num_tokens,
                               uint32_t num_experts, uint32_t top_k, int sigmoid_score, int renormalize, float scaling,
                               uint32_t local_offset, uint32_t experts, const RouteTables& rt, cudaStream_t stream,
                               const TokenQuant* quant);

// ---- router -----------------------------------------------------------------------
// `bias` (optional f32 [num_experts]) is added to the logits before scoring.
cudaError_t launch_router_topk(const void* logits, int logits_bf16, const float* bias,
                               int32_t* ids, float* weights, uint32_t num_tokens,
                               uint32_t num_experts, uint32_t top_k, int sigmoid_score,
                               int renormalize, float scaling, cudaStream_t stream);
qsfi_status validate_router_desc(const qscu_router_topk_desc* d);

// ---- permute / combine ----------------------------------------------------------
// dst[padded row] = src[token] for the rows of experts with more than `min_rows` rows (row_bytes a multiple of 16).
cudaError_t launch_gather_rows(const void* src, uint32_t row_bytes, const RouteTables& rt, uint32_t min_rows, void* dst,
                               cudaStream_t stream);
// The streaming kernels find an expert's token rows through the tables up to this many rows, and take more from a
// gathered copy. A gather4 load occupies the copy engine for about 80 cycles: twelve stay well below the 1400 cycles in
// which a stage's weights arrive from HBM, but the weights of an expert with several tiles come from L2, faster. bf16
// layer, 128 experts top-8, in place / line at 64 / at 48 rows: 1024 tokens 0.325 / 0.306 / 0.266 ms, 2048 tokens 0.510 /
// 0.335 / 0.335, 512 of a skewed router 0.213 / 0.190 / 0.178; all rows gathered: 512 experts top-10, 2048 tokens 0.630
// -> 0.659.
constexpr uint32_t kGatherRows = 48;
// Whether a batch may have such experts and is large enough to look: the pass costs a few microseconds.
inline bool gather_rows_pays(uint32_t num_tokens, uint32_t top_k, uint32_t experts)
{
    return num_tokens > kGatherRows && num_tokens * static_cast<uint64_t>(top_k) >= 8ull * experts;
}

struct CombineParams {
    const int32_t* route_prows;   // [T*K]
    const float* topk_weights;    // [T*K]
    const __nv_bfloat16* expert_out; // [pad_rows, H]
    __nv_bfloat16* out;           // [T, H]
    uint32_t num_tokens, top_k, hidden_size;
    // optional shared expert term: out += sigmoid(x . gate_w) * shared_out
    const __nv_bfloat16* shared_out; // [T, H] or NULL
    const int32_t* shared_row0;      // optional: row of token 0 in shared_out (NULL: 0)
    const __nv_bfloat16* hidden;     // [T, H] for the gate logit
    const __nv_bfloat16* gate_w;     // [H]
    int round_before_shared;         // 1: round the routed sum to bf16 first (upstream chain)
    int skip_empty;                  // 1: leave rows of tokens without any local route unwritten
    int early;                       // 1: the predecessor in the stream wrote nothing but expert_out and shared_out
    // optional post-MoE neighbours fused in (hidden_size <= 2048): residual += out (bf16, in
    // place) and out = rmsnorm(residual) * norm_weight, as qsfi_fused_add_rmsnorm would do
    __nv_bfloat16* residual;         // [T, H] or NULL
    const __nv_bfloat16* norm_weight; // [H]
    float norm_eps;
};

struct EpPullParams {
    const __nv_bfloat16* peer[32];   // every rank's partial-sum buffer [num_ranks * T, H] (peer-mapped)
    const int32_t* topk_ids;         // [T, K] this rank's routing (global expert ids)
    __nv_bfloat16* out;              // [T, H]
    const __nv_bfloat16* shared_out; // optional [T, H]
    const __nv_bfloat16* hidden;     // [T, H]
    const __nv_bfloat16* gate_w;     // [H]
    uint32_t num_tokens, top_k, hidden_size, num_ranks, my_rank, experts_per_rank;
    uint32_t dbg; // measurement only (QS3_EP_FINISH_DBG): 1 read the own rank's partial sums only
};
cudaError_t launch_ep_pull_combine(const EpPullParams& p, cudaStream_t stream);
struct EpPullTokensParams {
    const uint8_t* peer[32];    // every rank's symmetric token block (peer-mapped)
    uint64_t seg_offset[4];     // byte offset of segment j inside a token block
    uint64_t seg_bytes[4];      // bytes of segment j per rank (multiple of 16)
    uint8_t* dst[4];            // local buffer of segment j: [num_ranks, seg_bytes[j]]
    uint32_t num_ranks, num_segments;
};
cudaError_t launch_ep_pull_tokens(const EpPullTokensParams& p, cudaStream_t stream);
cudaError_t launch_combine(const CombineParams& p, cudaStream_t stream);
struct EpBarrierParams {
    uint32_t* pads[32];     // pads[r]: rank r's signal pad (num_ranks words) as mapped on this device
    uint32_t num_ranks, my_rank, epoch;
    uint32_t* epoch_counter; // optional: epoch = *counter + 1, stored back by the kernel
    uint64_t limit_cycles;
    uint32_t* err;
};
cudaError_t launch_ep_barrier(const EpBarrierParams& p, cudaStream_t stream);
cudaError_t launch_ep_route_targets(const int32_t* ids, const int32_t* map, uint32_t map_len, int32_t* out,
                                    uint32_t* mask, uint32_t tokens, uint32_t top_k, uint32_t per_rank,
                                    uint32_t ranks, cudaStream_t stream);
struct EpPullRoutedParams {
    const uint8_t* peer[32];   // every rank's peer-mapped token block
    uint64_t off_codes, off_scales, off_ids, off_wts, off_mask; // byte offsets of the segments in a block
    uint8_t *dst_codes, *dst_scales, *dst_ids, *dst_wts;        // local [num_ranks * num_tokens, ...] buffers
    uint32_t num_ranks, my_rank, num_tokens, top_k;
    uint32_t code_vecs, scale_vecs; // 16-byte vectors per row of codes (<= 64) / scales (<= 32)
};
cudaError_t launch_ep_pull_routed(const EpPullRoutedParams& p, cudaStream_t stream);
cudaError_t launch_ep_rank_routes(int32_t* rows, float* weights, uint32_t tokens, uint32_t ranks,
                                  cudaStream_t stream);

// ---- GEMMs ----------------------------------------------------------------------
enum GemmEpilogue {
    EPI_STORE_BF16 = 0,   // out = bf16(alpha * acc [+ beta * out])
    EPI_STORE_F32 = 1,    // out = alpha * acc [+ beta * out] [+ bias[n]]
    EPI_SWIGLU_BF16 = 2,  // out = bf16(silu(bf16(g)) * bf16(u))
    EPI_SWIGLU_NVFP4 = 3  // out = nvfp4(silu(g) * u), packed + tiled scales
};

struct GemmProblem {
    // A operand: [a_rows, k] row-major (bf16 elements or packed e2m1 bytes), pitch in BYTES
    const void* a;
    uint64_t a_rows;
    uint64_t a_pitch_bytes;
    const uint8_t* a_scale_tiled; // NVFP4 only
    // NVFP4 decode and bf16 streaming kernels: A rows still in token order (a_scale_linear: with row-major scales), found
    // through the routing tables; NULL: A rows are the padded rows
    const int32_t* row_tokens;
    const int32_t* indptr;
    const int32_t* pad_indptr;
    int a_scale_linear;
    const void* gathered; // bf16 streaming kernel, with row_tokens: padded-layout copy of the rows of experts with more
                          // than kGatherRows rows, or NULL
    int one_tile_per_cta; // bf16: not the streaming kernel
    int tables_ready; // NVFP4 decode and bf16 streaming kernels: the tile tables were complete before the predecessor in the stream started
    // decode kernel only: weights of a shared expert that is group number `groups` of the tile tables (NULL: none)
    const void* shared_b;
    const uint8_t* shared_b_scale_tiled;
    const float* shared_scale;    // optional f32 [1] multiplier, and that of the up rows
    const float* shared_scale_up;
    // B operand: [groups, b_rows, k]; b_rows = 2*n for gated problems
    const void* b;
    uint64_t b_pitch_bytes;
    const uint8_t* b_scale_tiled; // NVFP4 only, per group qs3_nvfp4_tiled_scale_bytes(b_rows, k)
    uint32_t groups;
    uint32_t n; // output features (gated: intermediate size)
    uint32_t k; // reduction length in elements
    int nvfp4;
    int gated;
    int epilogue;
    // tile tables (NULL: dense problem, tiles are consecutive 128-row blocks of A)
    const int32_t* tile_expert;
    const int32_t* tile_row0;
    const int32_t* tile_nrows;
    const int32_t* total_tiles;
    uint32_t max_tiles;
    uint32_t tile_rows;  // rows per tile of the tables: 128, or 32 / 64 (NVFP4 decode kernel, operands swapped)
    // pair tiles of the route sort (RouteTables::pair_*), NULL: no CTA-pair kernel for this problem
    const int32_t* pair_expert;
    const int32_t* pair_row0;
    const int32_t* pair_nrows;
    const int32_t* pair_counts;
    // output
    void* out;
    uint64_t out_pitch_elems;   // elements (bytes for packed NVFP4 output)
    uint8_t* out_scale_tiled;   // EPI_SWIGLU_NVFP4
    float alpha;                // 0 means 1
    float beta;
    const float* group_scale;   // optional per-group multiplier on acc
    const float* group_scale_up; // gated: optional multiplier of the up rows (NULL: group_scale)
    const float* bias;          // optional f32 [n] (EPI_STORE_F32)
    float out_global_scale;     // EPI_SWIGLU_NVFP4: global scale of the quantised output
};
// Chooses the tcgen05 kernel when the shape allows it and the plain CUDA-core
// kernel otherwise (tiny or unaligned shapes; bf16 only).
cudaError_t launch_gemm(const GemmProblem& p, cudaStream_t stream, const char** why_unsupported);
// Dense bf16 problems with few output tiles: k split over the CTAs of a cluster (gemm_splitk.cu).
bool gemm_splitk_supported(const GemmProblem& p);
// `rows` of A per tile, 0: this kernel's own choice.
cudaError_t launch_gemm_splitk(const GemmProblem& p, uint32_t rows, cudaStream_t stream, const char** why_unsupported);
float gemm_splitk_estimate(const GemmProblem& p, uint32_t rows, uint32_t sms); // microseconds, bf16 results
// Persistent 128 x 256 kernel for dense bf16 problems with more than 64 rows (gemm_dense.cu).
bool gemm_dense_bf16_supported(const GemmProblem& p);
enum DenseKernel : uint32_t { DENSE_ONE, DENSE_PAIR, DENSE_SPLIT };
struct DenseChoice {
    DenseKernel kernel;
    uint32_t width; // columns of a tile; DENSE_SPLIT: rows of A
};
DenseChoice gemm_dense_choice(const GemmProblem& p);
// DENSE_ONE and DENSE_PAIR
cudaError_t launch_gemm_dense_bf16(const GemmProblem& p, DenseChoice choice, cudaStream_t stream, const char** why_unsupported);
// NVFP4 GEMM on CTA pairs (256 x 256 instructions, weights cross L2 -> SM once per 256 rows; gemm_pair.cu).
bool nvfp4_pair_gemm_supported(const GemmProblem& p);
cudaError_t launch_nvfp4_pair_gemm(const GemmProblem& p, cudaStream_t stream, const char** why_unsupported);
// NVFP4 grouped GEMM for 32- and 64-row token tiles (few rows per expert): weights are the M side of the MMA.
cudaError_t launch_nvfp4_swap_gemm(const GemmProblem& p, cudaStream_t stream, const char** why_unsupported);
// Rows per token tile of an NVFP4 plan: 32 or 64 (decode kernel) when experts get few rows each, else 128.
uint32_t nvfp4_tile_rows(uint32_t routes, uint32_t experts, uint32_t hidden, uint32_t inter);
// Smaller tile height between which and 128 rows the sort chooses up to kAltMaxRoutes routes per expert, 0: none.
uint32_t nvfp4_alt_tile_rows(uint32_t routes, uint32_t experts, uint32_t hidden, uint32_t inter);
// Whether a sort of this size can choose between tile heights.
bool route_sort_can_choose(uint32_t routes, uint32_t experts);
bool gemm_tc_supported(const GemmProblem& p);
// bf16 grouped GEMM of the routed experts, weights streamed as the M side (bf16_stream.cu), and the rows per token
// tile of a bf16 plan.
bool bf16_stream_gemm_supported(const GemmProblem& p);
cudaError_t launch_bf16_stream_gemm(const GemmProblem& p, cudaStream_t stream, const char** why_unsupported);
uint32_t bf16_tile_rows(uint32_t routes, uint32_t experts, uint32_t hidden, uint32_t inter);
// Whether the grouped GEMMs of a bf16 plan run as one 128 x 128 tile per CTA (gemm_tc_kernel) on a gathered copy of all
// routed rows.
bool bf16_one_tile_per_cta(uint32_t routes, uint32_t experts, uint32_t hidden, uint32_t inter);

// ---- NVFP4 ----------------------------------------------------------------------
// Token rows in token order -> e2m1 codes and scales tiled by token row.
cudaError_t launch_nvfp4_quantize_rows(const __nv_bfloat16* x, uint32_t rows, uint32_t k, float global_scale,
                                       uint8_t* packed, uint8_t* scale_tiled, cudaStream_t stream);
// Gather of already-quantised token rows into the padded permuted layout of sorted routing tables with
// 128-row tiles, organised by destination tile (coalesced code rows, whole scale tiles; rows past a tile's last
// row keep stale codes and get zero scales). `src_scale_tiled`: the source scales are tiled by token row
// instead of row-major.
cudaError_t launch_nvfp4_gather_tiles(const uint8_t* hidden_packed, const uint8_t* hidden_scale, const RouteTables& rt,
                                      uint32_t hidden_size, uint8_t* packed, uint8_t* scale_tiled, cudaStream_t stream,
                                      int src_scale_tiled = 0);

// ---- FP8 (e4m3, 128 x 128 weight blocks, per-token 128-element activation groups) ----
// Rows of one token tile of the FP8 grouped GEMM for this many routes over this many experts.
uint32_t fp8_tile_rows(uint32_t routes, uint32_t experts);
// codes / scales = quantise(x) row by row (k a multiple of 128).
cudaError_t launch_fp8_quantize_rows(const __nv_bfloat16* x, uint32_t rows, uint32_t k, uint8_t* codes, float* scales,
                                     cudaStream_t stream);
cudaError_t launch_fp8_quantize_weight(const __nv_bfloat16* w, uint32_t experts, uint32_t rows, uint32_t k,
                                       uint8_t* codes, float* scales, cudaStream_t stream);
struct Fp8Gemm {
    const uint8_t* x;        // e4m3 [x_rows, k]: rows in the padded layout, or in token order with `row_tokens`
    const float* x_scale;    // [x_rows, k / 128]
    uint64_t x_rows;
    const int32_t* row_tokens; // NULL: x rows are the padded rows; else dense row -> x row (with the segment starts)
    const int32_t* indptr;
    const int32_t* pad_indptr;
    const uint8_t* gathered; // with row_tokens: padded-layout copy of the rows of experts with more than kGatherRows
                             // rows (128-row tiles: of all), or NULL
    const uint8_t* w;        // e4m3 [groups, gated ? 2n : n, k]
    const float* w_scale;    // [groups, ceil(rows / 128), k / 128]
    uint32_t groups, n, k;
    int gated;               // 1: out = quantise(silu(gate) * up) as e4m3 [x_rows, n] + out_scale
    const int32_t* tile_expert;
    const int32_t* tile_row0;
    const int32_t* tile_nrows;
    const int32_t* total_tiles;
    int tables_ready;        // the tables were complete before the predecessor in the stream started
    uint32_t max_tiles;
    uint32_t tile_rows;      // 64 (fp8_stream.cu) or 128 (token rows on the M side, fp8_rows.cu)
    uint64_t out_rows;       // padded rows
    void* out;               // gated: u8 [out_rows, n]; else bf16 [out_rows, n]
    float* out_scale;        // gated: f32 [out_rows, n / 128]
};
cudaError_t launch_fp8_gemm(const Fp8Gemm& g, cudaStream_t stream, const char** why_unsupported);
cudaError_t launch_fp8_stream_gemm(const Fp8Gemm& g, cudaStream_t stream, const char** why_unsupported);
cudaError_t launch_fp8_rows_gemm(const Fp8Gemm& g, cudaStream_t stream, const char** why_unsupported);

// ---- experts of a handful of tokens as matrix-vector products (gemv.cu) ----
enum GemvFormat { GEMV_BF16 = 0, GEMV_FP8 = 1, GEMV_NVFP4 = 2 };
struct GemvWeights { // of the routed experts, or of the shared one
    const uint8_t *gate_up, *down;               // [experts, 2 inter, hidden], [experts, hidden, inter]
    const void *gate_up_scale, *down_scale;      // NVFP4: tiled block scales; FP8: f32 block scales
    const float *gate_up_global, *gate_up_global_up, *down_global; // NVFP4, optional
};
struct GemvParams {
    const __nv_bfloat16* hidden;  // [tokens, hidden]
    const uint8_t* hidden_packed; // NVFP4: the tokens' codes, with scales tiled by token row (NULL: quantised here)
    const uint8_t* hidden_sf;
    const int32_t* ids;           // [tokens, top_k], given or written by the router of the same launch
    const float* weights;
    uint32_t num_tokens, hidden_size, inter, top_k, experts, local_offset;
    uint32_t shared;              // 1: a shared expert of the same intermediate size follows the routed slots
    int early;                    // the predecessor in the stream writes nothing but the logits
    GemvWeights routed, shared_weights;
    float act_global, act2_global;
    uint8_t* act;                 // [tokens * slots, inter]: bf16, f32 (FP8), e2m1 codes (NVFP4) with act_scale [.., inter / 16]
    uint8_t* act_scale;
    const __nv_bfloat16* shared_gate; // [hidden]
    __nv_bfloat16* out;           // [tokens, hidden]; or, with y2, the slots' rows, to be combined by a later launch:
    __nv_bfloat16* y2;            // row route_prows[route], the shared expert's in y2_shared at *shared_row0 (NULL: 0) + token
    __nv_bfloat16* y2_shared;
    const int32_t *route_prows, *shared_row0;
};
// Bytes of `act` for that many tokens.
inline size_t gemv_act_bytes(int fmt, size_t rows, size_t inter) { return rows * inter * (fmt == GEMV_BF16 ? 2 : fmt == GEMV_FP8 ? 4 : 1) / (fmt == GEMV_NVFP4 ? 2 : 1); }
// Whether such a call is taken. `num_experts`: of the router.
bool gemv_supported(int fmt, uint32_t num_tokens, uint32_t top_k, uint32_t num_experts, uint32_t experts, uint32_t hidden,
                    uint32_t inter, uint32_t shared_inter);
// `router`: routes the tokens first (NULL: ids and weights are given). Fills the tables of `rt` on the way.
cudaError_t launch_gemv(int fmt, const GemvParams& p, const RouterParams* router, const RouteTables& rt, cudaStream_t stream);

// ---- device helpers ---------------------------------------------------------------
#ifdef __CUDACC__
// Chained launches (programmatic dependent launch): a kernel launched by launch_chained may start while its
// predecessor in the stream still runs, so that launch latency, set-up and the fetch of its code overlap the
// predecessor's tail. The rules: every thread of such a kernel executes chain_begin() (or its two halves apart) before it touches
// global memory that a predecessor reads or writes, and before it exits; it first waits for the predecessor to complete, which has
// itself waited for its own, so at most two neighbouring kernels overlap and everything older is complete.
// A kernel that allocates tensor memory does so before it releases its successor: a successor that sits on the same SM
// allocates before it waits, and would hold the columns until the predecessor, which needs them, has completed.
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void chain_begin()
{
    chain_wait();
    chain_release();
}

// Work beside the main chain is launched unchained: a kernel that waits for its predecessor while it holds the shared
// memory and registers of its SMs keeps the small kernels of the other stream out.
extern thread_local bool launch_unchained;
struct UnchainedScope {
    const bool before = launch_unchained;
    explicit UnchainedScope(bool on = true) { launch_unchained = before || on; }
    ~UnchainedScope() { launch_unchained = before; }
};

template <typename... KArgs, typename... Args>
cudaError_t launch_chained_cluster(void (*kernel)(KArgs...), uint32_t cluster, dim3 grid, uint32_t block, size_t smem,
                                   cudaStream_t stream, Args&&... args)
{
    cudaLaunchConfig_t cfg {};
    cudaLaunchAttribute attr[2] = {};
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = launch_unchained ? 0 : 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim = { cluster, 1, 1 };
    cfg.gridDim = grid;
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = attr;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
    note_launch();
    return cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...);
}

template <typename... KArgs, typename... Args>
cudaError_t launch_chained(void (*kernel)(KArgs...), dim3 grid, uint32_t block, size_t smem, cudaStream_t stream,
                           Args&&... args)
{
    return launch_chained_cluster(kernel, 1, grid, block, smem, stream, args...);
}

__device__ __forceinline__ float bf16_bits_to_f32(uint32_t bits16)
{
    return __uint_as_float(bits16 << 16);
}
// upstream qscu.cu:253-256 / qsfi_moe.cu:461
__device__ __forceinline__ float sigmoid_fast(float v) { return 1.0f / (1.0f + __expf(-v)); }
#endif

} // namespace qs3
