// Router: logits in the declared dot order, score transform, k-pass top-k selection and weights.
//
// Contracts: strix::ds41::reference_router's product order (src/ds41_moe.cpp:72-82), the score transforms and the
// selection / weight rule of the shared route policy (include/strix/moe/route_policy.hpp:80-156). Expert ids are only
// reproducible when the choice values are bit-identical, so the logits keep the declared order: lane class l sums
// elements l, l + 32, ... ascending with separate multiply and add, then the butterfly d = 16 .. 1.
//
// HBM: the logits kernel streams the FP32 router matrix once per RT-row tile ([experts][hidden] * 4 B); the select
// kernel touches rows * experts * 4 B. Both are small beside the expert weights.
#include "declared_math.cuh"
#include "grouped_common.cuh"
#include "kernels.cuh"

namespace b200moe {
namespace {

// One warp computes an RT x ET tile of logits over the whole hidden width; lane = lane class.
template <int RT, int ET>
__global__ void __launch_bounds__(128) router_logits_kernel(const float* x, u32 x_stride, u32 rows, u32 hidden,
                                                            const float* w, u32 experts,
                                                            const float* logit_bias, float* logits) {
    chain_begin();
    const u32 lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const u32 e0 = (blockIdx.x * 4u + warp) * ET, r0 = blockIdx.y * RT;
    if (e0 >= experts) return;
    float acc[RT][ET];
#pragma unroll
    for (int r = 0; r < RT; ++r)
#pragma unroll
        for (int e = 0; e < ET; ++e) acc[r][e] = 0.0f;
    const float* xr[RT];
    const float* wr[ET];
#pragma unroll
    for (int r = 0; r < RT; ++r) xr[r] = x + u64(min(r0 + r, rows - 1)) * x_stride;
#pragma unroll
    for (int e = 0; e < ET; ++e) wr[e] = w + u64(min(e0 + e, experts - 1)) * hidden;
#pragma unroll 4
    for (u32 i = lane; i < hidden; i += 32) {
        float xv[RT], wv[ET];
#pragma unroll
        for (int r = 0; r < RT; ++r) xv[r] = xr[r][i];
#pragma unroll
        for (int e = 0; e < ET; ++e) wv[e] = load(wr[e] + i);
#pragma unroll
        for (int r = 0; r < RT; ++r)
#pragma unroll
            for (int e = 0; e < ET; ++e) acc[r][e] = __fadd_rn(acc[r][e], __fmul_rn(wv[e], xv[r]));
    }
#pragma unroll
    for (int r = 0; r < RT; ++r)
#pragma unroll
        for (int e = 0; e < ET; ++e) {
            float z = butterfly32(acc[r][e]);
            if (lane == 0 && r0 + r < rows && e0 + e < experts) {
                if (logit_bias) z = __fadd_rn(z, logit_bias[e0 + e]);
                logits[u64(r0 + r) * experts + e0 + e] = z;
            }
        }
}

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(static_cast<u32>(__cvta_generic_to_shared(dst))), "l"(src) : "memory");
}

// Windows of up to 4 rows: a warp is one expert and its CTA stages that expert's row (and the window's rows) in runs of 2048
// columns, every request of a run in flight at once. Bound by latency: the form above keeps four columns a warp in flight
// (4 rows x 128 experts x 2560: 20.9 us, 6.8 us here; 16 columns in flight by unrolling took 34.6, on cold instruction caches).
// Two experts a CTA spread a window over as many SMs as it has.
constexpr u32 kFewRun = 2048, kFewWarps = 2;
template <int RT>
__global__ void __launch_bounds__(kFewWarps * 32) router_logits_few_kernel(const float* x, u32 x_stride, u32 rows, u32 hidden, const float* w,
                                                                          u32 experts, const float* logit_bias, float* logits) {
    chain_begin();
    extern __shared__ __align__(16) float few_smem[];  // [RT rows | kFewWarps experts][kFewRun]
    const u32 tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, e0 = blockIdx.x * kFewWarps, e = e0 + warp;
    float acc[RT];
#pragma unroll
    for (int r = 0; r < RT; ++r) acc[r] = 0.0f;
    for (u32 c0 = 0; c0 < hidden; c0 += kFewRun) {
        const u32 n = min(kFewRun, hidden - c0);
        __syncthreads();  // the previous run has been consumed
        for (u32 j = 0; j < RT + kFewWarps; ++j) {
            const float* src = (j < RT ? x + u64(min(j, rows - 1)) * x_stride : w + u64(min(e0 + j - RT, experts - 1)) * hidden) + c0;
            for (u32 i = tid; i < n / 4; i += kFewWarps * 32) cp_async16(few_smem + j * kFewRun + 4 * i, src + 4 * i);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        const float* ws = few_smem + (RT + warp) * kFewRun;
#pragma unroll 8
        for (u32 i = lane; i < n; i += 32) {  // the lane class in ascending order (src/ds41_moe.cpp:72-82)
            const float wv = ws[i];
#pragma unroll
            for (int r = 0; r < RT; ++r) acc[r] = __fadd_rn(acc[r], __fmul_rn(wv, few_smem[r * kFewRun + i]));
        }
    }
#pragma unroll
    for (int r = 0; r < RT; ++r) {
        float z = butterfly32(acc[r]);
        if (lane == 0 && r < rows && e < experts) {
            if (logit_bias) z = __fadd_rn(z, logit_bias[e]);
            logits[u64(r) * experts + e] = z;
        }
    }
}

// Windows of more than 4 rows: a CTA owns 8 rows x 16 experts and walks the hidden width in chunks of COLS columns that
// all 128 threads stage into shared memory with 16-byte asynchronous copies, three chunks in flight; a warp keeps an
// 8 x 4 tile of lane-class sums. Chunks of 256 columns leave room for three CTAs an SM, of 512 for one: with more tiles than SMs the
// former hide each other's latency (8192 x 256 x 7168: 2309 us with 512, 1442 with 256, 1271 with two rows a packed instruction too; two FP32
// operations a product bound it at 835), a window with fewer tiles is a chain of chunks and wants the longer ones (64 x 256 x 7168: 23 against 33 us). The x tile
// is then read from HBM / L2 once per 16 experts instead of once per expert (a
// 64-row window over 256 experts of width 7168 pulled 470 MB through L2 in the form above), and the copies of two chunks
// cover the arithmetic of one. Same products, same order: lane l of a warp meets columns l, l + 32, ... ascending.
constexpr u32 kTileRows = 8, kTileExperts = 16, kTileStages = 3;
constexpr u32 tile_smem_bytes(u32 cols) { return kTileStages * (kTileRows + kTileExperts) * cols * 4u; }

template <u32 kTileCols>
__global__ void __launch_bounds__(128) router_logits_tile_kernel(const float* x, u32 x_stride, u32 rows, u32 hidden,
                                                                 const float* w, u32 experts,
                                                                 const float* logit_bias, float* logits) {
    chain_begin();
    extern __shared__ __align__(16) float tile_smem[];
    const u32 tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    constexpr u32 ET = kTileExperts / 4, kTileStageFloats = (kTileRows + kTileExperts) * kTileCols;
    const u32 r0 = blockIdx.y * kTileRows, e0 = blockIdx.x * kTileExperts;
    const u32 n_chunks = (hidden + kTileCols - 1) / kTileCols;
    auto issue = [&](u32 c) {
        if (c < n_chunks) {
            float* st = tile_smem + (c % kTileStages) * kTileStageFloats;
            const u32 col0 = c * kTileCols, nvec = (min(kTileCols, hidden - col0)) / 4;
            const u32 at = tid % (kTileCols / 4), j0 = tid / (kTileCols / 4);
            if (at < nvec) {
#pragma unroll
                for (u32 j = j0; j < kTileRows + kTileExperts; j += 512 / kTileCols) {
                    const float* src = j < kTileRows ? x + u64(min(r0 + j, rows - 1)) * x_stride : w + u64(min(e0 + j - kTileRows, experts - 1)) * hidden;
                    cp_async16(st + j * kTileCols + 4 * at, src + col0 + 4 * at);
                }
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");  // an empty group keeps the count of the wait below fixed
    };
    float2 acc[kTileRows / 2][ET];  // pairs of rows
#pragma unroll
    for (int r = 0; r < (int)kTileRows / 2; ++r)
#pragma unroll
        for (int e = 0; e < (int)ET; ++e) acc[r][e] = make_float2(0.0f, 0.0f);
    issue(0);
    issue(1);
    for (u32 c = 0; c < n_chunks; ++c) {
        issue(c + 2);
        asm volatile("cp.async.wait_group 2;" ::: "memory");
        __syncthreads();
        const float* st = tile_smem + (c % kTileStages) * kTileStageFloats;
        const u32 ncol = min(kTileCols, hidden - c * kTileCols);
#pragma unroll 4
        for (u32 col = lane; col < ncol; col += 32) {
            float2 xv[kTileRows / 2];
            float wv[ET];
#pragma unroll
            for (int r = 0; r < (int)kTileRows / 2; ++r) xv[r] = make_float2(st[2 * r * kTileCols + col], st[(2 * r + 1) * kTileCols + col]);
#pragma unroll
            for (int e = 0; e < (int)ET; ++e) wv[e] = st[(kTileRows + ET * warp + e) * kTileCols + col];
#pragma unroll
            for (int r = 0; r < (int)kTileRows / 2; ++r)
#pragma unroll
                for (int e = 0; e < (int)ET; ++e) {
                    if (kTileCols == 256) acc[r][e] = grouped::add2(grouped::mul2(grouped::both(wv[e]), xv[r]), acc[r][e]);
                    else acc[r][e] = make_float2(__fadd_rn(acc[r][e].x, __fmul_rn(wv[e], xv[r].x)), __fadd_rn(acc[r][e].y, __fmul_rn(wv[e], xv[r].y)));
                }
        }
        __syncthreads();  // the stage is refilled by the copies issued two iterations on
    }
#pragma unroll
    for (int r = 0; r < (int)kTileRows; ++r)
#pragma unroll
        for (int e = 0; e < (int)ET; ++e) {
            float z = butterfly32(r & 1 ? acc[r / 2][e].y : acc[r / 2][e].x);
            const u32 row = r0 + r, ex = e0 + ET * warp + e;
            if (lane == 0 && row < rows && ex < experts) {
                if (logit_bias) z = __fadd_rn(z, logit_bias[ex]);
                logits[u64(row) * experts + ex] = z;
            }
        }
}

}  // namespace
}  // namespace b200moe

#include "router_select.cuh"

namespace b200moe {
namespace {

// One warp per row; shared memory per warp: scores[experts] + choice[experts] + 32 group scores.
__global__ void __launch_bounds__(128) router_select_kernel(const float* logits, float* scores_out, const float* bias,
                                                            b200moe_route_policy p, u32 rows, u32* ids,
                                                            float* weights) {
    chain_begin();
    extern __shared__ __align__(16) float smem[];
    const u32 lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const u32 row = blockIdx.x * 4u + warp;
    if (row >= rows) return;
    select_detail::select_row<1024>(logits, scores_out, bias, p, row, lane, smem + warp * select_detail::scratch_floats(p.experts), ids, weights);
}

}  // namespace

int launch_router_logits(const b200moe_router_view& v, cudaStream_t stream, const b200moe_quantize_a8_view* fused_quantize) {
    const u32 E = v.policy.experts, xs = v.x_stride ? v.x_stride : v.hidden;
    if (v.rows == 0) return B200MOE_OK;
    if (fused_quantize) if (int rc = launch_quantize_a8(*fused_quantize, stream)) return rc;
#define B200_LOGITS(RT, ET)                                                                                   \
    small_launch(router_logits_kernel<RT, ET>, dim3((E + 4 * ET - 1) / (4 * ET), (v.rows + RT - 1) / RT), 128, 0, stream, v.x, xs, v.rows, v.hidden, v.weight, E, v.logit_bias, v.logits)
    const bool vec = aligned(v.x, 16) && aligned(v.weight, 16) && xs % 4 == 0 && v.hidden % 4 == 0;  // whole 16-byte units for the staged forms
#define B200_FEW(RT)                                                                                                                  \
    {                                                                                                                                 \
        constexpr u32 smem = (RT + kFewWarps) * kFewRun * sizeof(float);                                                              \
        if (int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(router_logits_few_kernel<RT>), smem)) return rc;               \
        small_launch(router_logits_few_kernel<RT>, (E + kFewWarps - 1) / kFewWarps, kFewWarps * 32, smem, stream, v.x, xs, v.rows, v.hidden, v.weight, E, v.logit_bias, v.logits); \
    }
#define B200_TILE(COLS)                                                                                                               \
    {                                                                                                                                 \
        if (int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(router_logits_tile_kernel<COLS>), tile_smem_bytes(COLS))) return rc; \
        small_launch(router_logits_tile_kernel<COLS>, grid, 128, tile_smem_bytes(COLS), stream, v.x, xs, v.rows, v.hidden, v.weight, E, v.logit_bias, v.logits); \
    }
    if (v.rows <= 4 && vec) {
        if (v.rows == 1) B200_FEW(1)
        else if (v.rows == 2) B200_FEW(2)
        else B200_FEW(4)
    } else if (v.rows == 1) B200_LOGITS(1, 1);
    else if (v.rows == 2) B200_LOGITS(2, 1);
    else if (v.rows <= 4) B200_LOGITS(4, 1);
    else if (vec) {
        const dim3 grid((E + kTileExperts - 1) / kTileExperts, (v.rows + kTileRows - 1) / kTileRows);
        if (u64(grid.x) * grid.y > static_cast<u32>(device_sm_count())) B200_TILE(256)
        else B200_TILE(512)
    } else if (v.rows <= 16) B200_LOGITS(8, 1);
    else B200_LOGITS(8, 4);
#undef B200_FEW
#undef B200_TILE
#undef B200_LOGITS
    return after_launch("router_logits");
}

int launch_router_select(const b200moe_router_view& v, cudaStream_t stream) {
    if (v.rows == 0) return B200MOE_OK;
    const u32 smem = 4u * select_detail::scratch_floats(v.policy.experts) * sizeof(float);
    small_launch(router_select_kernel, (v.rows + 3) / 4, 128, smem, stream, v.logits, v.scores, v.bias, v.policy, v.rows, v.ids, v.weights);
    return after_launch("router_select");
}

}  // namespace b200moe
