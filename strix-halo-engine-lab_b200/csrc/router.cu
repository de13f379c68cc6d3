// Router: logits in the declared dot order, score transform, k-pass top-k selection and weights.
//
// Contracts: strix::ds41::reference_router's product order (src/ds41_moe.cpp:72-82), the score transforms and the
// selection / weight rule of the shared route policy (include/strix/moe/route_policy.hpp:80-156). Expert ids are only
// reproducible when the choice values are bit-identical, so the logits keep the declared order: lane class l sums
// elements l, l + 32, ... ascending with separate multiply and add, then the butterfly d = 16 .. 1.
//
// HBM: the logits kernel streams the FP32 router matrix once per RT-row tile ([experts][hidden] * 4 B); the select
// kernel touches rows * experts * 4 B. Both are small beside the expert weights.
#include <algorithm>

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

// Windows of more than 4 rows: a CTA owns 8 WR rows x 4 ET experts and walks the hidden width in chunks of COLS columns that
// all its threads stage into shared memory with 16-byte asynchronous copies, three chunks in flight; a warp keeps an
// 8 x ET tile of lane-class sums. Same products, same order: lane l of a warp meets columns l, l + 32, ... ascending. Three sizes of it:
//  * 512 columns, 8 x 16: windows with no more tiles than multiprocessors, a chain of chunks (64 x 256 x 7168: 21 us, 33 with 256 columns).
//  * 256 columns, 8 x 16: room for three CTAs a multiprocessor, which hide each other's latency, and two rows a packed instruction.
//  * 128 columns, 16 x 32: two CTAs of eight warps, a warp 8 x 8. A column costs a warp 16 reads of shared memory for 64 products where the form above reads
//    12 for 32, and a row of x comes out of L2 half as often. 8192 x 256 x 7168 1243 -> 1108 us, 4096 x 128 x 2048 101 -> 89; two FP32 operations a
//    product bound them at 835 and 60. With few waves of its larger tiles it is no better: 1500 x 128 x 2560 50.9 and 50.0, 2048 x 128 x 2048 52.5
//    and 52.6, 1024 x 256 x 7168 169.7 and 171.9.
// A tile's end: the sums of 32 cells meet at once (butterfly32_all); cell by cell they took 160 exchanges instead of 31 (8 x 128 x 2048 8.2 -> 7.0 us,
// 4096 x 128 x 2048 109 -> 101).
constexpr u32 kTileStages = 3;
template <u32 WR, u32 ET>
struct LogitsTile {
    static constexpr u32 rows = 8 * WR, experts = 4 * ET, threads = 128 * WR;
    static constexpr u32 smem_bytes(u32 cols) { return kTileStages * (rows + experts) * cols * 4u; }
};

// butterfly32 of 32 values at once: each step hands half of what is left to the lane's partner, so that 31 exchanges do for 160. Lane l ends with value l.
__device__ __forceinline__ float butterfly32_all(float (&v)[32], u32 lane) {
#pragma unroll
    for (u32 d = 16; d; d >>= 1)
#pragma unroll
        for (u32 i = 0; i < d; ++i) {
            const bool up = lane & d;
            const float theirs = __shfl_xor_sync(0xffffffffu, up ? v[i] : v[i + d], d);
            v[i] = __fadd_rn(up ? v[i + d] : v[i], theirs);
        }
    return v[0];
}

template <u32 kTileCols, u32 WR, u32 ET>
__global__ void __launch_bounds__(128 * WR) router_logits_tile_kernel(const float* x, u32 x_stride, u32 rows, u32 hidden,
                                                                 const float* w, u32 experts,
                                                                 const float* logit_bias, float* logits) {
    chain_begin();
    extern __shared__ __align__(16) float tile_smem[];
    const u32 tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    constexpr u32 kTileRows = LogitsTile<WR, ET>::rows, kTileExperts = LogitsTile<WR, ET>::experts, kTileStageFloats = (kTileRows + kTileExperts) * kTileCols;
    const u32 wr = 8u * (warp >> 2), we = ET * (warp & 3u);  // the warp's first row and expert of the tile
    const u32 r0 = blockIdx.y * kTileRows, e0 = blockIdx.x * kTileExperts;
    const u32 n_chunks = (hidden + kTileCols - 1) / kTileCols;
    auto issue = [&](u32 c) {
        if (c < n_chunks) {
            float* st = tile_smem + (c % kTileStages) * kTileStageFloats;
            const u32 col0 = c * kTileCols, nvec = (min(kTileCols, hidden - col0)) / 4;
            const u32 at = tid % (kTileCols / 4), j0 = tid / (kTileCols / 4);
            if (at < nvec) {
#pragma unroll
                for (u32 j = j0; j < kTileRows + kTileExperts; j += 512 * WR / kTileCols) {
                    const float* src = j < kTileRows ? x + u64(min(r0 + j, rows - 1)) * x_stride : w + u64(min(e0 + j - kTileRows, experts - 1)) * hidden;
                    cp_async16(st + j * kTileCols + 4 * at, src + col0 + 4 * at);
                }
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");  // an empty group keeps the count of the wait below fixed
    };
    float2 acc[4][ET];  // pairs of rows
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int e = 0; e < (int)ET; ++e) acc[r][e] = make_float2(0.0f, 0.0f);
    issue(0);
    issue(1);
    for (u32 c = 0; c < n_chunks; ++c) {
        if (kTileCols == 512) {
            issue(c + 2);
            asm volatile("cp.async.wait_group 2;" ::: "memory");
            __syncthreads();
        } else {
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            __syncthreads();
            issue(c + 2);
        }
        const float* st = tile_smem + (c % kTileStages) * kTileStageFloats;
        const u32 ncol = min(kTileCols, hidden - c * kTileCols);
#pragma unroll 4
        for (u32 col = lane; col < ncol; col += 32) {
            float2 xv[4];
            float wv[ET];
#pragma unroll
            for (int r = 0; r < 4; ++r) xv[r] = make_float2(st[(wr + 2 * r) * kTileCols + col], st[(wr + 2 * r + 1) * kTileCols + col]);
#pragma unroll
            for (int e = 0; e < (int)ET; ++e) wv[e] = st[(kTileRows + we + e) * kTileCols + col];
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int e = 0; e < (int)ET; ++e) {
                    if (kTileCols <= 256) acc[r][e] = grouped::add2(grouped::mul2(grouped::both(wv[e]), xv[r]), acc[r][e]);
                    else acc[r][e] = make_float2(__fadd_rn(acc[r][e].x, __fmul_rn(wv[e], xv[r].x)), __fadd_rn(acc[r][e].y, __fmul_rn(wv[e], xv[r].y)));
                }
        }
        if (kTileCols == 512) __syncthreads();  // the stage is refilled by the copies issued two iterations on
    }
    constexpr u32 kSetRows = 32 / ET;  // 32 cells at a time
#pragma unroll
    for (u32 s = 0; s < 8 / kSetRows; ++s) {
        float v[32];
#pragma unroll
        for (u32 i = 0; i < 32; ++i) {
            const u32 r = kSetRows * s + i / ET;
            v[i] = r & 1u ? acc[r / 2][i % ET].y : acc[r / 2][i % ET].x;
        }
        float z = butterfly32_all(v, lane);
        const u32 row = r0 + wr + kSetRows * s + lane / ET, ex = e0 + we + lane % ET;
        if (row < rows && ex < experts) {
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

// One warp per row; shared memory per warp: scores[experts] + choice[experts] + 32 group scores. 32 experts a lane took 96 registers, five CTAs a multiprocessor: 3000 rows of 1024 a
// second wave, 32 us, 26 with six.
template <int EPL>
__global__ void __launch_bounds__(128, EPL == 32 ? 6 : 1) router_select_kernel(const float* logits, float* scores_out, const float* bias,
                                                            const __grid_constant__ b200moe_route_policy p, u32 rows, u32* ids,
                                                            float* weights) {
    chain_begin();
    extern __shared__ __align__(16) float smem[];
    const u32 lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const u32 row = blockIdx.x * 4u + warp;
    if (row >= rows) return;
    select_detail::select_row<EPL>(logits, scores_out, bias, p, row, lane, smem + warp * select_detail::scratch_floats(p.experts), ids, weights);
}

// One warp per row; shared memory per warp: scores[experts] + choice[experts] + 32 group scores.

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
#define B200_TILE(COLS, WR, ET)                                                                                                       \
    {                                                                                                                                 \
        using T = LogitsTile<WR, ET>;                                                                                                 \
        const auto kernel = router_logits_tile_kernel<COLS, WR, ET>;                                                                  \
        if (int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), T::smem_bytes(COLS))) return rc;                      \
        small_launch(kernel, dim3((E + T::experts - 1) / T::experts, (v.rows + T::rows - 1) / T::rows), T::threads, T::smem_bytes(COLS), stream, v.x, xs, v.rows, v.hidden, v.weight, E, v.logit_bias, v.logits); \
    }
    if (v.rows <= 4 && vec) {
        if (v.rows == 1) B200_FEW(1)
        else if (v.rows == 2) B200_FEW(2)
        else B200_FEW(4)
    } else if (v.rows == 1) B200_LOGITS(1, 1);
    else if (v.rows == 2) B200_LOGITS(2, 1);
    else if (v.rows <= 4) B200_LOGITS(4, 1);
    else if (vec) {
        // the figures are with the kernel
        auto tiles = [&](u32 rows, u32 experts) { return u64((v.rows + rows - 1) / rows) * ((E + experts - 1) / experts); };
        const u64 sms = static_cast<u32>(device_sm_count());
        if (tiles(LogitsTile<2, 8>::rows, LogitsTile<2, 8>::experts) >= 6 * sms) B200_TILE(128, 2, 8)
        else if (tiles(LogitsTile<1, 4>::rows, LogitsTile<1, 4>::experts) > sms) B200_TILE(256, 1, 4)
        else B200_TILE(512, 1, 4)
    } else if (v.rows <= 16) B200_LOGITS(8, 1);
    else B200_LOGITS(8, 4);
#undef B200_FEW
#undef B200_TILE
#undef B200_LOGITS
    return after_launch("router_logits");
}

int launch_router_select(const b200moe_router_view& v, cudaStream_t stream) {
    if (v.rows == 0) return B200MOE_OK;
    // A launch admitted early is placed wherever the one in front leaves room, by the dozen on the first multiprocessors that come free. So a CTA asks for its share of a
    // multiprocessor's shared memory, from seven CTAs for eight multiprocessors on (48 to 128 experts: from more than one each). Below 48 experts the logits in front leave
    // multiprocessors free that hold all of the CTAs, and it pays only from five a multiprocessor on. us, without and with: selection alone, 4096 rows of 128 8.4 and 6.3, of 256 13.1 and
    // 9.6; with logits over 512, 1400 rows of 160 22.6 and 18.1, 592 of 256 19.2 and 13.9, 1400 of 16 6.5 and 7.6.
    const u32 experts = v.policy.experts, ctas = (v.rows + 3) / 4, sms = static_cast<u32>(device_sm_count()), eighths = experts < 48u ? 40u : experts <= 128u ? 8u : 7u;
    const u32 share = u64(ctas) * 8u > u64(eighths) * sms ? 227u * 1024u / ((ctas + sms - 1) / sms) : 0u;
    const u32 scratch = 4u * select_detail::scratch_floats(experts) * sizeof(float), smem = std::max(scratch, share > 2048u ? std::min(share - 1024u, 100u * 1024u) & ~15u : 0u);
    // Groups that no row of takes the fast path (12, 20 or 48 experts, say) have a kernel of the general path alone: 64 rows, 96 experts in 8 groups 13.6 us, 15.9 with
    // that path called out of line, 384 experts 25.4 and 34.
    const auto kernel = !select_detail::fast_groups(v.policy) ? router_select_kernel<0> : experts <= 128u ? router_select_kernel<4> : experts <= 256u ? router_select_kernel<8> : router_select_kernel<32>;
    if (int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), smem)) return rc;
    small_launch(kernel, ctas, 128, smem, stream, v.logits, v.scores, v.bias, v.policy, v.rows, v.ids, v.weights);
    return after_launch("router_select");
}

}  // namespace b200moe
