// RMSNorm in front of the FFN, fused with the A8 quantiser of its output (the rows the router and the experts read).
// One CTA per row, several in short windows; 256 of a CTA's threads are the 256 lanes of the host rule, or 128 two each (src/cpu/core/reference.cpp:86-103): lane l runs
// a = fma(x[i], x[i], a) over i = l, l + L, ... (L = 128 below n = 512), the lanes fold by the halving tree, and
// s = 1 / sqrt(sum / n + eps) - IEEE division and square root. The second pass is warp-per-group: y = (x * s) * w for
// 32 consecutive values, written out and / or quantised by the A8 rule on the spot. HBM traffic: x once (the second
// pass hits L1 / L2), y and the A8 rows once.
#include <algorithm>

#include "kernels.cuh"

namespace b200moe {
namespace {

// One group of 32 values of a row's result, by a warp; whether the lane's value is finite.
__device__ __forceinline__ bool put_group(const b200moe_rmsnorm_view& v, u32 r, u32 g, u32 lane, float x, float weight, float s, u32 out_stride, u32 a8_stride) {
    const u32 i = 32u * g + lane;
    float y = __fmul_rn(x, s);
    if (v.weight) y = __fmul_rn(y, weight);
    if (v.out) v.out[u64(r) * out_stride + i] = y;
    if (v.a8.codes) {
        float delta;
        int sum;
        const int code = a8_quantize_lane(y, &delta, &sum);
        v.a8.codes[u64(r) * a8_stride + i] = static_cast<i8>(code);
        if (lane == 0) {
            v.a8.deltas[u64(r) * (a8_stride / 32) + g] = delta;
            if (v.a8.sums) v.a8.sums[u64(r) * (a8_stride / 32) + g] = sum;
        }
    }
    return finite_f(y);
}

// A row takes gridDim.y CTAs: each makes the whole sum (the row comes out of L2) and takes every gridDim.y-th set of a group a warp of the second pass, whose
// first values and weights are asked for with the row's. What bounds a short window is the chain of trips and of dependent instructions: asks for BATCH
// values a lane at once, adds zeros behind the row's end (fma(0, 0, a) is a), and every warp folds the lanes itself, in the tree's order, behind one barrier. One CTA a
// row that asked for eight values at once, folded by a barrier a level and asked for the weights behind the sum: 1 row of 2560 4.9 us, 2.1 now; of 7168 10.1 and 2.4.
template <u32 THREADS, u32 BATCH, bool CHAIN>
__global__ void __launch_bounds__(THREADS) rmsnorm_a8_kernel(b200moe_rmsnorm_view v) {
    chain_begin_if<CHAIN>();
    constexpr u32 kWarps = THREADS / 32u;
    __shared__ float partial[256];
    const u32 r = blockIdx.x, t = threadIdx.x, lane = t & 31u, n = v.n, groups = n / 32u;
    const u32 x_stride = v.x_stride ? v.x_stride : n, out_stride = v.out_stride ? v.out_stride : n, a8_stride = v.a8.stride ? v.a8.stride : v.a8.width;
    const float* x = v.x + u64(r) * x_stride;
    const u32 lanes = n >= 512u ? 256u : 128u;
    u32 g = kWarps * blockIdx.y + (t >> 5);
    float mine = 0.0f, weight = 1.0f;
    if (g < groups) { mine = x[32u * g + lane]; if (v.weight) weight = v.weight[32u * g + lane]; }
    constexpr u32 kHeld = THREADS < 256u ? 2u : 1u;  // lanes of the rule that a thread is
    float a[kHeld] = {};
    if (t < lanes) {
        for (u32 i0 = t; i0 < n; i0 += BATCH * lanes) {
            float xi[kHeld][BATCH];
#pragma unroll
            for (u32 k = 0; k < BATCH; ++k)
#pragma unroll
                for (u32 h = 0; h < kHeld; ++h) { const u32 i = i0 + k * lanes + 128u * h; xi[h][k] = i < n && (h == 0 || lanes == 256u) ? x[i] : 0.0f; }
#pragma unroll
            for (u32 k = 0; k < BATCH; ++k)
#pragma unroll
                for (u32 h = 0; h < kHeld; ++h) a[h] = __fmaf_rn(xi[h][k], xi[h][k], a[h]);
        }
        partial[t] = kHeld == 2u ? __fadd_rn(a[0], a[kHeld - 1u]) : a[0];  // the lane that is none has added nothing: + 0
    }
    __syncthreads();
    auto fold = [&]() {
        auto four = [&](u32 o, u32 d) { return __fadd_rn(__fadd_rn(partial[lane + o], partial[lane + o + 2u * d]), __fadd_rn(partial[lane + o + d], partial[lane + o + 3u * d])); };
        float p = kHeld == 1u && lanes == 256u ? __fadd_rn(four(0, 64), four(32, 64)) : four(0, 32);
#pragma unroll
        for (u32 h = 16; h > 0; h >>= 1) p = __fadd_rn(p, __shfl_down_sync(0xffffffffu, p, h));
        p = __shfl_sync(0xffffffffu, p, 0);
        return __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(p, static_cast<float>(n)), v.eps)));
    };
    const float s = fold();
    bool bad = false;
    for (;;) {
        if (g >= groups) break;
        const u32 next = g + kWarps * gridDim.y;
        const float value = mine, by = weight;
        if (next < groups) { mine = x[32u * next + lane]; if (v.weight) weight = v.weight[32u * next + lane]; }
        bad |= !put_group(v, r, g, lane, value, by, s, out_stride, a8_stride);
        g = next;
    }
    if (v.status && __any_sync(0xffffffffu, bad) && lane == 0) atomicOr(&v.status[r], B200MOE_ROW_NONFINITE_ACTIVATION);
}
// A CTA reads all of its row while others write theirs: not where the results lie on the rows.
bool apart(const void* a, u64 an, const void* b, u64 bn) {
    const uintptr_t x = reinterpret_cast<uintptr_t>(a), y = reinterpret_cast<uintptr_t>(b);
    return !b || x + an <= y || y + bn <= x;
}
bool results_apart(const b200moe_rmsnorm_view& v) {
    const u64 xb = (u64(v.rows - 1) * (v.x_stride ? v.x_stride : v.n) + v.n) * 4, ob = (u64(v.rows - 1) * (v.out_stride ? v.out_stride : v.n) + v.n) * 4;
    const u64 as = v.a8.stride ? v.a8.stride : v.a8.width, ab = u64(v.rows) * as;
    return apart(v.x, xb, v.out, ob) && apart(v.x, xb, v.a8.codes, ab) && apart(v.x, xb, v.a8.deltas, ab / 8) && apart(v.x, xb, v.a8.sums, ab / 8);
}

// A chained launch asks for as much of a row at once as may be: it waits for trips.
template <u32 THREADS>
void launch_parts(const b200moe_rmsnorm_view& v, u32 parts, cudaStream_t stream) {
    const auto kernel = v.n <= 8 * 256 ? rmsnorm_a8_kernel<THREADS, 8, true> : v.n <= 16 * 256 ? rmsnorm_a8_kernel<THREADS, 16, true> : rmsnorm_a8_kernel<THREADS, 32, true>;
    small_launch(kernel, dim3(v.rows, parts), THREADS, 0, stream, v);
}

}  // namespace

int launch_rmsnorm_a8(const b200moe_rmsnorm_view& v, cudaStream_t stream) {
    if (v.rows == 0 || v.n == 0) return B200MOE_OK;
    const u32 sms = static_cast<u32>(device_sm_count());
    // Up to two rows an SM a row takes as many CTAs of 256 threads as have a group for every warp and as two an SM allow, two up to two and a half an SM and for rows above 5120:
    // 64 rows of 7168 10.4 us with one CTA of 32 warps, 4.8 so, 5.7 with four CTAs an SM; 180 rows of 2048, one and two, 4.4 and 3.8, 220 rows 4.4 and 5.2, 260 rows of 512 2.5 and
    // 3.4. Results that lie on the rows keep one CTA a row, of 32 warps where these have groups.
    const u32 parts = std::min((v.n / 32u + 7u) / 8u, v.rows <= sms ? 2u * sms / v.rows : 4u * v.rows <= 5u * sms || v.n > 5120u ? 2u : 1u);
    // Above, a CTA of 128 threads a row leaves room for more rows and has less to do for short ones; one of 256 is sooner done with a row, which counts from 330 values for every
    // row an SM on. 256 and 128 threads: 8192 rows of 32 16.3 and 9.0 us, of 512 31.4 and 22.5, of 7168 217 and 213; 400 rows of 7168 14.7 and 19. Rows up to 2560 come
    // in one batch of ten values a lane (600 rows of 2560 without A8 1.14 times as long in two).
    if (!chain_pays(v.rows)) {
        if (u64(v.n) * sms >= 330u * u64(v.rows)) plain_launch(v.n > 8 * 256 && v.n <= 10 * 256 ? rmsnorm_a8_kernel<256, 10, false> : rmsnorm_a8_kernel<256, 8, false>, v.rows, 256, 0, stream, v);
        else plain_launch(rmsnorm_a8_kernel<128, 4, false>, v.rows, 128, 0, stream, v);
    }
    else if (results_apart(v)) launch_parts<256>(v, parts, stream);
    else if (v.n > 256u) launch_parts<1024>(v, 1, stream);
    else launch_parts<256>(v, 1, stream);
    return after_launch("rmsnorm_a8");
}

}  // namespace b200moe
