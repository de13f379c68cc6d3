// RMSNorm in front of the FFN, fused with the A8 quantiser of its output (the rows the router and the experts read).
// One CTA per row; 256 of its threads are the 256 lanes of the host rule (src/cpu/core/reference.cpp:86-103): lane l runs
// a = fma(x[i], x[i], a) over i = l, l + L, ... (L = 128 below n = 512), the lanes fold by the halving tree, and
// s = 1 / sqrt(sum / n + eps) - IEEE division and square root. The second pass is warp-per-group: y = (x * s) * w for
// 32 consecutive values, written out and / or quantised by the A8 rule on the spot. HBM traffic: x once (the second
// pass hits L1 / L2), y and the A8 rows once.
#include <algorithm>

#include "kernels.cuh"

namespace b200moe {
namespace {

// WARPS: warps of the CTA, 0 = as launched (8 to 32). A fixed number unrolls the second pass at 48 registers, five CTAs of 8 warps an
// SM; as launched it takes 29, eight CTAs.
template <u32 WARPS, bool CHAIN>
__global__ void __launch_bounds__(WARPS ? WARPS * 32u : 1024u) rmsnorm_a8_kernel(b200moe_rmsnorm_view v) {
    chain_begin_if<CHAIN>();
    __shared__ float partial[256];
    const u32 r = blockIdx.x, t = threadIdx.x, n = v.n;
    const u32 x_stride = v.x_stride ? v.x_stride : n, out_stride = v.out_stride ? v.out_stride : n;
    const float* x = v.x + u64(r) * x_stride;
    const u32 lanes = n >= 512u ? 256u : 128u;
    float a = 0.0f;
    if (t < lanes) {
#pragma unroll 8
        for (u32 i = t; i < n; i += lanes) { const float xi = x[i]; a = __fmaf_rn(xi, xi, a); }
        partial[t] = a;
    }
    __syncthreads();
    for (u32 h = lanes / 2; h >= 32; h >>= 1) {
        if (t < h) partial[t] = __fadd_rn(partial[t], partial[t + h]);
        __syncthreads();
    }
    if (t < 32) {  // the last five levels inside one warp: lane t < h adds lane t + h, as above
        float p = partial[t];
#pragma unroll
        for (u32 h = 16; h > 0; h >>= 1) p = __fadd_rn(p, __shfl_down_sync(0xffffffffu, p, h));
        if (t == 0) partial[0] = p;
    }
    __syncthreads();
    const float s = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(partial[0], static_cast<float>(n)), v.eps)));
    const u32 lane = t & 31u, warp = t >> 5, groups = n / 32;
    const u32 a8_stride = v.a8.stride ? v.a8.stride : v.a8.width;
    bool bad = false;
    for (u32 g = warp; g < groups; g += WARPS ? WARPS : blockDim.x >> 5) {
        const u32 i = 32u * g + lane;
        float y = __fmul_rn(x[i], s);
        if (v.weight) y = __fmul_rn(y, v.weight[i]);
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
        bad |= !finite_f(y);
    }
    if (v.status && __any_sync(0xffffffffu, bad) && lane == 0) atomicOr(&v.status[r], B200MOE_ROW_NONFINITE_ACTIVATION);
}

constexpr u32 kWideRow = 2048;

}  // namespace

int launch_rmsnorm_a8(const b200moe_rmsnorm_view& v, cudaStream_t stream) {
    if (v.rows == 0 || v.n == 0) return B200MOE_OK;
    // Up to two rows an SM a row takes a warp per group in the second pass, up to 32 (the first pass has 256 lanes by contract): 5.8 us
    // with 32 warps against 8.6 with eight for 1 row of 2560, 24.8 against 31.1 for 296 of 7168. Warps without a group only
    // cost: 1 row of 256 takes 2.97 us with 32 warps, 2.73 with eight, 296 rows 3.48 and 3.02. Above two rows an SM eight warps keep
    // more rows in flight, in the unrolled form while all rows fit on the SMs at once (740 rows of 7168: 38.6 us against 40.4
    // as launched; 1024 rows 50.3 as launched against 64.1 with five to six CTAs an SM) and are long enough for it to matter
    // (592 rows of 2048: 11.6 against 11.8; of 1024: 7.5 both).
    const u32 sms = static_cast<u32>(device_sm_count());
    const u32 warps = std::min(32u, (v.n / 32u + 7u) / 8u * 8u);
    if (chain_pays(v.rows)) small_launch(rmsnorm_a8_kernel<0, true>, v.rows, 32u * warps, 0, stream, v);
    else if (v.rows <= 5u * sms && v.n >= kWideRow) plain_launch(rmsnorm_a8_kernel<8, false>, v.rows, 256, 0, stream, v);
    else plain_launch(rmsnorm_a8_kernel<0, false>, v.rows, 256, 0, stream, v);
    return after_launch("rmsnorm_a8");
}

}  // namespace b200moe
