// A8 activation quantiser: one warp per (row, 32-value group) and one value per lane, or eight lanes per group and four values each.
// Contract: src/cpu/core/reference.cpp:35-55 (= src/ds41_formats.cpp:146-165).
// HBM traffic per row: width * 4 B in (2 B for bfloat16), width * 1.25 B out: negligible beside the expert weights.
#include <algorithm>

#include "kernels.cuh"

namespace b200moe {
namespace {

template <bool BF16>
__global__ void __launch_bounds__(256) quantize_a8_kernel(const void* x, u32 rows, u32 groups, u32 x_stride,
                                                          i8* codes, float* deltas,
                                                          i32* sums, u32 stride, u32* status) {
    chain_begin();
    const u32 lane = threadIdx.x & 31u;
    const u64 item = u64(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (item >= u64(rows) * groups) return;
    const u32 r = static_cast<u32>(item / groups), g = static_cast<u32>(item % groups);
    const u64 at = u64(r) * x_stride + 32u * g + lane;
    float v;
    if (BF16) v = __uint_as_float(static_cast<u32>(static_cast<const u16*>(x)[at]) << 16);
    else v = static_cast<const float*>(x)[at];
    float delta;
    int sum;
    const int code = a8_quantize_lane(v, &delta, &sum);
    codes[u64(r) * stride + 32u * g + lane] = static_cast<i8>(code);
    if (lane == 0) {
        deltas[u64(r) * (stride / 32) + g] = delta;
        if (sums) sums[u64(r) * (stride / 32) + g] = sum;
    }
    if (status) {
        const bool bad = __any_sync(0xffffffffu, !finite_f(v));
        if (bad && lane == 0) atomicOr(&status[r], B200MOE_ROW_NONFINITE_ACTIVATION);
    }
}

// The same rule with four values a lane and eight lanes a group: wide loads, three shuffles a reduction instead of five, a
// quarter of the warps. Bound by issue slots; with a division a value (72 % of them busy, and 62 % of the pipe that takes the reciprocals) and one for the item's row 8192 x 7168
// FP32 took 104 us, with one reciprocal a group, exact quotients near halves alone and a product for the row 86, 0.54 of the measured copy bandwidth; 1024 rows 13.1 -> 10.9 us, 4096 x 2048
// bfloat16 14.9 -> 13.5. With `wide` the bfloat16 values
// are also written out as FP32 for the router, instead of by a pass of their own before this one (8192 x 7168: 119 + 305 -> 218 us).
template <bool BF16>
__global__ void __launch_bounds__(256) quantize_a8_vec_kernel(const void* x, u32 items, u32 groups, u32 per_group, u32 shift, u32 x_stride, i8* codes,
                                                              float* deltas, i32* sums, u32 stride, u32* status,
                                                              float* wide, u32 wide_stride) {
    chain_begin();
    const u32 t = blockIdx.x * 256u + threadIdx.x, sub = t & 7u;
    const bool valid = (t >> 3) < items;
    const u32 item = valid ? t >> 3 : items - 1u;  // spare lanes of the last warp repeat its last group and store nothing
    const u32 r = static_cast<u32>(u64(item) * per_group >> shift), g = item - r * groups;  // item / groups: see the launch
    const u64 at = u64(r) * x_stride + 32u * g + 4u * sub;
    float v[4];
    if (BF16) {
        const uint2 b = load(reinterpret_cast<const uint2*>(static_cast<const u16*>(x) + at));
        v[0] = __uint_as_float(b.x << 16); v[1] = __uint_as_float(b.x & 0xffff0000u); v[2] = __uint_as_float(b.y << 16); v[3] = __uint_as_float(b.y & 0xffff0000u);
        if (wide && valid) *reinterpret_cast<float4*>(wide + u64(r) * wide_stride + 32u * g + 4u * sub) = make_float4(v[0], v[1], v[2], v[3]);
    } else {
        const float4 f = load(reinterpret_cast<const float4*>(static_cast<const float*>(x) + at));
        v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
    }
    float amax = fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3])));  // NaN operands are ignored (a8_quantize_lane)
#pragma unroll
    for (int d = 4; d; d >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, d));
    const bool tiny = amax > 0.0f && amax < 0x1p-119f;
    const float delta = (amax == 0.0f || tiny) ? 1.0f : __fdiv_rn(amax, 127.0f);
    const float inverse = __frcp_rn(delta);
    float quotient[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) quotient[i] = __fmul_rn(v[i], inverse);
    int sum = 0;
    u32 word = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float q = rintf(quotient[i]);
        // The product lies within 2^-15 of the quotient and the quotient's rounding within 2^-17 of it, so the integers can differ near a half alone (or where there is no number).
        if (!(fabsf(__fsub_rn(quotient[i], q)) < 0.5f - 0x1p-13f)) q = rintf(__fdiv_rn(v[i], delta));
        if (tiny) q = 0.0f;
        const float lo = (-127.0f < q) ? q : -127.0f;
        const int code = static_cast<int>((lo < 127.0f) ? lo : 127.0f);
        sum += code;
        word |= (static_cast<u32>(code) & 0xffu) << (8 * i);
    }
#pragma unroll
    for (int d = 4; d; d >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, d);
    if (!valid) return;
    *reinterpret_cast<u32*>(codes + u64(r) * stride + 32u * g + 4u * sub) = word;
    if (sub == 0) {
        deltas[u64(r) * (stride / 32) + g] = delta;
        if (sums) sums[u64(r) * (stride / 32) + g] = sum;
    }
    if (status && !(finite_f(v[0]) && finite_f(v[1]) && finite_f(v[2]) && finite_f(v[3]))) atomicOr(&status[r], B200MOE_ROW_NONFINITE_ACTIVATION);
}

// bfloat16 bit patterns widened to FP32 (exact): the router reads FP32 rows.
__global__ void __launch_bounds__(256) widen_bf16_kernel(const u16* in, float* out, u64 count) {
    chain_begin();
    for (u64 i = u64(blockIdx.x) * blockDim.x + threadIdx.x; i < count; i += u64(gridDim.x) * blockDim.x)
        out[i] = __uint_as_float(static_cast<u32>(in[i]) << 16);
}

}  // namespace

int launch_widen_bf16(const u16* in, float* out, u64 count, cudaStream_t stream) {
    if (count == 0) return B200MOE_OK;
    const u32 blocks = static_cast<u32>(std::min<u64>((count + 255) / 256, 148u * 16u));
    small_launch(widen_bf16_kernel, blocks, 256, 0, stream, in, out, count);
    return after_launch("widen_bf16");
}

// Four values a lane need whole 16- (FP32) or 8-byte (bfloat16) units in x and 4-byte units in the codes. The one-value form takes every other layout, and what its blocks of eight
// groups cover with three an SM: up to there a launch is one block's chain, whose reductions are one instruction each (FP32, us, one value and four: 1 row of 256 1.09 and 1.26, 8 of
// 2048 1.16 and 1.41, 8 of 7168 1.24 and 1.43, 16 of 7168, above the line, 1.43 and 1.45, 20 of 7168 2.02 and 1.41; bfloat16 alike).
bool quantize_a8_vec_ok(const b200moe_quantize_a8_view& v) {
    const u32 x_stride = v.x_stride ? v.x_stride : v.width;
    return aligned(v.x, v.x_is_bf16 ? 8 : 16) && x_stride % 4 == 0 && aligned(v.out.codes, 4) && u64(v.rows) * (v.width / 32) < (1ull << 28);
}

int launch_quantize_a8(const b200moe_quantize_a8_view& v, cudaStream_t stream, float* wide, u32 wide_stride) {
    const u32 groups = v.width / 32;
    const u64 items = u64(v.rows) * groups;
    if (items == 0) return B200MOE_OK;
    const u32 x_stride = v.x_stride ? v.x_stride : v.width, stride = v.out.stride ? v.out.stride : v.width;
    if (quantize_a8_vec_ok(v) && (wide || items > 3u * 8u * static_cast<u32>(device_sm_count()))) {
        const u32 vec_blocks = static_cast<u32>((items + 31) / 32);
        // n / groups = n * per_group >> shift for every n below 2^28: per_group * groups lies between 2^shift and 2^shift + groups, and groups is no more than 2^(shift - 28).
        u32 shift = 28;
        while ((1ull << (shift - 28)) < groups) ++shift;
        const u32 per_group = static_cast<u32>((1ull << shift) / groups + 1);
        if (v.x_is_bf16)
            small_launch(quantize_a8_vec_kernel<true>, vec_blocks, 256, 0, stream, v.x, static_cast<u32>(items), groups, per_group, shift, x_stride, v.out.codes, v.out.deltas, v.out.sums, stride, v.status, wide, wide_stride);
        else
            small_launch(quantize_a8_vec_kernel<false>, vec_blocks, 256, 0, stream, v.x, static_cast<u32>(items), groups, per_group, shift, x_stride, v.out.codes, v.out.deltas, v.out.sums, stride, v.status, nullptr, 0);
        return after_launch("quantize_a8");
    }
    const u32 blocks = static_cast<u32>((items + 7) / 8);
    if (v.x_is_bf16)
        small_launch(quantize_a8_kernel<true>, blocks, 256, 0, stream, v.x, v.rows, groups, x_stride, v.out.codes, v.out.deltas, v.out.sums, stride, v.status);
    else
        small_launch(quantize_a8_kernel<false>, blocks, 256, 0, stream, v.x, v.rows, groups, x_stride, v.out.codes, v.out.deltas, v.out.sums, stride, v.status);
    return after_launch("quantize_a8");
}

}  // namespace b200moe
