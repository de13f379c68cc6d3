// Front of a layer call over a decode window (up to 8 rows) in ONE launch: A8 of the activations and the router logits. Selection and routes follow in
// a launch of one block (routes.cu), above 256 experts in one each.
//
// Contracts are those of the stand-alone kernels (a8.cu, router.cu): logits in the declared lane-strided order without fused multiply-add
// (src/ds41_moe.cpp:72-82). Bits do not change; bfloat16 activations are widened (exactly) on the way.
//
// Shape: blocks [0, logit_blocks) take four experts each. The block copies its experts' current 2048 columns and those of every activation row to
// shared memory asynchronously, in four groups of columns, and works on a group while the next ones arrive; a warp walks the lane classes of its
// experts and rows in ascending order. Blocks past logit_blocks quantise the activations, a warp a group of 32.
// What bounds it: latency, of one trip to memory and of the serial chains. With selection and routes in the block that finishes last (a ticket in the
// workspace), which had to find their code and read the logits back, the front took 10 / 12.3 / 20 us (1 row over 64 and 128 experts, 8 rows over
// 128, hidden 2048), of it 6 to 12 us in that block.
#include <algorithm>

#include "declared_math.cuh"
#include "kernels.cuh"

namespace b200moe {
namespace {

constexpr u32 kRunElems = 2048, kGroupElems = 512, kBlockExperts = 4;

__device__ __forceinline__ u32 smem_addr(const void* p) { return static_cast<u32>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ float4 widen4(uint2 b) {
    return make_float4(__uint_as_float(b.x << 16), __uint_as_float(b.x & 0xffff0000u), __uint_as_float(b.y << 16), __uint_as_float(b.y & 0xffff0000u));
}

struct PrologueArgs {
    b200moe_router_view r;
    b200moe_quantize_a8_view q;
    u32 logit_blocks;
    u32 x_vec, w_vec;  // rows in whole units of four values on their boundary
};

// A warp takes EW experts x RW rows of the block's 4 x RT.
template <int RT, int EW, int RW>
__global__ void __launch_bounds__(32 * (int(kBlockExperts) / EW) * (RT / RW)) prologue_decode_kernel(PrologueArgs a) {
    constexpr u32 kWarps = (kBlockExperts / EW) * (RT / RW), kThreads = 32 * kWarps;
    extern __shared__ __align__(16) float xs[];  // [RT rows | experts][kRunElems]
    const u32 lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const b200moe_quantize_a8_view& qv = a.q;
    const u32 x_stride = qv.x_stride ? qv.x_stride : qv.width;
    const bool bf16 = qv.x_is_bf16;
    const u16* x16 = static_cast<const u16*>(qv.x);
    const float* x32 = static_cast<const float*>(qv.x);
    chain_begin();

    if (blockIdx.x >= a.logit_blocks) {  // ---- A8 quantiser: one warp per (row, 32-value group)
        const u32 groups = qv.width / 32;
        const u64 item = u64(blockIdx.x - a.logit_blocks) * kWarps + warp;
        if (item >= u64(qv.rows) * groups) return;
        const u32 r = static_cast<u32>(item / groups), g = static_cast<u32>(item % groups), st = qv.out.stride ? qv.out.stride : qv.width;
        const u64 at = u64(r) * x_stride + 32u * g + lane;
        const float v = bf16 ? __uint_as_float(static_cast<u32>(x16[at]) << 16) : x32[at];
        float delta;
        int sum;
        const int code = a8_quantize_lane(v, &delta, &sum);
        qv.out.codes[u64(r) * st + 32u * g + lane] = static_cast<i8>(code);
        if (lane == 0) {
            qv.out.deltas[u64(r) * (st / 32) + g] = delta;
            if (qv.out.sums) qv.out.sums[u64(r) * (st / 32) + g] = sum;
        }
        if (qv.status && __any_sync(0xffffffffu, !finite_f(v)) && lane == 0) atomicOr(&qv.status[r], B200MOE_ROW_NONFINITE_ACTIVATION);
        return;
    }

    // ---- router logits
    const b200moe_router_view& rv = a.r;
    const u32 E = rv.policy.experts, H = rv.hidden, rows = rv.rows;
    const u32 e_base = blockIdx.x * kBlockExperts, e0 = EW * (warp % (kBlockExperts / EW)), r0 = RW * (warp / (kBlockExperts / EW));
    float acc[EW][RW];
#pragma unroll
    for (int e = 0; e < EW; ++e)
#pragma unroll
        for (int r = 0; r < RW; ++r) acc[e][r] = 0.0f;
    // A warp copies the group's columns of one row at a time; every request of the run is in flight at once.
    auto copy_row = [&](u32 to, const float* src, u32 n, bool vec) {  // n values to xs[to ..]
        const u32 dst = smem_addr(xs + to);
        if (vec) {
#pragma unroll
            for (u32 i = 0; i < kGroupElems / 128; ++i)
                if (lane + 32u * i < n / 4) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 16u * (lane + 32u * i)), "l"(src + 4u * (lane + 32u * i)) : "memory");
        } else {
            for (u32 i = lane; i < n; i += 32) asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst + 4u * i), "l"(src + i) : "memory");
        }
    };
    for (u32 c0 = 0; c0 < H; c0 += kRunElems) {
        const u32 n_el = min(kRunElems, H - c0);
        if (c0) __syncthreads();  // the previous run has been consumed
#pragma unroll 1
        for (u32 g0 = 0; g0 < kRunElems; g0 += kGroupElems) {
            const u32 n = g0 < n_el ? min(kGroupElems, n_el - g0) : 0u;
#pragma unroll 1
            for (u32 j = warp; j < kBlockExperts + (bf16 ? 0u : rows); j += kWarps) {
                const bool is_w = j < kBlockExperts;
                const float* src = is_w ? rv.weight + u64(min(e_base + j, E - 1)) * H : x32 + u64(j - kBlockExperts) * x_stride;
                copy_row((is_w ? RT + j : j - kBlockExperts) * kRunElems + g0, src + c0 + g0, n, is_w ? a.w_vec : a.x_vec);
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
        if (bf16) {
#pragma unroll 1
            for (u32 r = 0; r < rows; ++r) {
                const u16* src = x16 + u64(r) * x_stride + c0;
                float* dst = xs + r * kRunElems;
                if (a.x_vec) {
#pragma unroll 4
                    for (u32 i = threadIdx.x; i < n_el / 4; i += kThreads) reinterpret_cast<float4*>(dst)[i] = widen4(reinterpret_cast<const uint2*>(src)[i]);
                } else {
                    for (u32 i = threadIdx.x; i < n_el; i += kThreads) dst[i] = __uint_as_float(static_cast<u32>(src[i]) << 16);
                }
            }
        }
#pragma unroll 1
        for (u32 g0 = 0; g0 < n_el; g0 += kGroupElems) {
            switch (g0 / kGroupElems) {
                case 0: asm volatile("cp.async.wait_group 3;" ::: "memory"); break;
                case 1: asm volatile("cp.async.wait_group 2;" ::: "memory"); break;
                case 2: asm volatile("cp.async.wait_group 1;" ::: "memory"); break;
                default: asm volatile("cp.async.wait_group 0;" ::: "memory"); break;
            }
            __syncthreads();
            const u32 g1 = min(g0 + kGroupElems, n_el);
            const float *ws = xs + (RT + e0) * kRunElems, *xr = xs + r0 * kRunElems;
#pragma unroll 8
            for (u32 i = g0 + lane; i < g1; i += 32) {  // the lane class in ascending order (src/ds41_moe.cpp:72-82)
                float w[EW], x[RW];
#pragma unroll
                for (int e = 0; e < EW; ++e) w[e] = ws[e * kRunElems + i];
#pragma unroll
                for (int r = 0; r < RW; ++r) x[r] = xr[r * kRunElems + i];
#pragma unroll
                for (int e = 0; e < EW; ++e)
#pragma unroll
                    for (int r = 0; r < RW; ++r) acc[e][r] = __fadd_rn(acc[e][r], __fmul_rn(w[e], x[r]));
            }
        }
    }
#pragma unroll
    for (int e = 0; e < EW; ++e)
#pragma unroll
        for (int r = 0; r < RW; ++r) {
            float z = butterfly32(acc[e][r]);
            const u32 ex = e_base + e0 + e, row = r0 + r;
            if (lane == 0 && row < rows && ex < E) {
                if (rv.logit_bias) z = __fadd_rn(z, rv.logit_bias[ex]);
                rv.logits[u64(row) * E + ex] = z;
            }
        }
}

}  // namespace

bool prologue_fusable(const b200moe_router_view& r) { return r.rows >= 1 && r.rows <= 8; }

int launch_prologue(const b200moe_router_view& r, const b200moe_quantize_a8_view& q, cudaStream_t stream) {
    PrologueArgs a{};
    a.r = r; a.q = q;
    a.logit_blocks = (r.policy.experts + kBlockExperts - 1) / kBlockExperts;
    const u32 xs = q.x_stride ? q.x_stride : q.width;
    a.x_vec = aligned(q.x, q.x_is_bf16 ? 8 : 16) && xs % 4 == 0 && r.hidden % 4 == 0;
    a.w_vec = aligned(r.weight, 16) && r.hidden % 4 == 0;
    const u64 items = u64(q.rows) * (q.width / 32);
#define B200_PRO(RT, EW, RW)                                                                                         \
    {                                                                                                                \
        constexpr u32 warps = (kBlockExperts / EW) * (RT / RW), smem = (RT + kBlockExperts) * kRunElems * 4u;        \
        const auto kernel = prologue_decode_kernel<RT, EW, RW>;                                                      \
        if (int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), smem)) return rc;                    \
        if (int rc = prefer_max_shared(reinterpret_cast<const void*>(kernel))) return rc;                            \
        chain_launch(kernel, a.logit_blocks + static_cast<u32>((items + warps - 1) / warps), 32 * warps, smem, stream, a); \
    }
    if (r.rows == 1) B200_PRO(1, 1, 1)
    else if (r.rows == 2) B200_PRO(2, 1, 2)
    else if (r.rows <= 4) B200_PRO(4, 1, 2)
    else B200_PRO(8, 2, 2)
#undef B200_PRO
    return after_launch("prologue_decode");
}

}  // namespace b200moe
