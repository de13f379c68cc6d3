// Routed experts, Qwen A8 family, GROUPED form for token blocks (prefill): the integer dots run on the tensor cores, everything
// after the dots is the same declared FP32 arithmetic as the decode kernels, so the results are bit for bit those of
// gemv_q4k.cu / gemv_q4k_stream.cu (contract: src/cpu/core/routed_expert.hpp:9-15, row rule routed_expert.cpp:73-108; the
// reference's own tensor-core form is project_kernel / down_kernel, src/cuda/core/moe_a8.cuh:76-206, :225-341).
//
// What bounds it: latency - no unit is full (512 tokens x 34,816 rows x 5120: issue slots 53 %, FP32 pipe 51, shared-memory wavefronts
// 54, integer MMA 18; warps wait on fixed latencies and loads for 1.9 and 1.3 issues per issue, three to four of them a scheduler),
// and about half the instructions are factor and code loads, masks and duplicates, a factor serving two chunks. The contract scales every 32-wide group's EXACT
// integer dot by its own factors: five FP32 operations per (row, token, group), i.e. 320 clocks per group of a 128 x 64 tile at
// 128 lanes a clock. The dots of the same group take 136 clocks of the register-to-register integer MMA (measured: 8.5 clocks
// per m16n8k32 and scheduler, 22.5 together with ten packed FP32 instructions), so the dots stay in REGISTERS. The form before
// this one (tcgen05 with accumulators in tensor memory, operands unpacked to shared memory) spent 980 clocks per group, most of
// them in its unpack -> MMA -> drain hand-overs: 1230 us for 512 tokens x 34,816 rows x 5120, 957 us now.
//
// Tile = (expert, 128 weight rows, kGN of the expert's tokens). gate/up: rows 0..63 are gate rows [64c, 64c + 64), rows
// 64..127 the up rows of the same outputs, so SwiGLU + the A8 rule of h finish inside the tile. down: 128 rows of H.
// A persistent CTA per SM walks tiles round-robin; a stage of the ring (three) is one super-block: 256 columns.
//   * helper warps (4): the tile's weight rows arrive by two tiled TMA copies (160 bytes x 64 rows: the 144 of the super-block
//     and 16 more, which puts rows 8 (mod 32) words apart - the fragment loads below are conflict free), the tokens' codes, deltas and
//     sums by 16-byte asynchronous copies (codes 288 bytes apart, for the same reason), one stage ahead; deltas and sums that do
//     not lie in 16-byte units come in 4-byte copies, whose eight-way bank conflicts cost 12 % of the kernel. A helper thread decodes the
//     factors of one weight row and transposes {E, S} of one token (half the groups each).
//   * consumer warps: warp = 32 rows x every kSplit-th 8-token chunk (a tile with few tokens still uses most warps). The
//     nibbles go from shared memory straight into A fragments (low nibbles by a mask, high nibbles left in place as 16 q), the
//     codes into B fragments; the MMA starts at the integer 0x4b400000, so its result read as a float is M + dot with
//     M = 1.5 * 2^23, and fma(D, M + dot, -D * M) is D * dot rounded once (D = d * scale has at most 17 significant bits, so
//     D * M is exact): no conversion. Packed FP32 instructions work on two tokens at a time; the four chains acc_p of a lane's
//     cells stay in registers; (a0 + a1) + (a2 + a3) at the end - exactly the decode kernels' order.
//     A super-block with a non-finite d takes the same steps with the dot converted first (inf - inf would turn an infinity
//     into a NaN).
// Every wait is bounded; on a timeout the roles stop working and the launch sets B200MOE_JOB_WAIT_ABORTED in the job summary.
#include <cuda.h>

#include "q4k_row.cuh"

namespace b200moe {
namespace {
using namespace q4k;

// Three consumer warps a scheduler with two chunks each: with two warps of four chunks (tiles of 64 tokens) the FP32 pipe sits idle
// while both wait for their shared-memory reads and MMAs (4096 x 8 tokens over 128 experts of 2048 x 768: gate/up 1437 us against
// 1346 us; 512 tokens x 17,408 -> 5120: down 517 against 400 us, where the narrower tiles also fill the last wave).
constexpr u32 kSplit = 3, kChunks = 2;           // consumer warps that share a tile's tokens; 8-token chunks of each
constexpr u32 kGM = 128, kGN = 8 * kSplit * kChunks;  // tile: weight rows x tokens
constexpr u32 kConsumers = 4 * kSplit, kHelpers = 4;  // warps
constexpr u32 kGThreads = (kConsumers + kHelpers) * 32;
constexpr u32 kStages = 3;
constexpr u32 kRowPitch = kQ4KBlock + 16, kCodePitch = 256 + 32;
constexpr u32 kRawBytes = kGM * kRowPitch, kCodeBytes = kGN * kCodePitch, kEsBytes = 8 * kGN * 8, kFacBytes = 8 * kGM * 8, kPrivBytes = kHelpers * 32 * 32;
constexpr u32 kStageBytes = kRawBytes + kCodeBytes + kEsBytes + kFacBytes + kPrivBytes;
constexpr u32 kOutPitch = kGM + 4;           // floats; twice the pitch is 8 (mod 32): the fragment stores meet every bank once
constexpr u32 kOutBytes = kGN * kOutPitch * 4;  // epilogue tile (gate/up)
constexpr u32 kMaxUnion = 1024;
constexpr u32 kBarBytes = 3 * kStages * 8 + 24 + kStages * 16 + 2 * 64 * 4;  // raw_full[], ready[], empty[]; abort flag; non-finite flags; token rows
constexpr u32 kGroupedSmem = kStages * kStageBytes + kOutBytes + (kMaxUnion + 2) * 4 + kBarBytes + 64;
static_assert(kGN <= 64 && kGN % 16 == 0, "a helper thread stages half the groups of one token");
static_assert(kGroupedSmem > 114u * 1024u && kGroupedSmem <= 227u * 1024u, "one CTA per SM, within the shared memory of an SM");
constexpr u32 kWaitLimit = 1u << 20;         // polls of up to a microsecond
constexpr float kMagic = 12582912.0f;        // 1.5 * 2^23 = the float with the bits 0x4b400000
// Register split between whole warp groups, out of what the launch gives every thread (65,536 over the threads, by eights).
constexpr u32 kLaunchRegs = 65536u / kGThreads / 8u * 8u, kHelperRegs = 80;
constexpr u32 kConsumerRegs = (kGThreads * kLaunchRegs - kHelpers * 32u * kHelperRegs) / (kConsumers * 32u) / 8u * 8u;
static_assert(kConsumers * 32 * kConsumerRegs + kHelpers * 32 * kHelperRegs <= kGThreads * kLaunchRegs, "setmaxnreg split exceeds the launch's registers");

// Two FP32 lanes per instruction (Blackwell packed FP32): each lane is one IEEE round-to-nearest operation, the same result
// as two scalar instructions at half the issue slots. A packed add fed by a packed multiply did not reproduce the scalar
// bits on B200 (it behaves as contracted), so an add is written as a * 1 + b, where the 1 is a kernel argument that no
// compiler stage can fold away: one rounding, of a + b.
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
    float2 c;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(reinterpret_cast<u64&>(c)) : "l"(reinterpret_cast<const u64&>(a)), "l"(reinterpret_cast<const u64&>(b)));
    return c;
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    float2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(reinterpret_cast<u64&>(d)) : "l"(reinterpret_cast<const u64&>(a)), "l"(reinterpret_cast<const u64&>(b)), "l"(reinterpret_cast<const u64&>(c)));
    return d;
}
__device__ __forceinline__ float2 both(float v) { return make_float2(v, v); }
// 16 weight rows x 8 tokens x one group: unsigned nibble bytes times signed codes, on top of the bits of kMagic.
__device__ __forceinline__ void mma_magic(float2 (&d)[2], u32 a0, u32 a1, u32 a2, u32 a3, u32 b0, u32 b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
        : "=r"(reinterpret_cast<u32&>(d[0].x)), "=r"(reinterpret_cast<u32&>(d[0].y)), "=r"(reinterpret_cast<u32&>(d[1].x)), "=r"(reinterpret_cast<u32&>(d[1].y))
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0x4b400000));
}
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(saddr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async4(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(saddr(dst)), "l"(src) : "memory");
}

struct GroupedArgs {
    b200moe_shape shape;
    b200moe_routes routes;
    b200moe_a8_rows in;      // x (gate/up: indexed by row) or act (down: indexed by slot)
    b200moe_a8_rows act;     // gate/up output
    float* gate_out;
    float* up_out;
    float* raw;              // down output [slots][hidden]
    u32* row_status;
    u32* summary;
    u32 n_row_tiles;         // inter / 64 (gate/up) or hidden / 128 (down)
    u32 K;                   // hidden (gate/up) or inter (down)
    u32 es_vec;              // the input's deltas and sums lie in whole 16-byte units
    float one;               // 1.0f, unknown to the compiler (mul2 / fma2)
};

struct Tile { u32 expert, eb, nt, c, tt; };

// Tile id -> (union expert, token tile, row tile): row tiles fastest, then the expert's token tiles, experts ascending.
__device__ __forceinline__ Tile find_tile(const GroupedArgs& a, const u32* cum, u32 n_union, u32 id) {
    const u32 q = id / a.n_row_tiles;
    Tile t;
    t.c = id - q * a.n_row_tiles;
    u32 lo = 0, hi = n_union;  // largest j with cum[j] <= q
    while (hi - lo > 1) {
        const u32 mid = (lo + hi) >> 1;
        if (cum[mid] <= q) lo = mid; else hi = mid;
    }
    t.tt = q - cum[lo];
    t.expert = a.routes.experts[lo];
    const u32 b0 = a.routes.begins[lo], b1 = a.routes.begins[lo + 1];
    t.eb = b0 + kGN * t.tt;
    t.nt = min(kGN, b1 - t.eb);
    return t;
}

// One super-block of the warp's 32 rows against the tokens of its chunks. rows: the lane's first weight row of the stage (nibbles
// of its k slice); codes: the lane's token row of chunk 0; es / fac: the lane's {E, E', S, S'} and {rows 0, 8, 16, 24} factors.
// acc[cc][i][p]: chain p of weight row 8 i + lane / 4 and two tokens of chunk kSplit cc + w. SLOW: the dot is converted first.
template <bool SLOW>
__device__ __forceinline__ void superblock(const unsigned char* rows, const unsigned char* codes, const float4* es, const float4* fac, u32 n_chunks,
                                           float2 one, float2 (&acc)[kChunks][4][4]) {
#pragma unroll
    for (int p = 0; p < 4; ++p) {
        uint2 q[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) q[i] = *reinterpret_cast<const uint2*>(rows + 8 * i * kRowPitch + 32 * p);
        float Dl[4], Ml[4], Dh[4], Mh[4], Nl[4], Nh[4];
        *reinterpret_cast<float4*>(Dl) = fac[(4 * p) * (kGM / 4)]; *reinterpret_cast<float4*>(Ml) = fac[(4 * p + 1) * (kGM / 4)];
        *reinterpret_cast<float4*>(Dh) = fac[(4 * p + 2) * (kGM / 4)]; *reinterpret_cast<float4*>(Mh) = fac[(4 * p + 3) * (kGM / 4)];
#pragma unroll
        for (int i = 0; i < 4; ++i) { Nl[i] = __fmul_rn(Dl[i], -kMagic); Nh[i] = __fmul_rn(Dh[i], -kMagic); }
#pragma unroll
        for (int cc = 0; cc < (int)kChunks; ++cc) {
            if (cc >= n_chunks) break;  // no valid token in these columns (warp-uniform)
            const unsigned char* c = codes + 8 * kSplit * cc * kCodePitch + 64 * p;
            const uint2 bl = *reinterpret_cast<const uint2*>(c), bh = *reinterpret_cast<const uint2*>(c + 32);
            const float4 el = es[(2 * p) * (kGN / 2) + 4 * kSplit * cc], eh = es[(2 * p + 1) * (kGN / 2) + 4 * kSplit * cc];
#pragma unroll
            for (int mt = 0; mt < 2; ++mt) {
                float2 l[2], h[2];
                const uint2 r0 = q[2 * mt], r1 = q[2 * mt + 1];
                mma_magic(l, r0.x & 0x0f0f0f0fu, r1.x & 0x0f0f0f0fu, r0.y & 0x0f0f0f0fu, r1.y & 0x0f0f0f0fu, bl.x, bl.y);
                mma_magic(h, r0.x & 0xf0f0f0f0u, r1.x & 0xf0f0f0f0u, r0.y & 0xf0f0f0f0u, r1.y & 0xf0f0f0f0u, bh.x, bh.y);
#pragma unroll
                for (int z = 0; z < 2; ++z) {
                    const int i = 2 * mt + z;
                    float2 al, ah;
                    if (SLOW) {
                        al = mul2(both(Dl[i]), make_float2(__fsub_rn(l[z].x, kMagic), __fsub_rn(l[z].y, kMagic)));
                        ah = mul2(both(Dh[i]), make_float2(__fsub_rn(h[z].x, kMagic), __fsub_rn(h[z].y, kMagic)));
                    } else {
                        al = fma2(both(Dl[i]), l[z], both(Nl[i]));
                        ah = fma2(both(Dh[i]), h[z], both(Nh[i]));
                    }
                    // x = E * ((D * float(dot)) - (DM * S)) for the pair's two groups; M holds -DM, and (-DM) * S = -(DM * S) exactly
                    const float2 sl = fma2(al, one, mul2(both(Ml[i]), make_float2(el.z, el.w)));
                    const float2 sh = fma2(ah, one, mul2(both(Mh[i]), make_float2(eh.z, eh.w)));
                    const float2 x = fma2(mul2(make_float2(el.x, el.y), sl), one, mul2(make_float2(eh.x, eh.y), sh));
                    acc[cc][i][p] = fma2(x, one, acc[cc][i][p]);
                }
            }
        }
    }
}

// SwiGLU + the A8 rule of up to four (token, 32 outputs) tasks of one warp, step by step over the four, so that their shuffle
// and division chains overlap. g, u: the lane's gate and up values; returns per task whether a value is not finite.
constexpr int kTasks = 4;
__device__ __forceinline__ u32 swiglu_a8(const float (&g)[kTasks], const float (&u)[kTasks], int (&code)[kTasks], float (&delta)[kTasks], int (&sum)[kTasks]) {
    float h[kTasks], amax[kTasks];
    u32 bad = 0;
#pragma unroll
    for (int i = 0; i < kTasks; ++i) { h[i] = swiglu_qwen(g[i], u[i]); amax[i] = fabsf(h[i]); }
#pragma unroll
    for (int i = 0; i < kTasks; ++i) bad |= __any_sync(0xffffffffu, !finite_f(g[i]) || !finite_f(u[i]) || !finite_f(h[i])) ? 1u << i : 0u;
#pragma unroll
    for (int d = 16; d; d >>= 1)
#pragma unroll
        for (int i = 0; i < kTasks; ++i) amax[i] = fmaxf(amax[i], __shfl_xor_sync(0xffffffffu, amax[i], d));
#pragma unroll
    for (int i = 0; i < kTasks; ++i) {  // a8_quantize_lane (common.cuh)
        const bool tiny = amax[i] > 0.0f && amax[i] < 0x1p-119f;
        delta[i] = (amax[i] == 0.0f || tiny) ? 1.0f : __fdiv_rn(amax[i], 127.0f);
        const float r = tiny ? 0.0f : rintf(__fdiv_rn(h[i], delta[i]));
        const float lo = (-127.0f < r) ? r : -127.0f;
        code[i] = static_cast<int>((lo < 127.0f) ? lo : 127.0f);
        sum[i] = __reduce_add_sync(0xffffffffu, code[i]);
    }
    return bad;
}

template <bool kDown>
__global__ void __launch_bounds__(kGThreads, 1) grouped_q4k_kernel(const __grid_constant__ CUtensorMap tm0, const __grid_constant__ CUtensorMap tm1,
                                                                   GroupedArgs a) {
    extern __shared__ __align__(128) unsigned char smem[];
    float* s_out = reinterpret_cast<float*>(smem + kStages * kStageBytes);          // [kGN][kOutPitch]
    u64* raw_full = reinterpret_cast<u64*>(smem + kStages * kStageBytes + kOutBytes);
    u64* ready = raw_full + kStages;
    u64* empty = ready + kStages;
    u32* s_abort_word = reinterpret_cast<u32*>(empty + kStages);                     // 24 bytes
    u32* s_slow = s_abort_word + 6;                                                  // [stage][row quarter]: a non-finite d among the rows
    u32* s_src = s_slow + kStages * 4;                                               // [tile parity][64]: A8 rows of the tile's tokens
    u32* cum = s_src + 2 * 64;                                                       // [kMaxUnion + 1]
    volatile u32* s_abort = s_abort_word;

    if (kDown && a.summary && *a.summary) return;  // a failed or aborted projection skips the stage (routed_expert.hpp:17-19)

    const u32 tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    const u32 n_union = min(a.routes.counts[0], kMaxUnion);
    for (u32 j = tid; j < n_union; j += kGThreads) cum[j + 1] = (a.routes.begins[j + 1] - a.routes.begins[j] + kGN - 1) / kGN;
    if (tid == 0) {
        cum[0] = 0;
        for (u32 i = 0; i < kStages; ++i) { mbar_init(&raw_full[i], 1); mbar_init(&ready[i], kHelpers); mbar_init(&empty[i], kConsumers); }
        *s_abort_word = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (warp == 0) {  // inclusive scan of the token-tile counts, 32 at a time
        u32 carry = 0;
        for (u32 j0 = 0; j0 < n_union; j0 += 32) {
            u32 v = j0 + lane < n_union ? cum[j0 + lane + 1] : 0u;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) { const u32 o = __shfl_up_sync(0xffffffffu, v, d); if (lane >= (u32)d) v += o; }
            if (j0 + lane < n_union) cum[j0 + lane + 1] = carry + v;
            carry += __shfl_sync(0xffffffffu, v, 31);
        }
    }
    __syncthreads();
    const u32 n_tiles = cum[n_union] * a.n_row_tiles;
    const u32 I = a.shape.inter, H = a.shape.hidden;
    const u32 nblocks = a.K / 256;
    bool ok = true;
    const u32 my_tiles = n_tiles > blockIdx.x ? (n_tiles - blockIdx.x + gridDim.x - 1) / gridDim.x : 0u;
    const u32 total = my_tiles * nblocks;  // stages of this CTA

    if (warp >= kConsumers) {
        // ================================================================================================= helpers
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kHelperRegs));
        const u32 lt = tid - kConsumers * 32;            // 0..127 = weight row of the tile
        const u32 hw = lt >> 5, tok = lt & 63u, half = lt >> 6;  // the token whose {E, S} this thread stages, and which half of the groups
        const u32 in_stride = a.in.stride ? a.in.stride : a.in.width, in_gs = in_stride / 32;
        u32 ik = 0, ib = 0, cy = 0;                      // tile and super-block of the next stage to request
        const float* t_deltas = nullptr;
        const i32* t_sums = nullptr;
        // Requests stage m: rows by TMA, codes and {E, S} by asynchronous copies (one commit group per thread and stage).
        auto request = [&](u32 m) {
            const u32 slot = m % kStages;
            unsigned char* st = smem + slot * kStageBytes;
            if (ok && m >= kStages) ok = mbar_wait(&empty[slot], (m / kStages - 1u) & 1u, kWaitLimit, s_abort);
            if (ib == 0) {  // a new tile: every helper thread publishes the A8 row of its token
                const Tile t = find_tile(a, cum, n_union, blockIdx.x + ik * gridDim.x);
                const u32 ent = t.eb + min(tok, t.nt - 1u);
                const u32 src = kDown ? a.routes.slots[ent] : a.routes.rows[ent];
                if (half == 0) s_src[(ik & 1u) * 64u + tok] = src;
                t_deltas = a.in.deltas + u64(src) * in_gs + 4u * half;
                t_sums = a.in.sums + u64(src) * in_gs + 4u * half;
                cy = kDown ? t.expert * H + kGM * t.c : t.expert * I + 64u * t.c;
                asm volatile("bar.sync 1, %0;" ::"n"(kHelpers * 32) : "memory");
            }
            if (ok) {
                if (lt == 0) {
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the consumers' reads precede the copies below
                    mbar_expect_tx(&raw_full[slot], kRawBytes);
                    tma_2d(st, &tm0, ib * kQ4KBlock, cy, &raw_full[slot]);
                    tma_2d(st + 64u * kRowPitch, kDown ? &tm0 : &tm1, ib * kQ4KBlock, kDown ? cy + 64u : cy, &raw_full[slot]);
                }
                const u32* src = s_src + (ik & 1u) * 64u;
                unsigned char* sc = st + kRawBytes;
#pragma unroll
                for (u32 i = 0; i < kGN / 8; ++i) {  // a half warp copies the 256 codes of one token
                    const u32 tk = (kGN / 4) * hw + 2u * i + (lane >> 4);
                    cp_async16(sc + tk * kCodePitch + 16u * (lane & 15u), a.in.codes + u64(src[tk]) * in_stride + 256u * ib + 16u * (lane & 15u));
                }
                unsigned char* pv = st + kRawBytes + kCodeBytes + kEsBytes + kFacBytes + 32u * lt;
                if (a.es_vec) {
                    cp_async16(pv, t_deltas + 8u * ib);
                    cp_async16(pv + 16, t_sums + 8u * ib);
                } else {
#pragma unroll
                    for (u32 i = 0; i < 4; ++i) {
                        cp_async4(pv + 4u * i, t_deltas + 8u * ib + i);
                        cp_async4(pv + 16u + 4u * i, t_sums + 8u * ib + i);
                    }
                }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
            if (++ib == nblocks) { ib = 0; ++ik; }
        };
        if (total) request(0);
        u32 asked = total ? 1u : 0u;
        for (u32 m = 0; m < total; ++m) {
            if (m + 1 < total) { request(m + 1); ++asked; }
            else asm volatile("cp.async.commit_group;" ::: "memory");  // an empty group keeps the count of the wait below fixed
            const u32 slot = m % kStages;
            unsigned char* st = smem + slot * kStageBytes;
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            if (ok) ok = mbar_wait(&raw_full[slot], (m / kStages) & 1u, kWaitLimit, s_abort);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) continue;  // no more requests or hand-overs; the tile barrier above is still met by every helper
            const uint4 hdr = *reinterpret_cast<const uint4*>(st + lt * kRowPitch);
            const bool slow = __any_sync(0xffffffffu, (hdr.x & 0x7c00u) == 0x7c00u);
            if (lane == 0) s_slow[slot * 4u + hw] = slow ? 1u : 0u;
            // the row's factors, [group][D | -DM][quarter][row % 8][row / 8 % 4]: a lane's four rows are one 128-bit load;
            // the high nibbles' dots come as 16 * dot
            float* fac = reinterpret_cast<float*>(st + kRawBytes + kCodeBytes + kEsBytes) + (lt & ~31u) + (lt & 7u) * 4u + ((lt >> 3) & 3u);
#pragma unroll
            for (u32 p = 0; p < 4; ++p) {
                const Factors f = q4k_factors(hdr, p);
                fac[(4 * p) * kGM] = f.Dl; fac[(4 * p + 1) * kGM] = -f.DMl;
                fac[(4 * p + 2) * kGM] = __fmul_rn(f.Dh, 0.0625f); fac[(4 * p + 3) * kGM] = -f.DMh;
            }
            const unsigned char* pv = st + kRawBytes + kCodeBytes + kEsBytes + kFacBytes + 32u * lt;
            const float4 e = *reinterpret_cast<const float4*>(pv);
            const int4 sm = *reinterpret_cast<const int4*>(pv + 16);
            if (tok < kGN) {
                float* es = reinterpret_cast<float*>(st + kRawBytes + kCodeBytes) + (4u * half * (kGN / 2) + (tok >> 1)) * 4u + (tok & 1u);  // [group][token pair] {E, E', S, S'}
                es[0] = e.x; es[2] = static_cast<float>(sm.x);
                es[2 * kGN] = e.y; es[2 * kGN + 2] = static_cast<float>(sm.y);
                es[4 * kGN] = e.z; es[4 * kGN + 2] = static_cast<float>(sm.z);
                es[6 * kGN] = e.w; es[6 * kGN + 2] = static_cast<float>(sm.w);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&ready[slot]);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        if (*s_abort && lt == 0)  // wait (bounded) for the copies still in flight before the CTA retires
            for (u32 n = asked > kStages ? asked - kStages : 0u; n < asked; ++n)
                for (u32 i = 0; i < (kWaitLimit >> 8); ++i)
                    if (mbar_try_wait(&raw_full[n % kStages], (n / kStages) & 1u, kWaitHintNs)) break;
    } else {
        // ================================================================================================ consumers
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kConsumerRegs));
        const u32 quarter = warp & 3u, w = warp >> 2;   // 32 rows of the tile; the 8-token chunks alternate between the kSplit warps of a quarter
        const u32 fr = lane >> 2, ft = lane & 3u;       // fragments: rows 32 quarter + 8 i + fr (i = 0 .. 3), tokens 2 ft, 2 ft + 1 of a chunk
        const u32 act_stride = a.act.stride ? a.act.stride : a.act.width;
        const float2 one = both(a.one);
        u32 m = 0;
        for (u32 id = blockIdx.x; id < n_tiles; id += gridDim.x) {
            const Tile t = find_tile(a, cum, n_union, id);
            const u32 n_chunks = t.nt > 8u * w ? (t.nt - 8u * w + 8u * kSplit - 1u) / (8u * kSplit) : 0u;  // chunks w, w + kSplit, ...
            float2 acc[kChunks][4][4];
#pragma unroll
            for (int i = 0; i < (int)kChunks * 16; ++i) (&acc[0][0][0])[i] = make_float2(0.0f, 0.0f);
            for (u32 b = 0; b < nblocks; ++b, ++m) {
                const u32 slot = m % kStages, parity = (m / kStages) & 1u;
                if (ok) ok = mbar_wait(&ready[slot], parity, kWaitLimit, s_abort);
                if (ok) ok = mbar_wait(&raw_full[slot], parity, kWaitLimit, s_abort);  // complete by now: orders the TMA's writes before our reads
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) continue;
                const unsigned char* st = smem + slot * kStageBytes;
                const unsigned char* rows = st + (32u * quarter + fr) * kRowPitch + 16u + 8u * ft;
                const unsigned char* codes = st + kRawBytes + (8u * w + fr) * kCodePitch + 8u * ft;
                const float4* es = reinterpret_cast<const float4*>(st + kRawBytes + kCodeBytes) + 4u * w + ft;
                const float4* fac = reinterpret_cast<const float4*>(st + kRawBytes + kCodeBytes + kEsBytes) + 8u * quarter + fr;
                if (n_chunks) {
                    if (s_slow[slot * 4u + quarter]) superblock<true>(rows, codes, es, fac, n_chunks, one, acc);
                    else superblock<false>(rows, codes, es, fac, n_chunks, one, acc);
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&empty[slot]);
            }
            // (a0 + a1) + (a2 + a3)
            auto fold = [&](const float2* c, int second) {
                return second ? __fadd_rn(__fadd_rn(c[0].y, c[1].y), __fadd_rn(c[2].y, c[3].y)) : __fadd_rn(__fadd_rn(c[0].x, c[1].x), __fadd_rn(c[2].x, c[3].x));
            };
            if (kDown) {
                if (ok) {
#pragma unroll
                    for (int cz = 0; cz < 2 * (int)kChunks; ++cz) {
                        const u32 tk = 8u * (kSplit * (cz >> 1) + w) + 2u * ft + (cz & 1);
                        if (tk < t.nt) {
                            float* out = a.raw + u64(a.routes.slots[t.eb + tk]) * H + kGM * t.c + 32u * quarter + fr;
#pragma unroll
                            for (int i = 0; i < 4; ++i) out[8 * i] = fold(acc[cz >> 1][i], cz & 1);
                        }
                    }
                }
            } else {
                asm volatile("bar.sync 3, %0;" ::"n"(kConsumers * 32) : "memory");  // the previous tile's epilogue has read s_out
#pragma unroll
                for (int cz = 0; cz < 2 * (int)kChunks; ++cz) {
                    float* out = s_out + (8u * (kSplit * (cz >> 1) + w) + 2u * ft + (cz & 1)) * kOutPitch + 32u * quarter + fr;
#pragma unroll
                    for (int i = 0; i < 4; ++i) out[8 * i] = fold(acc[cz >> 1][i], cz & 1);
                }
                asm volatile("bar.sync 3, %0;" ::"n"(kConsumers * 32) : "memory");
                // SwiGLU + the A8 rule: a task is (token, 32 outputs), two per token; a warp takes the four of two tokens at a time
                for (u32 tk0 = 2u * warp; ok && tk0 < t.nt; tk0 += 2u * kConsumers) {
                    float g[kTasks], u[kTasks], delta[kTasks];
                    int code[kTasks], sum[kTasks];
#pragma unroll
                    for (int i = 0; i < kTasks; ++i) {
                        const float* row = s_out + min(tk0 + (i >> 1), t.nt - 1u) * kOutPitch + 32u * (i & 1) + lane;
                        g[i] = row[0]; u[i] = row[64];
                    }
                    const u32 bad = swiglu_a8(g, u, code, delta, sum);
#pragma unroll
                    for (int i = 0; i < kTasks; ++i) {
                        const u32 tk = tk0 + (i >> 1);
                        if (tk >= t.nt) break;
                        const u32 slot = a.routes.slots[t.eb + tk], group = 2u * t.c + (i & 1), o_col = 32u * group + lane;
                        if (a.gate_out) { a.gate_out[u64(slot) * I + o_col] = g[i]; a.up_out[u64(slot) * I + o_col] = u[i]; }
                        if (bad >> i & 1u) {  // fail closed: nothing of the group is written (routed_expert.cpp:147-156)
                            if (lane == 0) {
                                if (a.row_status) atomicOr(&a.row_status[a.routes.rows[t.eb + tk]], B200MOE_ROW_PROJECTION_NONFINITE);
                                if (a.summary) atomicOr(a.summary, B200MOE_ROW_PROJECTION_NONFINITE);
                            }
                            continue;
                        }
                        a.act.codes[u64(slot) * act_stride + o_col] = static_cast<i8>(code[i]);
                        if (lane == 0) {
                            a.act.deltas[u64(slot) * (act_stride / 32) + group] = delta[i];
                            if (a.act.sums) a.act.sums[u64(slot) * (act_stride / 32) + group] = sum[i];
                        }
                    }
                }
            }
        }
    }
    if (!ok && lane == 0 && a.summary) atomicOr(a.summary, kAbortBit);
}

// Tensor map of a [rows][row_bytes] byte tensor with boxes of kRowPitch bytes x 64 rows (no swizzle, no interleave). The
// encoder is the driver's cuTensorMapEncodeTiled, looked up through the runtime (no link against the driver library).
int encode_rows_map(const u8* base, u64 row_bytes, u64 rows, CUtensorMap* out) {
    typedef CUresult (*EncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                 const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static EncodeFn fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q{};
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) p = nullptr;
        return reinterpret_cast<EncodeFn>(p);
    }();
    if (!fn) return fail(B200MOE_ERR_CUDA, "grouped: cuTensorMapEncodeTiled is not available from this driver");
    const cuuint64_t dims[2] = {row_bytes, rows};
    const cuuint64_t strides[1] = {row_bytes};       // bytes between rows: a multiple of 16 (144 per super-block)
    const cuuint32_t box[2] = {kRowPitch, 64};  // 16 bytes past the super-block: the next one's, or the fill value at the end of a row
    const cuuint32_t elem[2] = {1, 1};
    const CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<u8*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                          CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(B200MOE_ERR_CUDA, "grouped: cuTensorMapEncodeTiled failed (%d)", static_cast<int>(r));
    return B200MOE_OK;
}

bool es_units(const b200moe_a8_rows& x) {
    const u32 stride = x.stride ? x.stride : x.width;
    return stride % 128 == 0 && aligned(x.deltas, 16) && aligned(x.sums, 16);
}

bool grouped_shape_ok(const b200moe_shape& s) {
    return s.gate_type == B200MOE_TYPE_Q4_K && s.down_type == B200MOE_TYPE_Q4_K && s.hidden % 256 == 0 && s.inter % 256 == 0 &&
           s.hidden % kGM == 0 && s.inter % 64 == 0 && s.experts <= kMaxUnion;
}

int grid_size() {
    int dev = 0, n = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n;
}

}  // namespace

bool grouped_fits(const b200moe_shape& s, bool have_sums) { return have_sums && grouped_shape_ok(s); }

int launch_gate_up_q4k_grouped(const b200moe_gate_up_view& v, cudaStream_t stream) {
    if (v.max_union == 0) return B200MOE_OK;
    GroupedArgs a{};
    a.shape = v.shape; a.routes = v.routes; a.in = v.x; a.act = v.act;
    a.gate_out = v.gate_out; a.up_out = v.up_out; a.row_status = v.row_status; a.summary = v.summary;
    a.n_row_tiles = v.shape.inter / 64; a.K = v.shape.hidden; a.one = 1.0f; a.es_vec = es_units(v.x);
    CUtensorMap tm0, tm1;
    const u64 rb = u64(v.shape.hidden / 256) * kQ4KBlock, rows = u64(v.shape.experts) * v.shape.inter;
    if (int rc = encode_rows_map(v.weights.gate, rb, rows, &tm0)) return rc;
    if (int rc = encode_rows_map(v.weights.up, rb, rows, &tm1)) return rc;
    if (int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(grouped_q4k_kernel<false>), kGroupedSmem)) return rc;
    grouped_q4k_kernel<false><<<grid_size(), kGThreads, kGroupedSmem, stream>>>(tm0, tm1, a);
    return after_launch("gate_up_q4k_grouped");
}

int launch_down_q4k_grouped(const b200moe_down_view& v, cudaStream_t stream) {
    if (v.max_union == 0) return B200MOE_OK;
    GroupedArgs a{};
    a.shape = v.shape; a.routes = v.routes; a.in = v.act; a.raw = v.raw;
    a.summary = const_cast<u32*>(v.summary);
    a.n_row_tiles = v.shape.hidden / kGM; a.K = v.shape.inter; a.one = 1.0f; a.es_vec = es_units(v.act);
    CUtensorMap tm0;
    if (int rc = encode_rows_map(v.weights.down, u64(v.shape.inter / 256) * kQ4KBlock, u64(v.shape.experts) * v.shape.hidden, &tm0)) return rc;
    if (int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(grouped_q4k_kernel<true>), kGroupedSmem)) return rc;
    grouped_q4k_kernel<true><<<grid_size(), kGThreads, kGroupedSmem, stream>>>(tm0, tm0, a);
    return after_launch("down_q4k_grouped");
}

}  // namespace b200moe
