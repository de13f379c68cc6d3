// Routed experts, Qwen A8 family, decode form for ANY row length: a persistent kernel that streams SEGMENTS of the
// weight rows - and of the activations they meet - through shared memory with the TMA engine.
//
// Same arithmetic as gemv_q4k.cu (the contract of src/cpu/core/routed_expert.hpp:9-15, bit for bit). What this form adds
// over gemv_q4k_stream.cu is that nothing is sized by the row length or by the window: hidden 7168 (4032-byte gate rows),
// inter 17408 (9792-byte down rows) and 64-row windows stream exactly like the small layers.
//
//  * Work item = (virtual expert, 64 weight rows): 32 gate + 32 up rows of one output group, or 64 down rows. A virtual
//    expert is an expert of the window's union with at most kKE = 8 of its entries; an expert with more entries appears
//    several times (its rows are then streamed again, out of L2). Every CTA builds the same virtual list in shared memory
//    from the routes, ordered by entry count (longest items first); the items are dealt out over the whole grid through a
//    claim word in device memory (wide_common.cuh).
//  * A stage = S = 3 super-blocks of the item's 64 rows (one or two tiled TMA copies of 432 bytes x 32 / 64 rows: the rows
//    lie 432 bytes apart in shared memory, an odd count of 16-byte units, which keeps the 128-bit reads of eight rows
//    conflict free) PLUS the same K range of the A8 rows of the item's entries (codes, deltas, sums: three bulk copies per
//    entry, or 16-byte asynchronous copies), all counted on one mbarrier. The consumers therefore find everything a stage needs in shared memory.
//  * Two groups of eight consumer warps share a CTA, each with its own ring of stages and its own producer warp; a group's
//    producer claims the next item of the grid while its consumers still work on the stages in the ring. The serial chains
//    acc_p += pair_p never leave their lane.
//  * Two forms of the integer dots, chosen per item by its entry count. One entry: dp4a, lane = (pair p, one of the warp's 8 rows); (a0 + a1) +
//    (a2 + a3) is two xor-shuffles at the end of the item. From two entries: mma.sync.m16n8k32 (A = nibbles of 16 rows as unsigned bytes, the high ones
//    left in place as 16 q; B = the codes of up to 8 entries, signed), a warp 32 rows of ONE chain; the four chains meet in shared memory at the end of
//    the item. With up to 4 entries the eight columns hold them twice, and a lane works for one of the two row tiles only. The row pair of a lane's
//    cells shares every packed FP32 instruction; both forms produce the contract's bits.
//  * gate/up: the group meets on an mbarrier once per item and a warp an entry runs SwiGLU + the A8 rule; down: a warp an entry stores the sums.
// What bounds it: the latency of dependent instructions with four consumer warps a scheduler (64 rows over 64 experts of 7168 -> 2048: 62 % of the issue
// slots, 67 % of the shared memory's cycles, 49 % of the DRAM's). A warp with 8 rows of four chains, whose factors met 8 rows and which took the tensor cores from
// 5 entries and dp4a of up to 4 entries below, read shared memory twice as much: 64 rows of the large layer (256 experts) 880 to 917 us a call, 804 to 855
// now; dense 5120 x 17408, 8 rows, 84.5 and 77.9; 37 rows over 128 experts of 2048 -> 768 112.0 and 109.3. Copies of 144-byte rows (a super-block
// each) into a ring of 4 stages of two super-blocks instead of 2 of three: dense 1 row 49.8 -> 57.5, 8 rows 84.4 -> 98.3.
//
// Every wait is bounded (plan.wait_limit polls): a waiter that runs out raises the CTA's abort flag, every role leaves
// its loops, the producers wait (bounded) for the copies they still have in flight, B200MOE_JOB_WAIT_ABORTED is set in the
// job summary and the kernel returns - the host reads a status, the GPU never hangs.
//
// Roofline: HBM. Algorithmic bytes per item = 64 rows x K / 256 x 144 (+ the entries' A8 bytes).
#include <algorithm>
#include <type_traits>

#include "grouped_common.cuh"
#include "wide_common.cuh"

namespace b200moe {

namespace {
using namespace q4k;
using namespace wide;
using namespace grouped;  // packed FP32

constexpr u32 kItemRows = 64, kHalfRows = 32;           // an item's two halves: gate and up rows (gate/up), or the first and second 32 of 64 down rows
constexpr u32 kDpEntries = 1;                           // items of one entry take dp4a, items with more the tensor cores
constexpr u32 kFewEntries = 4;                          // up to so many a lane of the mma form works for one of the two row tiles only
constexpr u32 kFacFloats = kHalfRows * 4;               // per-warp scratch of the mma form, a super-block: a pair's four factors of 32 rows
constexpr u32 kMeetPitch = 36, kMeetFloats = 4 * 2 * kKE * kMeetPitch;  // [pair][half][entry][32 + 4]: a half warp's stores (8 rows, 4 entry pairs) meet every bank once

constexpr u32 kMaxStages = 8;
struct WidePlan {
    u32 S;              // super-blocks per stage
    u32 nb;             // super-blocks per row
    u32 nseg;           // stages per item
    u32 stages;         // ring depth per group
    u32 w_bytes;        // 64 * S * 144
    u32 x_entry_bytes;  // >= S * 320: codes, deltas, sums of one entry over the stage's K range (+ padding)
    u32 stage_bytes;
    u32 n_chunks;       // items per (virtual) expert
    u32 max_union;      // bound of the union
    u32 n_bound;        // ... that the routes' arrays are known to hold too, or 0
    u32 vmax;           // capacity of the virtual expert list
    u32 wait_limit;
    u32 stall_stage;    // test hook: group 0's producer stops before this stage (0xffffffff: never)
    u32 early;          // routes and weights are complete before the launch in front was admitted (ChainHints)
    u32 dense_rows;     // rows of a dense block: its entries need no routes; 0 otherwise
};

struct WideArgs {
    b200moe_routes routes;
    b200moe_a8_rows in;    // x (gate/up) or the A8 of h (down)
    b200moe_a8_rows act;   // gate/up output
    float* gate_out;
    float* up_out;
    float* raw;            // down output
    u32* row_status;
    u32* summary;
    u32 rows_per_expert;   // weight rows of one expert: inter (gate/up) or hidden (down)
    u32 out_width;         // inter (gate/up) or hidden (down)
    u32 raw_vec;           // raw lies on an 8-byte boundary
};

// Stage geometry for S super-blocks per stage, as compile-time constants: address
// arithmetic on run-time strides was a measurable part of the instructions. Weight rows lie S * 144 bytes apart, S odd: an odd multiple of 4 (mod 32) words, so a
// warp's 128-bit reads of 8 rows and its fragments' word reads are conflict free.
constexpr u32 x_entry_bytes_of(u32 S) {  // codes, deltas, sums of one entry over a stage, padded so that entries lie an odd multiple of
    u32 b = S * 320u;                     // 4 (mod 32) words apart: the fragments' word reads of eight entries meet every bank once
    while ((b / 4) % 8 != 4) b += 16;
    return b;
}
template <u32 S_>
struct Geo {
    static constexpr u32 S = S_;
    static constexpr u32 row_bytes = S * kQ4KBlock, half_bytes = kHalfRows * row_bytes;
    static constexpr u32 w_bytes = 2 * half_bytes;
    static constexpr u32 x_entry_bytes = x_entry_bytes_of(S);
};

// (a0 + a1) + (a2 + a3) over the four pair lanes of a row (lane = 8 * p + row); every lane of the row gets the value.
__device__ __forceinline__ float tree4(float a) {
    a = __fadd_rn(a, __shfl_xor_sync(0xffffffffu, a, 8));
    return __fadd_rn(a, __shfl_xor_sync(0xffffffffu, a, 16));
}

// Decoded factors of one super-block for pair p as the chains use them: D of the even group, D / 16 of the odd one (the high nibbles stay in
// place: their dots come as 16 * dot), and -DM of both. A scale's byte goes behind the exponent of 2^23, less 2^23.
__device__ __forceinline__ float4 pair_factors(const uint4& hdr, u32 p) {
    const float d = half_bits_to_float(hdr.x & 0xffffu), dm = -half_bits_to_float(hdr.x >> 16);
    const u32 sc = p < 2u ? hdr.y & 0x3f3f3f3fu : (hdr.w & 0x0f0f0f0fu) | ((hdr.y >> 2) & 0x30303030u);
    const u32 mn = p < 2u ? hdr.z & 0x3f3f3f3fu : ((hdr.w >> 4) & 0x0f0f0f0fu) | ((hdr.z >> 2) & 0x30303030u);
    const u32 sel = 0x7440u + 2u * (p & 1u);
    auto byte = [](u32 w, u32 s) { return __fsub_rn(__uint_as_float(__byte_perm(w, 0x4b000000u, s)), 8388608.0f); };
    return make_float4(__fmul_rn(d, byte(sc, sel)), __fmul_rn(__fmul_rn(d, 0.0625f), byte(sc, sel + 1u)), __fmul_rn(dm, byte(mn, sel)), __fmul_rn(dm, byte(mn, sel + 1u)));
}

// One stage of one weight row (this lane's pair p of nbk super-blocks, ascending) against one staged A8 row. blk: the row's first
// super-block of the stage; xs: the entry's area of the stage {codes[S * 256], deltas[S * 8], sums[S * 8]}.
template <class G>
__device__ __forceinline__ void stage_row(const unsigned char* blk, u32 nbk, u32 p, const unsigned char* xs, float& acc) {
    constexpr u32 S = G::S;
#pragma unroll
    for (u32 b = 0; b < S; ++b, blk += kQ4KBlock) {
        if (b >= nbk) break;
        const uint4* w = reinterpret_cast<const uint4*>(blk);
        const uint4 hdr = w[0], q0 = w[1 + 2 * p], q1 = w[2 + 2 * p];
        const float4 f = pair_factors(hdr, p);
        const Nibbles n = split_nibbles(q0, q1);
        const uint4* c = reinterpret_cast<const uint4*>(xs + 256u * b + 64u * p);
        const uint4 c0 = c[0], c1 = c[1], c2 = c[2], c3 = c[3];
        const float2 e = *reinterpret_cast<const float2*>(xs + 256u * S + 32u * b + 8u * p);
        const float2 sm = to_float(*reinterpret_cast<const int2*>(xs + 288u * S + 32u * b + 8u * p));
        int l, h;
        dots(n, c0, c1, c2, c3, &l, &h);
        // x = E * ((D * float(dot)) - (DM * S)) for the pair's two groups; f holds -DM, and (-DM) * S = -(DM * S) exactly
        const float sl = __fadd_rn(__fmul_rn(f.x, static_cast<float>(l)), __fmul_rn(f.z, sm.x));
        const float sh = __fadd_rn(__fmul_rn(f.y, static_cast<float>(h)), __fmul_rn(f.w, sm.y));
        acc = __fadd_rn(acc, __fadd_rn(__fmul_rn(e.x, sl), __fmul_rn(e.y, sh)));
    }
}
// ---- the mma form of one stage ---------------------------------------------------------------------------------------
// 16 weight rows x 8 entries x one group: unsigned nibble bytes times signed codes. d[0], d[1]: row lane / 4, entries 2 (lane % 4) and the next; d[2],
// d[3]: row lane / 4 + 8.
__device__ __forceinline__ void mma_u8s8(int (&d)[4], const u32 (&a)[4], u32 mask, u32 b0, u32 b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
        : "r"(a[0] & mask), "r"(a[1] & mask), "r"(a[2] & mask), "r"(a[3] & mask), "r"(b0), "r"(b1), "r"(0));
}
// One stage of the warp's 32 weight rows and chain (pair p) against up to 8 staged A8 rows with tensor-core dots. blk: the half's first row and super-block
// of the stage; fac: the warp's scratch, S x kFacFloats. acc[j][e]: the chain of rows 16 j + lane / 4 and the row 8 further with entry 2 (lane % 4) + e; these two rows
// share every packed instruction. MANY: items of five entries or more. Else the eight columns hold the entries twice, and of a lane's cells the first
// tile's count in lanes with lane % 4 < 2, the second tile's in the others: acc[0] alone is used, and half of the work after the dots falls away.
// Absent entries compute on stale shared memory and are never stored.
// Why 32 rows of one chain, and not 8 rows of four chains as before: what bounds the loop is what it reads from shared memory (128 bytes a clock). A token's
// codes, deltas and sums are read once per 32 rows and a row's factors once per two entries and row pair: 44 (MANY) or 36 wavefronts a warp and super-block
// where the form before took 88; dp4a takes 32 for one entry and 20 more for every further one.
template <bool MANY, class G>
__device__ __forceinline__ void stage_rows_mma(const unsigned char* blk, u32 nbk, u32 p, u32 lane, const unsigned char* xs, float* fac, float2 (&acc)[MANY ? 2 : 1][2]) {
    constexpr u32 x_entry_bytes = G::x_entry_bytes, S = G::S;
    const u32 g = lane >> 2, t = lane & 3u;
    {   // the factors, lane = row: rows i and i + 8 of a tile meet by a shuffle, so that a row pair lies in natural register pairs
        const bool high = lane & 8u;
        float4* put = reinterpret_cast<float4*>(fac) + 8u * (lane >> 4) + (lane & 7u) + (high ? 16u : 0u);  // [tile][row pair]{D, D, D', D'}, then {-DM, -DM, -DM', -DM'}
        __syncwarp();   // the previous stage's readers are done with the scratch
#pragma unroll
        for (u32 b = 0; b < S; ++b) {
            if (b >= nbk) break;
            const float4 f = pair_factors(*reinterpret_cast<const uint4*>(blk + b * kQ4KBlock + lane * G::row_bytes), p);
            const float u = __shfl_xor_sync(0xffffffffu, high ? f.x : f.z, 8), v = __shfl_xor_sync(0xffffffffu, high ? f.y : f.w, 8);
            put[b * (kFacFloats / 4)] = high ? make_float4(u, f.z, v, f.w) : make_float4(f.x, u, f.y, v);
        }
        __syncwarp();
    }
    const unsigned char* rows = blk + g * G::row_bytes + 16u + 32u * p + 4u * t;
    const unsigned char* codes = xs + (MANY ? g : g & 3u) * x_entry_bytes + 64u * p + 4u * t;
    const unsigned char* es = xs + 2u * (MANY ? t : t & 1u) * x_entry_bytes + 256u * S + 8u * p;
    const float4* get = reinterpret_cast<const float4*>(fac) + g;
    const bool second = t >= 2u;  // of the few form
#pragma unroll
    for (u32 b = 0; b < nbk; ++b) {
        u32 a[2][4], bl[2], bh[2];
#pragma unroll
        for (u32 j = 0; j < 2; ++j)
#pragma unroll
            for (u32 i = 0; i < 4; ++i) a[j][i] = *reinterpret_cast<const u32*>(rows + (16u * j + 8u * (i & 1u)) * G::row_bytes + 16u * (i >> 1));
#pragma unroll
        for (u32 i = 0; i < 2; ++i) { bl[i] = *reinterpret_cast<const u32*>(codes + 16u * i); bh[i] = *reinterpret_cast<const u32*>(codes + 32u + 16u * i); }
        float2 E[2], Sg[2];
#pragma unroll
        for (u32 e = 0; e < 2; ++e) {
            E[e] = *reinterpret_cast<const float2*>(es + e * x_entry_bytes);
            Sg[e] = to_float(*reinterpret_cast<const int2*>(es + e * x_entry_bytes + 32u * S));
        }
        int l[2][4], h[2][4];
#pragma unroll
        for (u32 j = 0; j < 2; ++j) {
            mma_u8s8(l[j], a[j], 0x0f0f0f0fu, bl[0], bl[1]);
            mma_u8s8(h[j], a[j], 0xf0f0f0f0u, bh[0], bh[1]);
        }
        if (!MANY) {
#pragma unroll
            for (u32 i = 0; i < 4; ++i) { l[0][i] = second ? l[1][i] : l[0][i]; h[0][i] = second ? h[1][i] : h[0][i]; }
        }
#pragma unroll
        for (u32 j = 0; j < (MANY ? 2u : 1u); ++j) {
            const u32 tile = MANY ? j : (second ? 1u : 0u);
            const float4 d4 = get[8u * tile], m4 = get[8u * tile + 16u];
            const float2 Dl = make_float2(d4.x, d4.y), Dh = make_float2(d4.z, d4.w), Ml = make_float2(m4.x, m4.y), Mh = make_float2(m4.z, m4.w);
#pragma unroll
            for (u32 e = 0; e < 2; ++e) {
                const float2 sl = add2(mul2(Dl, to_float(make_int2(l[j][e], l[j][e + 2]))), mul2(Ml, both(Sg[e].x)));
                const float2 sh = add2(mul2(Dh, to_float(make_int2(h[j][e], h[j][e + 2]))), mul2(Mh, both(Sg[e].y)));
                acc[j][e] = add2(add2(mul2(both(E[e].x), sl), mul2(both(E[e].y), sh)), acc[j][e]);
            }
        }
        rows += kQ4KBlock; codes += 256; es += 32; get += kFacFloats / 4;
    }
}

// 18 warps: two of the SM's four register partitions (16 K registers each) hold five warps, which caps a thread at
// 16384 / (5 x 32) = 102 registers, 96 after rounding - what this launch bound gives (112 was tried: the launch is refused).
// ASYNC: how the entries' A8 rows come in. A bulk copy holds the producer for about 180 clocks, 24 of them a stage for eight entries; asynchronous copies cost
// instructions that a stage of few entries does not repay. Bulk and asynchronous, us a call: dense 5120 x 17408, 8 rows 77.8 and 74.8, 16 rows 112.5 and
// 109.7, 5 rows 70.8 and 72.7, 1 row 43.9 and 50. A choice per item inside one kernel costs the items of one entry 1.5 us of these 43.9.
template <bool DOWN, u32 S_, bool ASYNC>
__global__ void __launch_bounds__(kThreads, 1)
q4k_wide_kernel(const __grid_constant__ CUtensorMap tm0, const __grid_constant__ CUtensorMap tm1, WideArgs a, WidePlan plan) {
    using G = Geo<S_>;
    extern __shared__ __align__(128) unsigned char smem[];
    // An early launch makes its list and asks for the weights of its groups' first items before it waits for the launch in front. Every path waits.
    const bool early = plan.early;
    u32* claim = a.routes.counts + 3;  // the grid's claim word (wide_common.cuh)

    unsigned char* at = smem + kGroups * plan.stages * plan.stage_bytes;
    float* s_meet = reinterpret_cast<float*>(at);  // [group][kMeetFloats]: an item's chains
    at += kGroups * kMeetFloats * 4;
    VExpert* table = reinterpret_cast<VExpert*>(at);
    at += (u64(plan.vmax) * sizeof(VExpert) + 15) & ~u64(15);  // what follows holds 8- and 16-byte objects
    float* s_fac = reinterpret_cast<float*>(at);  // [consumer warp][S][kFacFloats]
    at += kConsumerWarps * S_ * kFacFloats * 4;
    u64* full = reinterpret_cast<u64*>(at);
    u64* empty = full + kGroups * plan.stages;
    u64* met = empty + kGroups * plan.stages;  // a group's item: its chains are there
    u64* left = met + kGroups;                 // ... and have been read
    at += (2 * kGroups * plan.stages + 2 * kGroups) * 8;
    u32* slot_item = reinterpret_cast<u32*>(at);
    at += kGroups * plan.stages * 4;
    u32* ctl = reinterpret_cast<u32*>(at);  // [0] abort flag, [1] producers that have retired, [2] virtual experts, [3] items
    volatile u32* abort_flag = ctl;

    const u32 tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    if (tid < kGroups * plan.stages) { mbar_init(&full[tid], 1); mbar_init(&empty[tid], kGroupWarps); }
    if (tid < 2 * kGroups) mbar_init(&met[tid], kGroupWarps);
    if (tid < 2) ctl[tid] = 0;  // the list's builder writes the others, and for a dense block there is no barrier between here and there
    if (tid < kGroups * plan.stages + 2 * kGroups) asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");

    if (!early) chain_begin();
    if (DOWN && !early && block_skips(a.summary)) return;  // a failed or aborted projection skips the whole stage (routed_expert.hpp:17-19)

    // ---- the virtual expert list (the stage area is free until the first copy is issued: it holds the copied routes)
    if (plan.dense_rows) build_dense_list(plan.dense_rows, plan.n_chunks, table, ctl);
    else build_work_list(a.routes, plan.n_bound ? plan.n_bound : min(load_l2(a.routes.counts), plan.max_union), plan.max_union, plan.vmax, plan.n_chunks, reinterpret_cast<u32*>(smem), table, ctl);
    const u32 n_items = ctl[3];
    if (n_items == 0) {  // every CTA alike: nobody claims, the claim word stays zero
        if (early) chain_begin();
        return;
    }

    // ------------------------------------------------------------------------------------------ producer warps
    if (warp >= kConsumerWarps) {
        const u32 g = warp - kConsumerWarps;
        u64* g_full = full + g * plan.stages;
        u64* g_empty = empty + g * plan.stages;
        u32* g_item = slot_item + g * plan.stages;
        unsigned char* g_stage = smem + g * plan.stages * plan.stage_bytes;
        const u32 e = lane / 3u, part = lane - 3u * e;  // bulk copies: lanes 0 .. 3 * ne - 1 copy one piece of one entry each
        const u32 in_stride = a.in.stride ? a.in.stride : a.in.width, in_gs = in_stride / 32;
        u32 t = 0, slot = 0, use = 0;  // stage count, ring position, lap
        bool ok = true, first = true;
        // ASYNC: 16-byte asynchronous copies, 20 units a super-block and entry {16 of codes, 2 of deltas, 2 of sums}; a lane takes units `lane` and `lane` + 32 of every entry.
        auto copy_entries = [&](u32 s, u32 nbk, u32 ne, u32 my_row, unsigned char* xd) {
#pragma unroll
            for (u32 half = 0; half < (20u * G::S + 31u) / 32u; ++half) {
                const u32 u = lane + 32u * half;
                const bool is_codes = u < 16u * nbk, is_deltas = u < 18u * nbk;
                const unsigned char* base = is_codes ? reinterpret_cast<const unsigned char*>(a.in.codes) + s * G::S * 256u + 16u * u
                                          : is_deltas ? reinterpret_cast<const unsigned char*>(a.in.deltas) + s * G::S * 32u + 16u * (u - 16u * nbk)
                                                      : reinterpret_cast<const unsigned char*>(a.in.sums) + s * G::S * 32u + 16u * (u - 18u * nbk);
                const u32 pitch = is_codes ? in_stride : in_stride / 8u;  // bytes between rows
                unsigned char* to = xd + (is_codes ? 16u * u : is_deltas ? 256u * G::S + 16u * (u - 16u * nbk) : 288u * G::S + 16u * (u - 18u * nbk));
                for (u32 e = 0; e < ne; ++e) {
                    const u32 row = __shfl_sync(0xffffffffu, my_row, e);
                    if (u < 20u * nbk) cp_async16(to + e * G::x_entry_bytes, base + u64(row) * pitch);
                }
            }
        };
        auto ask_weights = [&](u32 s, const VExpert& ve, u32 chunk, unsigned char* dst, u64* bar) {  // one lane
            const u32 x = s * G::S * (kQ4KBlock / 8);  // 64-bit elements: a multiple of 18, i.e. of 144 bytes
            const u32 y = ve.expert() * a.rows_per_expert + (DOWN ? kItemRows : kHalfRows) * chunk;
            tma_2d(dst, &tm0, x, y, bar);
            tma_2d(dst + G::half_bytes, &tm1, x, DOWN ? y + kHalfRows : y, bar);
        };
        u32 ahead = 0;  // stages of the first item whose weights were asked for before the wait
        if (early) {
            const u32 k = g * gridDim.x + blockIdx.x;
            if (k < n_items) {
                ahead = min(plan.nseg, plan.stages);
                if (g == 0) ahead = min(ahead, plan.stall_stage);
                if (lane == 0) {
                    const u32 jv = k / plan.n_chunks;
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the list was made in the stages' memory
                    for (u32 s = 0; s < ahead; ++s) {
                        mbar_expect_more(&g_full[s], G::w_bytes);
                        ask_weights(s, table[jv], k - jv * plan.n_chunks, g_stage + s * plan.stage_bytes, &g_full[s]);
                    }
                }
            }
            chain_begin();
            if (DOWN && a.summary && *a.summary) {  // the stage is skipped: the weights land (the wait is bounded) before the CTA retires
                if (lane == 0) {
                    for (u32 s = 0; s < ahead; ++s) mbar_arrive(&g_full[s]);
                    for (u32 s = 0; s < ahead; ++s)
                        for (u32 i = 0; i < (plan.wait_limit >> 4) + 64u; ++i)
                            if (mbar_try_wait(&g_full[s], 0)) break;
                }
                return;
            }
        }
        for (;;) {
            // A group's first item needs no round trip: group 0 of CTA b takes item b, group 1 item gridDim.x + b - so a
            // launch with fewer items than groups runs one group per SM, which has the SM's issue slots to itself.
            u32 k = g * gridDim.x + blockIdx.x;
            if (!first) {
                if (lane == 0) k = gridDim.x * kGroups + claim_item(claim);
                k = __shfl_sync(0xffffffffu, k, 0);
            }
            first = false;
            const bool end = k >= n_items;
            const u32 item = k;
            VExpert ve{0};
            u32 chunk = 0;
            if (!end) {
                const u32 jv = item / plan.n_chunks;
                chunk = item - jv * plan.n_chunks;
                ve = table[jv];
            }
            const u32 ve_ne = ve.ne();
            const u32 mine = ASYNC ? lane : e;  // the entry whose row the lane reads
            u32 r = 0;
            if (mine < ve_ne) r = plan.dense_rows ? ve.begin() + mine : load((DOWN ? a.routes.slots : a.routes.rows) + ve.begin() + mine);
            const u32 nsegs = end ? 1u : plan.nseg;
            for (u32 s = 0; s < nsegs; ++s, ++t, ++slot) {
                if (slot == plan.stages) { slot = 0; ++use; }
                if (use) ok = mbar_wait(&g_empty[slot], (use - 1u) & 1u, plan.wait_limit, abort_flag);  // the slot's previous use is done
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                if (g == 0 && t == plan.stall_stage) { ok = false; break; }  // test hook: stop feeding, raise nothing
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the consumers' reads precede the copies below
                if (end) {
                    if (lane == 0) { g_item[slot] = kEndItem; mbar_arrive(&g_full[slot]); }
                    continue;
                }
                const u32 nbk = min(G::S, plan.nb - s * G::S);
                unsigned char* dst = g_stage + slot * plan.stage_bytes;
                if (lane == 0) {
                    g_item[slot] = item;
                    const u32 w_bytes = t < ahead ? 0u : G::w_bytes;  // whole boxes: what lies past the row is filled
                    if (ASYNC) mbar_expect_more(&g_full[slot], w_bytes);
                    else mbar_expect_tx(&g_full[slot], w_bytes + ve_ne * nbk * 320u);
                }
                __syncwarp();
                if (lane == 0 && t >= ahead) ask_weights(s, ve, chunk, dst, &g_full[slot]);
                if (ASYNC) {  // the arrival that lets the stage complete comes behind the lanes' copies, each of which adds one of its own while it is under way
                    copy_entries(s, nbk, ve_ne, r, dst + G::w_bytes);
                    asm volatile("cp.async.mbarrier.arrive.shared::cta.b64 [%0];" ::"r"(saddr(&g_full[slot])) : "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&g_full[slot]);
                } else if (e < ve_ne) {
                    unsigned char* xd = dst + G::w_bytes + e * G::x_entry_bytes;
                    if (part == 0) bulk_g2s(xd, a.in.codes + u64(r) * in_stride + u64(s) * G::S * 256u, nbk * 256u, &g_full[slot]);
                    else if (part == 1) bulk_g2s(xd + 256u * G::S, a.in.deltas + u64(r) * in_gs + u64(s) * G::S * 8u, nbk * 32u, &g_full[slot]);
                    else bulk_g2s(xd + 288u * G::S, a.in.sums + u64(r) * in_gs + u64(s) * G::S * 8u, nbk * 32u, &g_full[slot]);
                }
            }
            if (!ok || end) break;
        }
        if (ASYNC) asm volatile("cp.async.wait_all;" ::: "memory");
        if (!ok && lane == 0) {  // wait (bounded) for the copies still in flight before the CTA retires
            for (u32 n = t > plan.stages ? t - plan.stages : 0u; n < t; ++n)
                for (u32 i = 0; i < (plan.wait_limit >> 4) + 64u; ++i)
                    if (mbar_try_wait(&g_full[n % plan.stages], (n / plan.stages) & 1u)) break;
        }
        if (lane == 0) retire_claims(claim, ctl);
        return;
    }

    // ------------------------------------------------------------------------------------------ consumer warps
    if (early) {
        chain_begin();
        if (DOWN && a.summary && *a.summary) return;
    }
    const u32 g = warp / kGroupWarps, w = warp % kGroupWarps;
    const u32 p = lane >> 3, rr = lane & 7u;     // dp4a form: lane = (pair, one of the warp's 8 rows)
    const u32 mp = w & 3u, half = w >> 2;        // mma form: the warp's chain and half of the item
    const u32 me = lane >> 2, mt = lane & 3u;
    float* fac = s_fac + warp * (S_ * kFacFloats);
    float* meet = s_meet + g * kMeetFloats;
    u64* g_full = full + g * plan.stages;
    u64* g_empty = empty + g * plan.stages;
    const u32* g_item = slot_item + g * plan.stages;
    const unsigned char* g_stage = smem + g * plan.stages * plan.stage_bytes;
    const u32 act_stride = DOWN ? 0u : (a.act.stride ? a.act.stride : a.act.width);
    u32 slot = 0, phase = 0, kl = 0;  // ring position of the group's next stage, kept incrementally (no divisions in the loop); meetings so far
    bool ok = true;
    for (;;) {
        ok = mbar_wait(&g_full[slot], phase, plan.wait_limit, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        const u32 item = g_item[slot];
        if (item == kEndItem) break;
        const u32 jv = item / plan.n_chunks, chunk = item - jv * plan.n_chunks;
        const VExpert ve = table[jv];
        const u32 ne = ve.ne(), vbegin = ve.begin();
        const bool mma = ne > kDpEntries;
        const u32 slot_id = w >= ne ? 0u : plan.dense_rows ? vbegin + w : load(a.routes.slots + vbegin + w);  // asked for before the stages, used behind them
        // the item's stages, with the form fixed at compile time inside the loop
        auto stages = [&](auto step) {
            for (u32 s = 0; s < plan.nseg; ++s) {
                if (s) {
                    ok = mbar_wait(&g_full[slot], phase, plan.wait_limit, abort_flag);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) return;
                }
                const unsigned char* st = g_stage + slot * plan.stage_bytes;
                step(st, min(G::S, plan.nb - s * G::S));
                __syncwarp();
                if (lane == 0) mbar_arrive(&g_empty[slot]);  // the stage is free for the producer
                if (++slot == plan.stages) { slot = 0; phase ^= 1u; }
            }
        };
        // the chains meet in shared memory, once the previous item's have been read
        auto hand_over = [&](auto store) {
            if (kl) ok = mbar_wait(&left[g], (kl - 1u) & 1u, plan.wait_limit, abort_flag);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) return;
            store();
            __syncwarp();
            if (lane == 0) mbar_arrive(&met[g]);
            ok = mbar_wait(&met[g], kl & 1u, plan.wait_limit, abort_flag);
            ok = __all_sync(0xffffffffu, ok);
        };
        auto run_mma = [&](auto many) {
            constexpr bool MANY = decltype(many)::value;
            float2 acc[MANY ? 2 : 1][2];
#pragma unroll
            for (u32 j = 0; j < (MANY ? 2u : 1u); ++j) { acc[j][0] = make_float2(0.0f, 0.0f); acc[j][1] = make_float2(0.0f, 0.0f); }
            stages([&](const unsigned char* st, u32 nbk) { stage_rows_mma<MANY, G>(st + half * G::half_bytes, nbk, mp, lane, st + G::w_bytes, fac, acc); });
            if (!ok) return;
            hand_over([&]() {
#pragma unroll
                for (u32 j = 0; j < (MANY ? 2u : 1u); ++j)
#pragma unroll
                    for (u32 e = 0; e < 2; ++e) {
                        const u32 tile = MANY ? j : mt >> 1, entry = 2u * (MANY ? mt : mt & 1u) + e;
                        float* to = meet + ((2u * mp + half) * kKE + entry) * kMeetPitch + 16u * tile + me;
                        to[0] = acc[j][e].x;
                        to[8] = acc[j][e].y;
                    }
            });
        };
        if (!mma) {
            const u32 only_slot = !DOWN ? 0u : plan.dense_rows ? vbegin : load(a.routes.slots + vbegin);
            float acc = 0.0f;
            stages([&](const unsigned char* st, u32 nbk) { stage_row<G>(st + half * G::half_bytes + (8u * mp + rr) * G::row_bytes, nbk, p, st + G::w_bytes, acc); });
            if (!ok) break;
            const float val = tree4(acc);
            if (DOWN) {
                if (p == 0) a.raw[u64(only_slot) * a.out_width + kItemRows * chunk + 8u * w + rr] = val;
                continue;
            }
            hand_over([&]() { if (p == 0) meet[half * kKE * kMeetPitch + 8u * mp + rr] = val; });
        } else if (ne > kFewEntries) {
            run_mma(std::true_type{});
        } else {
            run_mma(std::false_type{});
        }
        if (!ok) break;
        if (w < ne) {
            const float* mine = meet + w * kMeetPitch;
            constexpr u32 kHalf = kKE * kMeetPitch, kPair = 2 * kHalf;
            if (DOWN) {  // two neighbouring outputs of entry w a lane
                float2 c[4];
#pragma unroll
                for (u32 i = 0; i < 4; ++i) c[i] = *reinterpret_cast<const float2*>(mine + i * kPair + (lane >> 4) * kHalf + 2u * (lane & 15u));
                const float v0 = __fadd_rn(__fadd_rn(c[0].x, c[1].x), __fadd_rn(c[2].x, c[3].x)), v1 = __fadd_rn(__fadd_rn(c[0].y, c[1].y), __fadd_rn(c[2].y, c[3].y));
                float* dst = a.raw + u64(slot_id) * a.out_width + kItemRows * chunk + 2u * lane;
                if (a.raw_vec) *reinterpret_cast<float2*>(dst) = make_float2(v0, v1);
                else { dst[0] = v0; dst[1] = v1; }
            } else {  // SwiGLU + the A8 rule over the 32 outputs of entry w
                float gv = mine[lane], uv = mine[kHalf + lane];
                if (mma) {
                    gv = __fadd_rn(__fadd_rn(gv, mine[kPair + lane]), __fadd_rn(mine[2 * kPair + lane], mine[3 * kPair + lane]));
                    uv = __fadd_rn(__fadd_rn(uv, mine[kPair + kHalf + lane]), __fadd_rn(mine[2 * kPair + kHalf + lane], mine[3 * kPair + kHalf + lane]));
                }
                const u32 o_col = 32u * chunk + lane;
                if (a.gate_out) { a.gate_out[u64(slot_id) * a.out_width + o_col] = gv; a.up_out[u64(slot_id) * a.out_width + o_col] = uv; }
                const float h = swiglu_qwen(gv, uv);
                const bool bad = __any_sync(0xffffffffu, !finite_f(gv) || !finite_f(uv) || !finite_f(h));
                if (bad) {  // fail closed: nothing of the group is written (routed_expert.cpp:147-156)
                    if (lane == 0) {
                        if (a.row_status) atomicOr(&a.row_status[plan.dense_rows ? vbegin + w : load(a.routes.rows + vbegin + w)], B200MOE_ROW_PROJECTION_NONFINITE);
                        if (a.summary) atomicOr(a.summary, B200MOE_ROW_PROJECTION_NONFINITE);
                    }
                } else {
                    float delta;
                    int sum;
                    const int code = a8_quantize_lane(h, &delta, &sum);
                    a.act.codes[u64(slot_id) * act_stride + o_col] = static_cast<i8>(code);
                    if (lane == 0) {
                        a.act.deltas[u64(slot_id) * (act_stride / 32) + chunk] = delta;
                        if (a.act.sums) a.act.sums[u64(slot_id) * (act_stride / 32) + chunk] = sum;
                    }
                }
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&left[g]);
        ++kl;
    }
    if (!ok && lane == 0 && a.summary) atomicOr(a.summary, kAbortBit);
}

u32 round_up(u32 v, u32 a) { return (v + a - 1) / a * a; }

u32 fixed_smem(const WidePlan& p) {
    return kGroups * kMeetFloats * 4 + round_up(p.vmax * static_cast<u32>(sizeof(VExpert)), 16) + kConsumerWarps * p.S * kFacFloats * 4 +
           (2 * kGroups * p.stages + 2 * kGroups) * 8 + kGroups * p.stages * 4 + 64;
}
u32 plan_smem(const WidePlan& p) { return kGroups * p.stages * p.stage_bytes + fixed_smem(p); }

// K: the row length; n_chunks: items per expert; slots: rows * top_k of the window. False when the form does not apply.
bool make_plan(u32 K, u32 n_chunks, u32 max_union, u64 slots, WidePlan* p) {
    if (K == 0 || K % 256 || max_union == 0 || slots == 0 || slots > 8192) return false;
    p->nb = K / 256;
    p->S = p->nb >= 3 ? 3u : 1u;  // odd: see Geo
    p->nseg = (p->nb + p->S - 1) / p->S;
    p->w_bytes = kItemRows * p->S * kQ4KBlock;
    p->x_entry_bytes = x_entry_bytes_of(p->S);
    // a stage holds the A8 segments of as many entries as a virtual expert of this window can have: windows of fewer than
    // kKE slots get smaller stages and with them a deeper ring
    p->stage_bytes = round_up(p->w_bytes + static_cast<u32>(std::min<u64>(kKE, slots)) * p->x_entry_bytes, 128);
    p->n_chunks = n_chunks;
    p->max_union = max_union;
    p->vmax = max_union + static_cast<u32>(slots / kKE) + 1;
    if (u64(p->vmax) * n_chunks + 4096 >= kClaimMask) return false;  // items and the groups' closing claims fit the claim word's count
    for (p->stages = kMaxStages; p->stages >= 2; --p->stages)
        if (plan_smem(*p) <= kSmemBudget) break;
    if (p->stages < 2) return false;
    if (work_list_scratch_words(max_union, p->vmax) * 4 > kGroups * p->stages * p->stage_bytes) return false;  // the work list is built in the stage area
    p->wait_limit = kDefaultWaitLimit;
    p->stall_stage = 0xffffffffu;
    return true;
}

// The entries' A8 rows are moved by bulk copies: 16-byte aligned sources at every (row, stage) offset.
bool a8_bulk_ok(const b200moe_a8_rows& x) {
    const u32 stride = x.stride ? x.stride : x.width;
    return x.sums && aligned(x.codes, 16) && aligned(x.deltas, 16) && aligned(x.sums, 16) && stride % 128 == 0;
}

// Windows whose experts have kKE entries or more on average: their A8 rows come in by asynchronous copies (the figures are with the kernel).
bool whole_items(u32 max_union, u64 slots) { return slots >= u64(kKE) * max_union; }

void apply_hooks(WidePlan* p) {
    const u32 limit = debug_value(B200MOE_DEBUG_WAIT_LIMIT), stall = debug_value(B200MOE_DEBUG_STALL_STAGE);
    if (limit) p->wait_limit = limit;
    if (stall) p->stall_stage = stall - 1u;
}

}  // namespace

bool wide_gate_up_fits(const b200moe_gate_up_view& v, u32 rows) {
    WidePlan p{};
    return v.shape.gate_type == B200MOE_TYPE_Q4_K && rows && a8_bulk_ok(v.x) && v.shape.inter % 32 == 0 &&
           make_plan(v.shape.hidden, v.shape.inter / 32, v.max_union, u64(rows) * v.shape.top_k, &p);
}
bool wide_down_fits(const b200moe_down_view& v, u32 rows) {
    WidePlan p{};
    return v.shape.down_type == B200MOE_TYPE_Q4_K && rows && a8_bulk_ok(v.act) && v.shape.hidden % 64 == 0 &&
           make_plan(v.shape.inter, v.shape.hidden / 64, v.max_union, u64(rows) * v.shape.top_k, &p);
}

int launch_gate_up_q4k_wide(const b200moe_gate_up_view& v, u32 rows, const ChainHints& hints, cudaStream_t stream) {
    if (v.max_union == 0) return B200MOE_OK;
    WidePlan p{};
    if (!make_plan(v.shape.hidden, v.shape.inter / 32, v.max_union, u64(rows) * v.shape.top_k, &p))
        return fail(B200MOE_ERR_UNSUPPORTED, "gate_up: the segment-streaming form does not apply to this shape");
    apply_hooks(&p);
    p.early = hints.routes_done || hints.dense_rows; p.dense_rows = hints.dense_rows; p.n_bound = static_cast<u32>(std::min<u64>(v.max_union, hints.slots));
    WideArgs a{};
    a.routes = v.routes; a.in = v.x; a.act = v.act; a.gate_out = v.gate_out; a.up_out = v.up_out;
    a.row_status = v.row_status; a.summary = v.summary; a.rows_per_expert = v.shape.inter; a.out_width = v.shape.inter;
    CUtensorMap tm0, tm1;
    const u64 rb = u64(p.nb) * kQ4KBlock, total_rows = u64(v.shape.experts) * v.shape.inter;
    if (int rc = rows_map(v.weights.gate, rb, total_rows, p.S * kQ4KBlock, kHalfRows, &tm0)) return rc;
    if (int rc = rows_map(v.weights.up, rb, total_rows, p.S * kQ4KBlock, kHalfRows, &tm1)) return rc;
    const u32 smem = plan_smem(p);
    const auto kernel = p.S != 3 ? q4k_wide_kernel<false, 1, false> : whole_items(v.max_union, u64(rows) * v.shape.top_k) ? q4k_wide_kernel<false, 3, true> : q4k_wide_kernel<false, 3, false>;
    if (int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), smem)) return rc;
    chain_launch(kernel, device_sm_count(), kThreads, smem, stream, tm0, tm1, a, p);
    return after_launch("gate_up_q4k_wide");
}

int launch_down_q4k_wide(const b200moe_down_view& v, u32 rows, const ChainHints& hints, cudaStream_t stream) {
    if (v.max_union == 0) return B200MOE_OK;
    WidePlan p{};
    if (!make_plan(v.shape.inter, v.shape.hidden / 64, v.max_union, u64(rows) * v.shape.top_k, &p))
        return fail(B200MOE_ERR_UNSUPPORTED, "down: the segment-streaming form does not apply to this shape");
    apply_hooks(&p);
    p.early = hints.routes_done || hints.dense_rows; p.dense_rows = hints.dense_rows; p.n_bound = static_cast<u32>(std::min<u64>(v.max_union, hints.slots));
    WideArgs a{};
    a.routes = v.routes; a.in = v.act; a.raw = v.raw; a.summary = const_cast<u32*>(v.summary);
    a.rows_per_expert = v.shape.hidden; a.out_width = v.shape.hidden; a.raw_vec = aligned(v.raw, 8);
    CUtensorMap tm0;
    if (int rc = rows_map(v.weights.down, u64(p.nb) * kQ4KBlock, u64(v.shape.experts) * v.shape.hidden, p.S * kQ4KBlock, kHalfRows, &tm0)) return rc;
    const u32 smem = plan_smem(p);
    const auto kernel = p.S != 3 ? q4k_wide_kernel<true, 1, false> : whole_items(v.max_union, u64(rows) * v.shape.top_k) ? q4k_wide_kernel<true, 3, true> : q4k_wide_kernel<true, 3, false>;
    if (int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), smem)) return rc;
    chain_launch(kernel, device_sm_count(), kThreads, smem, stream, tm0, tm0, a, p);
    return after_launch("down_q4k_wide");
}

}  // namespace b200moe
