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
//    conflict free) PLUS the same K range of the A8 rows of the item's entries (codes, deltas, sums: tiled copies of a dense block's neighbouring
//    rows; otherwise an untiled copy of each entry's codes and 16-byte asynchronous copies of the deltas and sums), all counted on one mbarrier. The consumers therefore find everything a stage needs in shared memory.
//  * Two groups of eight consumer warps share a CTA, each with its own ring of stages and its own producer warp; a group's
//    producer claims the next item of the grid while its consumers still work on the stages in the ring. The serial chains
//    acc_p += pair_p never leave their lane.
//  * Two forms of the integer dots, chosen per item by its entry count. One entry: dp4a, lane = (pair p, one of the warp's 8 rows); (a0 + a1) +
//    (a2 + a3) is two xor-shuffles at the end of the item. From two entries: mma.sync.m16n8k32 (A = nibbles of 16 rows as unsigned bytes, the high ones
//    left in place as 16 q; B = the codes of up to 8 entries, signed), a warp 32 rows of ONE chain; the four chains meet in shared memory at the end of
//    the item. With up to 4 entries the eight columns hold them twice, and a lane works for one of the two row tiles only. The pair's two groups
//    of a cell share every packed FP32 instruction; both forms produce the contract's bits.
//  * Where there are no more items than CTAs (rows of several stages: a dense block's down) an item is both groups': each takes every other stage, makes what its
//    super-blocks add to the chains, gets the chains from the other group, adds in order and hands them on (PAIR).
//  * gate/up: the group meets on an mbarrier once per item and a warp an entry runs SwiGLU + the A8 rule; down: a warp an entry stores the sums.
// What bounds it: the latency of dependent instructions with four consumer warps a scheduler (64 experts of 7168 -> 2048, 64 rows: 64 % of the issue
// slots, 58 % of the shared memory's cycles, 57 % of the DRAM's). Measured forms before: a warp with 8 rows of four chains, whose factors met 8 rows and which took the tensor cores from
// 5 entries and dp4a of up to 4 entries below, read shared memory twice as much (64 rows of the large layer, 256 experts, 880 to 917 us a call, 804 to 855 with 32 rows of one chain; rows, not
// groups, as the lanes of the packed instructions then 725 to 745 in a graph, 680 to 696 now). Copies of 144-byte rows (a super-block each) into a ring of 4 stages of two super-blocks instead
// of 2 of three: dense 5120 x 17408 1 row 49.8 -> 57.5, 8 rows 84.4 -> 98.3.
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
    u32 cap;            // entries that a stage holds: 1, 4 or 8
    u32 stage_bytes;
    u32 boxes;          // the entries' A8 rows are neighbours and come by tiled copies (dense blocks)
    u32 pair;           // an item's stages are shared by the CTA's two groups
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

struct WideMaps { CUtensorMap w0, w1, codes, deltas, sums; };  // weight rows (up: w1), a dense block's A8 rows

// Stage geometry for S super-blocks per stage and CAP entries (1, 4 or 8), as compile-time constants: address arithmetic on run-time strides was a measurable
// part of the instructions. Weight rows lie S * 144 (Q5_K: 176) bytes apart, S odd: an odd multiple of 4 (mod 32) words, so a warp's 128-bit reads of 8 rows and its
// fragments' word reads are conflict free. The entries' codes lie S * 256 + 16 bytes apart, 4 (mod 32) words: eight entries' word reads meet every bank once.
template <u32 S_, u32 CAP_, bool Q5K_ = false>
struct Geo {
    static constexpr bool Q5K = Q5K_;  // 32 bytes of fifth bits lie between a super-block's header and its nibbles
    static constexpr u32 S = S_, CAP = CAP_, block = Q5K ? kQ5KBlock : kQ4KBlock, nibbles = Q5K ? 48u : 16u;
    static constexpr u32 row_bytes = S * block, half_bytes = kHalfRows * row_bytes;
    static constexpr u32 w_bytes = 2 * half_bytes;
    static constexpr u32 box_codes = CAP == 1 ? S * 256u : S * 256u + 16u, box_group = S * 32u;  // bytes of an entry's codes (with their gap), deltas, sums
    static constexpr u32 off_deltas = (CAP * box_codes + 127u) / 128u * 128u, off_sums = off_deltas + CAP * box_group;
    static constexpr u32 x_bytes = off_sums + CAP * box_group;
    static constexpr u32 stage_bytes = (w_bytes + x_bytes + 127u) / 128u * 128u;
    static constexpr u32 boxes_tx = CAP * (box_codes + 2u * box_group);  // what the tiled copies bring: whole boxes, what lies past the tensor is filled
};
template <u32 S, u32 CAP, bool Q5K> constexpr bool lands() {  // a tiled copy lands on 128 bytes
    using G = Geo<S, CAP, Q5K>;
    return G::w_bytes % 128 == 0 && G::half_bytes % 128 == 0 && G::off_deltas % 128 == 0 && G::off_sums % 128 == 0 && G::stage_bytes % 128 == 0;
}
static_assert(lands<3, 8, false>() && lands<3, 4, false>() && lands<1, 8, false>() && lands<1, 4, false>());
static_assert(lands<3, 8, true>() && lands<3, 4, true>() && lands<1, 8, true>() && lands<1, 4, true>());

// (a0 + a1) + (a2 + a3) over the four pair lanes of a row (lane = 8 * p + row); every lane of the row gets the value.
__device__ __forceinline__ float tree4(float a) {
    a = __fadd_rn(a, __shfl_xor_sync(0xffffffffu, a, 8));
    return __fadd_rn(a, __shfl_xor_sync(0xffffffffu, a, 16));
}

// Decoded factors of one super-block for pair p as the chains use them: D of the even group, D of the odd one - of Q4_K D / 16, whose high nibbles stay in
// place: their dots come as 16 * dot -, and -DM of both. A scale's byte goes behind the exponent of 2^23, less 2^23.
template <bool Q5K>
__device__ __forceinline__ float4 pair_factors(const uint4& hdr, u32 p) {
    const float d = half_bits_to_float(hdr.x & 0xffffu), dm = half_bits_to_float(hdr.x >> 16);
    const u32 sel = 0x7440u + 2u * (p & 1u);
    u32 sc, mn;
    if (p < 2u) { sc = hdr.y & 0x3f3f3f3fu; mn = hdr.z & 0x3f3f3f3fu; }
    else { sc = (hdr.w & 0x0f0f0f0fu) | ((hdr.y >> 2) & 0x30303030u); mn = ((hdr.w >> 4) & 0x0f0f0f0fu) | ((hdr.z >> 2) & 0x30303030u); }
    auto two = [&](u32 w, u32 base) { return make_float2(__uint_as_float(__byte_perm(w, base, sel)), __uint_as_float(__byte_perm(w, base, sel + 1u))); };
    const float2 D = mul2(make_float2(d, Q5K ? d : __fmul_rn(d, 0.0625f)), add2(two(sc, 0x4b000000u), both(-8388608.0f)));
    const float2 M = mul2(both(dm), add2(two(mn, 0xcb000000u), both(8388608.0f)));
    return make_float4(D.x, D.y, M.x, M.y);
}

__device__ __forceinline__ uint4 lds128(u32 a) { uint4 v; asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a)); return v; }
__device__ __forceinline__ void sts128(u32 a, const float4& v) { asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" :: "r"(a), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory"); }
// The pair's term of one row and entry: x = E * ((D * float(dot)) - (DM * S)) of its two groups, which share the packed instructions, added. f holds -DM, and
// (-DM) * S = -(DM * S) exactly. The groups, and not two rows or entries, because all operands then lie in natural register pairs: rows paired, whose entry factors
// had to be doubled by moves, took 197 instructions a super-block of 32 rows x 8 entries.
__device__ __forceinline__ float pair_term(const float4& f, int2 dot, float2 E, float2 S) {
    const float2 x = mul2(E, add2(mul2(make_float2(f.x, f.y), to_float(dot)), mul2(make_float2(f.z, f.w), S)));
    return __fadd_rn(x.x, x.y);
}

// Bit j of the four bytes of a word of high bits as bit 4 of four quants.
__device__ __forceinline__ u32 fifth_bits(u32 h, u32 j) { return ((h >> j) << 4) & 0x10101010u; }

// One stage of one weight row (this lane's pair p of nbk super-blocks, ascending) against one staged A8 row. blk: the row's first
// super-block of the stage; xs: the stage's A8 rows, of which the first is meant.
template <class G, class Put>
__device__ __forceinline__ void stage_row(u32 blk, u32 nbk, u32 p, u32 xs, Put put_term) {
    constexpr u32 S = G::S;
    const u32 q = blk + G::nibbles + 32u * p, cs = xs + 64u * p, es = xs + G::off_deltas + 8u * p;
#pragma unroll
    for (u32 b = 0; b < S; ++b) {
        if (b >= nbk) break;
        const uint4 hdr = lds128(blk + b * G::block), q0 = lds128(q + b * G::block), q1 = lds128(q + b * G::block + 16u);
        const float4 f = pair_factors<G::Q5K>(hdr, p);
        Nibbles n = split_nibbles(q0, q1);
        if (G::Q5K) {
            const uint4 h0 = lds128(blk + b * G::block + 16u), h1 = lds128(blk + b * G::block + 32u);
            const u32 h[8] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w};
#pragma unroll
            for (int i = 0; i < 8; ++i) { n.lo[i] |= fifth_bits(h[i], 2u * p); n.hi[i] = (n.hi[i] >> 4) | fifth_bits(h[i], 2u * p + 1u); }
        }
        const uint4 c0 = lds128(cs + 256u * b), c1 = lds128(cs + 256u * b + 16u), c2 = lds128(cs + 256u * b + 32u), c3 = lds128(cs + 256u * b + 48u);
        const uint2 d = lds64(es + 32u * b), m = lds64(es + (G::off_sums - G::off_deltas) + 32u * b);
        int l, h;
        dots(n, c0, c1, c2, c3, &l, &h);
        put_term(b, 0, pair_term(f, make_int2(l, h), make_float2(__uint_as_float(d.x), __uint_as_float(d.y)), to_float(make_int2(static_cast<int>(m.x), static_cast<int>(m.y)))));
    }
}
// ---- the mma form of one stage ---------------------------------------------------------------------------------------
// 16 weight rows x 8 entries x one group: unsigned nibble bytes times signed codes. d[0], d[1]: row lane / 4, entries 2 (lane % 4) and the next; d[2],
// d[3]: row lane / 4 + 8.
__device__ __forceinline__ void mma_u8s8(int (&d)[4], const u32 (&a)[4], u32 b0, u32 b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "r"(0));
}
// The entry of MMA column c where the columns hold eight: a lane's two cells are entries t and t + 4, so that four lanes' reads of deltas and sums meet every bank once.
__device__ __forceinline__ u32 entry_of(u32 c) { return (c >> 1) + 4u * (c & 1u); }
// One stage of the warp's 32 weight rows and chain (pair p) against up to 8 staged A8 rows with tensor-core dots. blk: the half's first row and super-block
// of the stage; fac: the warp's scratch, S x kFacFloats. Chain 4 j + 2 r + e of a lane: row 16 j + 8 r + lane / 4 with the lane's entry e. MANY: items of five entries or
// more, a lane's entries are t = lane % 4 and t + 4. Else the eight columns hold the entries twice, and of a lane's cells the first tile's count in lanes with
// t < 2, the second tile's in the others: four chains, entries 2 (t % 2) and the next, and half of the work after the dots falls away.
// Absent entries compute on other entries' or stale shared memory and are never stored.
// Why 32 rows of one chain, and not 8 rows of four chains as before: what bounds the loop is what it reads from shared memory (128 bytes a clock). A token's
// codes, deltas and sums are read once per 32 rows and a row's factors once per two entries: 44 (MANY) or 36 wavefronts a warp and super-block
// where the form before took 88; dp4a takes 32 for one entry and 20 more for every further one.
// Shared memory is read by explicit 32-bit addresses: out of pointers the compiler made reads with 806,000 bank conflicts a launch (dense 5120 x 17408, 8 rows, gate/up: of
// 4.11 M wavefronts; 64,000 of 3.37 M now), a call 60.9 us, 59.5 now.
template <bool MANY, class G, class Put>
__device__ __forceinline__ void stage_rows_mma(u32 blk, u32 nbk, u32 p, u32 lane, u32 xs, u32 fac, Put put_term) {
    constexpr u32 S = G::S;
    const u32 g = lane >> 2, t = lane & 3u;
    const u32 head = blk + lane * G::row_bytes, put = fac + 16u * lane;
    // the previous stage's readers are done with the scratch: they met before they handed the stage back
#pragma unroll
    for (u32 b = 0; b < S; ++b) {  // the factors, lane = row
        if (b >= nbk) break;
        sts128(put + b * (kHalfRows * 16u), pair_factors<G::Q5K>(lds128(head + b * G::block), p));
    }
    __syncwarp();
    const u32 rows = blk + g * G::row_bytes + G::nibbles + 32u * p + 4u * t, high = blk + g * G::row_bytes + 16u + 4u * t;
    const u32 codes = xs + (MANY ? entry_of(g) : g & 3u) * G::box_codes + 4u * t + 64u * p;
    const u32 es = xs + G::off_deltas + (MANY ? t : 2u * (t & 1u)) * G::box_group + 8u * p;
    const bool second = t >= 2u;  // of the few form
    const u32 get = fac + 16u * g + (!MANY && second ? 256u : 0u);
#pragma unroll
    for (u32 b = 0; b < S; ++b) {
        if (b >= nbk) break;
        const u32 cb = codes + 256u * b;
        u32 lo[2][4], hi[2][4], bl[2], bh[2];
#pragma unroll
        for (u32 j = 0; j < 2; ++j)
#pragma unroll
            for (u32 i = 0; i < 4; ++i) {
                const u32 at = b * G::block + (16u * j + 8u * (i & 1u)) * G::row_bytes + 16u * (i >> 1), q = lds32(rows + at);
                lo[j][i] = q & 0x0f0f0f0fu;
                hi[j][i] = q & 0xf0f0f0f0u;
                if (G::Q5K) {
                    const u32 h = lds32(high + at);
                    lo[j][i] |= fifth_bits(h, 2u * p);
                    hi[j][i] = (hi[j][i] >> 4) | fifth_bits(h, 2u * p + 1u);
                }
            }
#pragma unroll
        for (u32 i = 0; i < 2; ++i) { bl[i] = lds32(cb + 16u * i); bh[i] = lds32(cb + 32u + 16u * i); }
        float2 E[2], Sg[2];
#pragma unroll
        for (u32 e = 0; e < 2; ++e) {
            const uint2 d = lds64(es + 32u * b + (MANY ? 4u : 1u) * e * G::box_group), m = lds64(es + 32u * b + (MANY ? 4u : 1u) * e * G::box_group + (G::off_sums - G::off_deltas));
            E[e] = make_float2(__uint_as_float(d.x), __uint_as_float(d.y));
            Sg[e] = to_float(make_int2(static_cast<int>(m.x), static_cast<int>(m.y)));
        }
        int l[2][4], h[2][4];
#pragma unroll
        for (u32 j = 0; j < 2; ++j) {
            mma_u8s8(l[j], lo[j], bl[0], bl[1]);
            mma_u8s8(h[j], hi[j], bh[0], bh[1]);
        }
        if (!MANY) {
#pragma unroll
            for (u32 i = 0; i < 4; ++i) { l[0][i] = second ? l[1][i] : l[0][i]; h[0][i] = second ? h[1][i] : h[0][i]; }
        }
#pragma unroll
        for (u32 j = 0; j < (MANY ? 2u : 1u); ++j)
#pragma unroll
            for (u32 r = 0; r < 2; ++r) {
                const uint4 v = lds128(get + b * (kHalfRows * 16u) + 256u * j + 128u * r);
                const float4 f = make_float4(__uint_as_float(v.x), __uint_as_float(v.y), __uint_as_float(v.z), __uint_as_float(v.w));
#pragma unroll
                for (u32 e = 0; e < 2; ++e) put_term(b, 4 * j + 2 * r + e, pair_term(f, make_int2(l[j][2 * r + e], h[j][2 * r + e]), E[e], Sg[e]));
            }
    }
}

// 18 warps: two of the SM's four register partitions (16 K registers each) hold five warps, which caps a thread at
// 16384 / (5 x 32) = 102 registers, 96 after rounding - what this launch bound gives (112 was tried: the launch is refused).
template <bool DOWN, u32 S_, u32 CAP_, bool PAIR, bool Q5K>
__global__ void __launch_bounds__(kThreads, 1)
q4k_wide_kernel(const __grid_constant__ WideMaps maps, WideArgs a, WidePlan plan) {
    using G = Geo<S_, CAP_, Q5K>;
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
    u64* passed = left + kGroups;              // PAIR: [group][warp] the chains are there for the group's next stage
    at += (2 * kGroups * plan.stages + 2 * kGroups + (PAIR ? kConsumerWarps : 0u)) * 8;
    u32* slot_item = reinterpret_cast<u32*>(at);
    at += kGroups * plan.stages * 4;
    float* s_pass = reinterpret_cast<float*>((reinterpret_cast<uintptr_t>(at) + 64 + 15) & ~uintptr_t(15));  // PAIR: [group][warp][cells][lane]
    u32* ctl = reinterpret_cast<u32*>(at);  // [0] abort flag, [1] producers that have retired, [2] virtual experts, [3] items, [4] PAIR: the summary
    volatile u32* abort_flag = ctl;

    const u32 tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    if (tid < kGroups * plan.stages) { mbar_init(&full[tid], 1); mbar_init(&empty[tid], kGroupWarps); }
    if (tid < 2 * kGroups) mbar_init(&met[tid], kGroupWarps);
    if (PAIR && tid < kConsumerWarps) mbar_init(&passed[tid], 1);
    if (tid < 2) ctl[tid] = 0;  // the list's builder writes the others, and for a dense block there is no barrier between here and there
    if (tid < kGroups * plan.stages + (PAIR ? kConsumerWarps : 2 * kGroups)) asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");

    if (!early) chain_begin();
    if (DOWN && !early && block_skips(a.summary)) {  // a failed or aborted projection skips the whole stage (routed_expert.hpp:17-19)
        if (!PAIR && tid == 0) retire_block(claim);
        return;
    }

    // ---- the virtual expert list (the stage area is free until the first copy is issued: it holds the copied routes)
    if (plan.dense_rows) build_dense_list(plan.dense_rows, plan.n_chunks, table, ctl);
    else build_work_list(a.routes, plan.n_bound ? plan.n_bound : min(load_l2(a.routes.counts), plan.max_union), plan.max_union, plan.vmax, plan.n_chunks, reinterpret_cast<u32*>(smem), table, ctl);
    const u32 n_items = ctl[3];
    const u32 my_segs = PAIR ? (plan.nseg + 1u - (warp < kConsumerWarps ? warp / kGroupWarps : warp - kConsumerWarps)) / 2u : plan.nseg;  // stages of an item that are the group's
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
        const u32 in_stride = a.in.stride ? a.in.stride : a.in.width, in_gs = in_stride / 32;
        const u32 e = lane >> 2, part = lane & 3u;  // entries that lie anywhere: four lanes an entry, the first for the codes, two each for the deltas and the sums
        u32 t = 0, slot = 0, use = 0;  // stage count, ring position, lap
        bool ok = true;
        auto ask_weights = [&](u32 s, const VExpert& ve, u32 chunk, unsigned char* dst, u64* bar) {  // one lane
            const u32 x = s * G::S * (G::block / 8);  // 64-bit elements: a multiple of 18 or 22, i.e. of 144 or 176 bytes
            const u32 y = ve.expert() * a.rows_per_expert + (DOWN ? kItemRows : kHalfRows) * chunk;
            tma_2d(dst, &maps.w0, x, y, bar);
            tma_2d(dst + G::half_bytes, &maps.w1, x, DOWN ? y + kHalfRows : y, bar);
        };
        u32 ahead = 0;  // stages of the first item whose weights were asked for before the wait
        if (early) {
            const u32 k = PAIR ? blockIdx.x : g * gridDim.x + blockIdx.x;
            if (k < n_items) {
                ahead = min(my_segs, plan.stages);
                if (g == 0) ahead = min(ahead, plan.stall_stage);
                if (lane == 0) {
                    const u32 jv = k / plan.n_chunks;
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the list was made in the stages' memory
                    for (u32 s = 0; s < ahead; ++s) {
                        mbar_expect_more(&g_full[s], G::w_bytes);
                        ask_weights(PAIR ? 2u * s + g : s, table[jv], k - jv * plan.n_chunks, g_stage + s * plan.stage_bytes, &g_full[s]);
                    }
                }
            }
            chain_begin();
            // The stage is skipped: the group leaves as one, its consumers by an end mark, once the weights have landed (the wait is bounded). The groups of PAIR, which wait for
            // each other, share an answer; the others need none of the other's, and a barrier took 0.3 and 0.7 us of a call (128 experts of 2048 x 768, 1 and 37 rows).
            u32 skips = DOWN && a.summary ? *a.summary : 0u;
            if (DOWN && PAIR) {
                if (lane == 0 && g == 0) ctl[4] = skips;
                asm volatile("bar.sync 1, %0;" ::"r"(kGroups * 32u) : "memory");
                skips = ctl[4];
            }
            if (DOWN && skips) {
                if (lane == 0) {
                    g_item[0] = kEndItem;
                    for (u32 s = 0; s < max(ahead, 1u); ++s) mbar_arrive(&g_full[s]);
                    for (u32 s = 0; s < ahead; ++s)
                        for (u32 i = 0; i < (plan.wait_limit >> 4) + 64u; ++i)
                            if (mbar_try_wait(&g_full[s], 0)) break;
                    if (!PAIR) retire_claims(claim, ctl);  // the other group, other CTAs may have items
                }
                return;
            }
        }
        // A group's first item needs no round trip: group 0 of CTA b takes item b, group 1 item gridDim.x + b - so a
        // launch with fewer items than groups runs one group per SM, which has the SM's issue slots to itself. The next item is claimed ahead of the wait for
        // the place of an item's last stage, and the places of its entries' A8 rows are asked for behind that stage: neither trip to memory is waited for
        // (128 experts of 2048 x 768, us a call: 1 row 23.6 -> 22.9, 8 rows 51.5 -> 50.0).
        u32 item = PAIR ? blockIdx.x : g * gridDim.x + blockIdx.x, next = 0;
        for (;;) {
            const bool end = item >= n_items;
            VExpert ve{0};
            u32 chunk = 0;
            if (!end) {
                const u32 jv = item / plan.n_chunks;
                chunk = item - jv * plan.n_chunks;
                ve = table[jv];
            }
            const u32 ve_ne = ve.ne();
            u32 row = 0;
            if (e < ve_ne && !end) { const u32 at = ve.begin() + e; row = plan.dense_rows ? at : load((DOWN ? a.routes.slots : a.routes.rows) + at); }
            const u32 nsegs = end ? 1u : my_segs;
            for (u32 i = 0; i < nsegs; ++i, ++t, ++slot) {
                const u32 s = PAIR ? 2u * i + g : i;
                if (slot == plan.stages) { slot = 0; ++use; }
                if (!PAIR && !end && i + 1u == nsegs && lane == 0) next = claim_item(claim);
                if (use) ok = warp_wait(&g_empty[slot], (use - 1u) & 1u, plan.wait_limit, abort_flag);  // the slot's previous use is done
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
                    mbar_expect_more(&g_full[slot], (t < ahead ? 0u : G::w_bytes) + (plan.boxes ? G::boxes_tx : ve_ne * nbk * 256u));
                    if (t >= ahead) ask_weights(s, ve, chunk, dst, &g_full[slot]);
                }
                __syncwarp();  // the bytes are expected
                unsigned char* xd = dst + G::w_bytes;
                if (plan.boxes) {
                    if (lane == 0) {
                        tma_2d(xd, &maps.codes, s * (G::S * 32u), ve.begin(), &g_full[slot]);  // 64-bit elements
                        tma_2d(xd + G::off_deltas, &maps.deltas, s * (G::S * 4u), ve.begin(), &g_full[slot]);
                        tma_2d(xd + G::off_sums, &maps.sums, s * (G::S * 4u), ve.begin(), &g_full[slot]);
                    }
                } else {  // the arrival that lets the stage complete comes behind the lanes' copies, each of which adds one of its own while it is under way
                    if (e < ve_ne) {
                        if (part == 0) bulk_g2s(xd + e * G::box_codes, a.in.codes + u64(row) * in_stride + u64(s) * G::S * 256u, nbk * 256u, &g_full[slot]);
                        const unsigned char* from = (part & 2u ? reinterpret_cast<const unsigned char*>(a.in.sums) : reinterpret_cast<const unsigned char*>(a.in.deltas)) + (u64(row) * in_gs + u64(s) * G::S * 8u) * 4u + 16u * (part & 1u);
                        unsigned char* to = xd + (part & 2u ? G::off_sums : G::off_deltas) + e * G::box_group + 16u * (part & 1u);
#pragma unroll
                        for (u32 b = 0; b < G::S; ++b)
                            if (b < nbk) cp_async16(to + 32u * b, from + 32u * b);
                    }
                    asm volatile("cp.async.mbarrier.arrive.shared::cta.b64 [%0];" ::"r"(saddr(&g_full[slot])) : "memory");
                    __syncwarp();
                }
                if (lane == 0) mbar_arrive(&g_full[slot]);
                __syncwarp();
            }
            if (!ok || end) break;
            item = PAIR ? n_items : gridDim.x * kGroups + __shfl_sync(0xffffffffu, next, 0);  // PAIR: there are no more items than CTAs
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        if (!ok && lane == 0) {  // wait (bounded) for the copies still in flight before the CTA retires
            for (u32 n = t > plan.stages ? t - plan.stages : 0u; n < t; ++n)
                for (u32 i = 0; i < (plan.wait_limit >> 4) + 64u; ++i)
                    if (mbar_try_wait(&g_full[n % plan.stages], (n / plan.stages) & 1u)) break;
        }
        if (!PAIR && lane == 0) retire_claims(claim, ctl);
        return;
    }

    // ------------------------------------------------------------------------------------------ consumer warps
    if (early) chain_begin();
    const u32 g = warp / kGroupWarps, w = warp % kGroupWarps;
    const u32 p = lane >> 3, rr = lane & 7u;     // dp4a form: lane = (pair, one of the warp's 8 rows)
    const u32 mp = w & 3u, half = w >> 2;        // mma form: the warp's chain and half of the item
    const u32 me = lane >> 2, mt = lane & 3u;
    float* fac = s_fac + warp * (S_ * kFacFloats);
    float* meet = s_meet + g * kMeetFloats;
    u64* g_full = full + g * plan.stages;
    u64* g_empty = empty + g * plan.stages;
    const u32* g_item = slot_item + g * plan.stages;
    const u32 g_stage = saddr(smem) + g * plan.stages * plan.stage_bytes;
    const u32 act_stride = DOWN ? 0u : (a.act.stride ? a.act.stride : a.act.width);
    u32 slot = 0, phase = 0, kl = 0;  // ring position of the group's next stage, kept incrementally (no divisions in the loop); meetings so far
    bool ok = true;
    for (;;) {
        ok = warp_wait(&g_full[slot], phase, plan.wait_limit, abort_flag);
        if (!ok) break;
        const u32 item = g_item[slot];
        if (item == kEndItem) break;
        const u32 jv = item / plan.n_chunks, chunk = item - jv * plan.n_chunks;
        const VExpert ve = table[jv];
        const u32 ne = ve.ne(), vbegin = ve.begin();
        const bool mma = G::CAP > 1 && ne > kDpEntries;
        const u32 slot_id = w >= ne ? 0u : plan.dense_rows ? vbegin + w : load(a.routes.slots + vbegin + w);  // asked for before the stages, used behind them
        // The item's stages, with the form fixed at compile time inside the loop: `terms` makes what the stage's super-blocks add to the chains. PAIR: the chains go
        // to the other group's warp of the same rows after each stage, and the last stage's group ends the item.
        auto stages = [&](auto& chain, auto terms) {
            constexpr u32 N = sizeof(chain) / 4u;
#pragma unroll
            for (float& c : chain) c = 0.0f;
            for (u32 i = 0; i < my_segs; ++i) {
                const u32 s = PAIR ? 2u * i + g : i, nbk = min(G::S, plan.nb - s * G::S);
                if (i) {
                    ok = warp_wait(&g_full[slot], phase, plan.wait_limit, abort_flag);
                    if (!ok) return;
                }
                float term[G::S][N];
                terms(g_stage + slot * plan.stage_bytes, nbk, [&](u32 b, u32 c, float v) {
                    if (PAIR) term[b][c] = v;
                    else chain[c] = __fadd_rn(chain[c], v);
                });
                __syncwarp();
                if (lane == 0) mbar_arrive(&g_empty[slot]);  // the stage is free for the producer
                if (++slot == plan.stages) { slot = 0; phase ^= 1u; }
                float* mine = s_pass + warp * (32u * N);
                if (PAIR && s) {
                    ok = warp_wait(&passed[warp], (i - 1u + g) & 1u, plan.wait_limit, abort_flag);
                    if (!ok) return;
#pragma unroll
                    for (u32 c = 0; c < N; ++c) chain[c] = mine[32u * c + lane];
                }
#pragma unroll
                for (u32 b = 0; b < G::S; ++b) {
                    if (!PAIR || b >= nbk) break;
#pragma unroll
                    for (u32 c = 0; c < N; ++c) chain[c] = __fadd_rn(chain[c], term[b][c]);
                }
                if (PAIR && s + 1u < plan.nseg) {
                    float* theirs = s_pass + (warp ^ kGroupWarps) * (32u * N);
#pragma unroll
                    for (u32 c = 0; c < N; ++c) theirs[32u * c + lane] = chain[c];
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&passed[warp ^ kGroupWarps]);
                }
            }
        };
        const bool ends_item = !PAIR || ((plan.nseg - 1u) & 1u) == g;
        // the chains meet in shared memory, once the previous item's have been read
        auto hand_over = [&](auto store) {
            if (kl) ok = warp_wait(&left[g], (kl - 1u) & 1u, plan.wait_limit, abort_flag);
            if (!ok) return;
            store();
            __syncwarp();
            if (lane == 0) mbar_arrive(&met[g]);
            ok = warp_wait(&met[g], kl & 1u, plan.wait_limit, abort_flag);
        };
        auto run_mma = [&](auto many) {
            constexpr bool MANY = decltype(many)::value;
            float acc[MANY ? 8 : 4];
            stages(acc, [&](u32 st, u32 nbk, auto put) { stage_rows_mma<MANY, G>(st + half * G::half_bytes, nbk, mp, lane, st + G::w_bytes, saddr(fac), put); });
            if (!ok || !ends_item) return;
            hand_over([&]() {
#pragma unroll
                for (u32 j = 0; j < (MANY ? 2u : 1u); ++j)
#pragma unroll
                    for (u32 e = 0; e < 2; ++e) {
                        const u32 tile = MANY ? j : mt >> 1, entry = MANY ? mt + 4u * e : 2u * (mt & 1u) + e;
                        float* to = meet + ((2u * mp + half) * kKE + entry) * kMeetPitch + 16u * tile + me;
                        to[0] = acc[4 * j + e];
                        to[8] = acc[4 * j + 2 + e];
                    }
            });
        };
        if (!mma) {
            const u32 only_slot = !DOWN ? 0u : plan.dense_rows ? vbegin : load(a.routes.slots + vbegin);
            float acc[1];
            stages(acc, [&](u32 st, u32 nbk, auto put) { stage_row<G>(st + half * G::half_bytes + (8u * mp + rr) * G::row_bytes, nbk, p, st + G::w_bytes, put); });
            if (!ok) break;
            if (!ends_item) continue;
            const float val = tree4(acc[0]);
            if (DOWN) {
                if (p == 0) a.raw[u64(only_slot) * a.out_width + kItemRows * chunk + 8u * w + rr] = val;
                continue;
            }
            hand_over([&]() { if (p == 0) meet[half * kKE * kMeetPitch + 8u * mp + rr] = val; });
        } else if (G::CAP > kFewEntries && ne > kFewEntries) {
            if constexpr (G::CAP > kFewEntries) run_mma(std::true_type{});
        } else {
            if constexpr (G::CAP > 1) run_mma(std::false_type{});
        }
        if (!ok) break;
        if (!ends_item) continue;
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
           (2 * kGroups * p.stages + 2 * kGroups) * 8 + kGroups * p.stages * 4 + 64 + (p.pair ? kConsumerWarps * 8 + 16 + kConsumerWarps * 128 * p.cap : 0u);
}
u32 plan_smem(const WidePlan& p) { return kGroups * p.stages * p.stage_bytes + fixed_smem(p); }

// K: the row length; n_chunks: items per expert; slots: rows * top_k of the window. False when the form does not apply.
bool make_plan(bool q5k, u32 K, u32 n_chunks, u32 max_union, u64 slots, WidePlan* p) {
    if (K == 0 || K % 256 || max_union == 0 || slots == 0 || slots > 8192) return false;
    p->nb = K / 256;
    p->S = p->nb >= 3 ? 3u : 1u;  // odd: see Geo
    p->nseg = (p->nb + p->S - 1) / p->S;
    // a stage holds the A8 segments of as many entries as a virtual expert of this window can have: windows of fewer than
    // kKE slots get smaller stages and with them a deeper ring
    p->cap = slots == 1 ? 1u : slots <= 4 ? 4u : 8u;
    auto bytes = [&](auto s3, auto s1) { return p->S == 3 ? decltype(s3)::stage_bytes : decltype(s1)::stage_bytes; };
    if (q5k) p->stage_bytes = p->cap == 1 ? bytes(Geo<3, 1, true>{}, Geo<1, 1, true>{}) : p->cap == 4 ? bytes(Geo<3, 4, true>{}, Geo<1, 4, true>{}) : bytes(Geo<3, 8, true>{}, Geo<1, 8, true>{});
    else p->stage_bytes = p->cap == 1 ? bytes(Geo<3, 1>{}, Geo<1, 1>{}) : p->cap == 4 ? bytes(Geo<3, 4>{}, Geo<1, 4>{}) : bytes(Geo<3, 8>{}, Geo<1, 8>{});
    p->n_chunks = n_chunks;
    p->max_union = max_union;
    p->vmax = max_union + static_cast<u32>(slots / kKE) + 1;
    if (u64(p->vmax) * n_chunks + 4096 >= kClaimMask) return false;  // items and the groups' closing claims fit the claim word's count
    // PAIR where the items, virtual experts at most union + (entries beyond one each) / kKE times the chunks, are no more than CTAs, so that the second group would
    // have nothing to do. Down of a dense 5120 x 17408 block (80 items of 23 stages): 1 row 29,700 -> 24,400 clocks, 8 rows 53,400 -> 46,800; a call 39.6 -> 38.1 and
    // 59.5 -> 58.0 us.
    p->pair = p->S == 3 && p->nseg > 1 && (max_union + (slots - std::min<u64>(slots, max_union)) / kKE) * n_chunks <= static_cast<u32>(device_sm_count());
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

// The tensor maps of a dense block's A8 rows: exactly the window's rows. Rows shorter than a box come by untiled copies. Why boxes: to ask for one untiled copy takes a
// producer 70 clocks, for 24 (8 entries) 1,690 of the 2,030 that its consumers work on the stage; three boxes are asked for by one lane. Dense 5120 x 17408, us a call, all
// changes of the kernel together: 8 rows 66.1 -> 55.6, 1 row (three untiled copies a stage) 42.7 -> 37.5. Routed entries lie anywhere: one untiled copy of each entry's codes,
// and the deltas and sums, two thirds of the copies and a fifth of the bytes, as three asynchronous copies a lane. All untiled and so, us a call: 64 rows of the large layer
// 719 and 680, 37 rows over 128 experts of 2048 -> 768 93.9 and 91.9, one row 22.5 and 21.7. Gathering copies of four rows took 681 there, but raised an illegal memory access
// where the rows began a mapping: not understood, not used.
int entry_maps(const b200moe_a8_rows& x, u32 K, WidePlan* p, WideMaps* m) {
    m->codes = m->deltas = m->sums = m->w0;
    const u32 codes = p->S * 256u + 16u, group = p->S * 32u;  // Geo::box_codes, box_group
    p->boxes = p->dense_rows && p->cap > 1 && K >= codes;
    if (!p->boxes) return B200MOE_OK;
    const u64 pitch = x.stride ? x.stride : x.width;
    if (int rc = pitched_map(reinterpret_cast<const u8*>(x.codes), K, pitch, p->dense_rows, codes, p->cap, &m->codes)) return rc;
    if (int rc = pitched_map(reinterpret_cast<const u8*>(x.deltas), K / 8, pitch / 8, p->dense_rows, group, p->cap, &m->deltas)) return rc;
    return pitched_map(reinterpret_cast<const u8*>(x.sums), K / 8, pitch / 8, p->dense_rows, group, p->cap, &m->sums);
}
template <bool DOWN, bool Q5K>
int launch_wide(const WideMaps& m, const WideArgs& a, const WidePlan& p, cudaStream_t stream) {
    const auto kernel = p.pair ? (p.cap == 1 ? q4k_wide_kernel<DOWN, 3, 1, true, Q5K> : p.cap == 4 ? q4k_wide_kernel<DOWN, 3, 4, true, Q5K> : q4k_wide_kernel<DOWN, 3, 8, true, Q5K>)
                        : p.S == 3 ? (p.cap == 1 ? q4k_wide_kernel<DOWN, 3, 1, false, Q5K> : p.cap == 4 ? q4k_wide_kernel<DOWN, 3, 4, false, Q5K> : q4k_wide_kernel<DOWN, 3, 8, false, Q5K>)
                                   : (p.cap == 1 ? q4k_wide_kernel<DOWN, 1, 1, false, Q5K> : p.cap == 4 ? q4k_wide_kernel<DOWN, 1, 4, false, Q5K> : q4k_wide_kernel<DOWN, 1, 8, false, Q5K>);
    const u32 smem = plan_smem(p);
    if (int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), smem)) return rc;
    chain_launch(kernel, device_sm_count(), kThreads, smem, stream, m, a, p);
    return after_launch(DOWN ? "down_q4k_wide" : "gate_up_q4k_wide");
}

void apply_hooks(WidePlan* p) {
    const u32 limit = debug_value(B200MOE_DEBUG_WAIT_LIMIT), stall = debug_value(B200MOE_DEBUG_STALL_STAGE);
    if (limit) p->wait_limit = limit;
    if (stall) p->stall_stage = stall - 1u;
}

}  // namespace

bool wide_gate_up_fits(const b200moe_gate_up_view& v, u32 rows) {
    WidePlan p{};
    return is_kquant(v.shape.gate_type) && rows && a8_bulk_ok(v.x) && v.shape.inter % 32 == 0 &&
           make_plan(v.shape.gate_type == B200MOE_TYPE_Q5_K, v.shape.hidden, v.shape.inter / 32, v.max_union, u64(rows) * v.shape.top_k, &p);
}
bool wide_down_fits(const b200moe_down_view& v, u32 rows) {
    WidePlan p{};
    return v.shape.down_type == B200MOE_TYPE_Q4_K && rows && a8_bulk_ok(v.act) && v.shape.hidden % 64 == 0 &&
           make_plan(false, v.shape.inter, v.shape.hidden / 64, v.max_union, u64(rows) * v.shape.top_k, &p);
}

int launch_gate_up_q4k_wide(const b200moe_gate_up_view& v, u32 rows, const ChainHints& hints, cudaStream_t stream) {
    if (v.max_union == 0) return B200MOE_OK;
    WidePlan p{};
    const bool q5k = v.shape.gate_type == B200MOE_TYPE_Q5_K;
    if (!make_plan(q5k, v.shape.hidden, v.shape.inter / 32, v.max_union, u64(rows) * v.shape.top_k, &p))
        return fail(B200MOE_ERR_UNSUPPORTED, "gate_up: the segment-streaming form does not apply to this shape");
    apply_hooks(&p);
    p.early = hints.routes_done || hints.dense_rows; p.dense_rows = hints.dense_rows; p.n_bound = static_cast<u32>(std::min<u64>(v.max_union, hints.slots));
    WideArgs a{};
    a.routes = v.routes; a.in = v.x; a.act = v.act; a.gate_out = v.gate_out; a.up_out = v.up_out;
    a.row_status = v.row_status; a.summary = v.summary; a.rows_per_expert = v.shape.inter; a.out_width = v.shape.inter;
    WideMaps m;
    const u32 block = q5k ? kQ5KBlock : kQ4KBlock;
    const u64 rb = u64(p.nb) * block, total_rows = u64(v.shape.experts) * v.shape.inter;
    if (int rc = rows_map(v.weights.gate, rb, total_rows, p.S * block, kHalfRows, &m.w0)) return rc;
    if (int rc = rows_map(v.weights.up, rb, total_rows, p.S * block, kHalfRows, &m.w1)) return rc;
    if (int rc = entry_maps(v.x, v.shape.hidden, &p, &m)) return rc;
    return q5k ? launch_wide<false, true>(m, a, p, stream) : launch_wide<false, false>(m, a, p, stream);
}

int launch_down_q4k_wide(const b200moe_down_view& v, u32 rows, const ChainHints& hints, cudaStream_t stream) {
    if (v.max_union == 0) return B200MOE_OK;
    WidePlan p{};
    if (!make_plan(false, v.shape.inter, v.shape.hidden / 64, v.max_union, u64(rows) * v.shape.top_k, &p))
        return fail(B200MOE_ERR_UNSUPPORTED, "down: the segment-streaming form does not apply to this shape");
    apply_hooks(&p);
    p.early = hints.routes_done || hints.dense_rows; p.dense_rows = hints.dense_rows; p.n_bound = static_cast<u32>(std::min<u64>(v.max_union, hints.slots));
    WideArgs a{};
    a.routes = v.routes; a.in = v.act; a.raw = v.raw; a.summary = const_cast<u32*>(v.summary);
    a.rows_per_expert = v.shape.hidden; a.out_width = v.shape.hidden; a.raw_vec = aligned(v.raw, 8);
    WideMaps m;
    const u64 rb = u64(p.nb) * kQ4KBlock;
    if (int rc = rows_map(v.weights.down, rb, u64(v.shape.experts) * v.shape.hidden, p.S * kQ4KBlock, kHalfRows, &m.w0)) return rc;
    m.w1 = m.w0;
    if (int rc = entry_maps(v.act, v.shape.inter, &p, &m)) return rc;
    return launch_wide<true, false>(m, a, p, stream);
}

}  // namespace b200moe
