// Routed experts, Qwen A8 family, GROUPED form for token blocks (prefill): the integer dots run on the tensor cores, everything
// after the dots is the same declared FP32 arithmetic as the decode kernels, so the results are bit for bit those of
// gemv_q4k.cu / gemv_q4k_stream.cu (contract: src/cpu/core/routed_expert.hpp:9-15, row rule routed_expert.cpp:73-108; the
// reference's own tensor-core form is project_kernel / down_kernel, src/cuda/core/moe_a8.cuh:76-206, :225-341).
//
// What bounds it: register reads. The contract scales every 32-wide group's EXACT integer dot by its own factors: five FP32 operations
// per (row, token, group), ten packed instructions per MMA of 16 tokens x 8 rows x 32. On a loop of its own, in clocks of a scheduler per
// such MMA: the ten alone 20 to 22 (a packed product or sum reads two register pairs and takes two clocks, an fma of three distinct
// pairs takes three), with the MMA 28 (its ten operand and result registers go through the same ports; its time ADDS), 30 with the
// conversion of the dots and the sums written as fma, 31 with a barrier per 32 MMAs. The kernel spends 36 to 38; the end of a tile (the
// chains' meeting, SwiGLU + the A8 rule) is paid where the other two thirds' warps leave the schedulers free.
// gate/up of 4096 x 8 tokens, skewed, over 128 experts of 2048 -> 2 x 768: 1070 us (1124 while all twelve consumer warps met at a tile's end, with gate rows in
// one half of the tile's rows and their up rows in the other); of 512 tokens x 34,816 rows x 5120, whose tiles are longer: 805 us (810).
// The dots out of tensor memory (tcgen05.mma kind::i8) leave the ports free (24 clocks a unit on a loop of its own), but what that form
// adds - nibbles unpacked to shared memory, MMA and commit latencies between two barriers, more code than a scheduler's instruction
// cache holds - cost more: 1180 to 1480 us, in 16 consumer warps of one chain or 8 of two.
//
// Tile = (expert, 192 weight rows, kGN of the expert's tokens). gate/up: rows 0..95 are gate rows [96c, 96c + 96), rows 96..191 the up
// rows of the same outputs; a third of the consumers takes 32 of the gate rows and their up rows, so SwiGLU + the A8 rule of h finish inside the third. down: 192 rows of H. The last row tile of an expert
// ends with it and may repeat rows of the tile before (the same bits twice): a read past an expert's rows could leave the tensor, which may
// hold fewer experts than the shape counts.
// A persistent CTA per SM walks tiles round-robin; a stage of the ring (three) is one super-block: 256 columns, 4 pairs of groups (chains).
//   * helper warps (4): the tile's weight rows arrive by two tiled TMA copies (144 bytes x 96 rows: consecutive rows lie 4 (mod 32) words
//     apart, the fragment loads below are conflict free), the tokens' codes, deltas and sums by 16-byte asynchronous copies (codes 272
//     bytes apart, for the same reason), up to three stages ahead of the consumers. A thread of the first three warps decodes the factors of two weight rows, a lane
//     of the fourth lays out the {E, S} of one token.
//   * consumer warps (12): warp = 64 rows x all tokens of ONE of the four chains. The nibbles go from shared memory straight into B
//     fragments (low nibbles by a mask, high nibbles left in place as 16 q), the codes into A fragments; a lane's two neighbouring cells
//     are two weight rows of one token, so the rows' factors are natural register pairs and the packed instructions take a token's
//     factors as one register for both halves. A row's factors are read once per 32 tokens, a token's once per 64 rows.
//     The four chains of a row third meet through shared memory at the end of a tile, (a0 + a1) + (a2 + a3); gate/up then runs
//     SwiGLU + the A8 rule, a warp two tokens at a time. A third's barriers are its own: the thirds drift apart and end their tiles at different times.
// Every wait is bounded; on a timeout the roles stop working, the first helper waits (bounded) for the copies in flight and the launch sets
// B200MOE_JOB_WAIT_ABORTED in the job summary.
#include <cuda.h>

#include "grouped_common.cuh"
#include "wide_common.cuh"

namespace b200moe {
namespace {
using namespace q4k;
using namespace grouped;

constexpr u32 kTokTiles = 2;                     // 16-token MMA tiles of a CTA tile
constexpr u32 kRowTiles = 8;                     // 8-row MMA tiles of a consumer warp
constexpr u32 kThirds = 3;                       // consumer warps of a chain
constexpr u32 kGM = 64 * kThirds, kGN = 16 * kTokTiles;  // tile: weight rows x tokens
constexpr u32 kOutRows = kGM / 2;                // gate/up: outputs of a tile
constexpr u32 kConsumers = 4 * kThirds, kHelpers = 4;    // warps
constexpr u32 kGThreads = (kConsumers + kHelpers) * 32;
constexpr u32 kStages = 3;
constexpr u32 kCodePitch = 256 + 16;
constexpr u32 kRawBytes = kGM * kQ4KBlock, kCodeBytes = kGN * kCodePitch, kEsBytes = 4 * kGN * 16, kFacBytes = 4 * kGM * 16, kPrivBytes = kGN * 64;
constexpr u32 kStageBytes = (kRawBytes + kCodeBytes + kEsBytes + kFacBytes + kPrivBytes + 127) / 128 * 128;
constexpr u32 kOffCode = kRawBytes, kOffEs = kOffCode + kCodeBytes, kOffFac = kOffEs + kEsBytes, kOffPriv = kOffFac + kFacBytes;  // in a stage
constexpr u32 kOutPitch = 64 + 8;                // floats: the 8-byte stores of a half warp (four tokens, four row pairs) meet every bank once
constexpr u32 kOutBytes = kGN * kOutPitch * 4;   // a third's epilogue tile (gate/up): 32 gate and 32 up values a token
constexpr u32 kFoldCells = kRowTiles / 2 * kTokTiles * 2;      // float2 cells of a lane that change hands when two chains meet
constexpr u32 kFoldBytes = kConsumers * kFoldCells * 32 * 8;
static_assert(kOutBytes <= kFoldBytes / kThirds, "a third's epilogue tile takes the place of the buffers that its chains met in");
// What the consumers need of a tile: {first row, tokens, first entry}, its tokens' A8 rows, its tokens' slots. The helpers run at most
// kStages stages ahead of the consumers, a tile has at least one stage and its places are read until its end: eight places.
constexpr u32 kTilePlaces = 8, kTileWords = 4 + 2 * kGN;
constexpr u32 kOffFold = kStages * kStageBytes, kOffBars = kOffFold + kFoldBytes, kOffTile = kOffBars + 3 * kStages * 8 + 8,
              kOffCum = kOffTile + kTilePlaces * kTileWords * 4;
constexpr u32 kGroupedSmem = kOffCum + 2 * kTileCounts * 4;
static_assert((kOutRows * kQ4KBlock) % 128 == 0 && kOffBars % 8 == 0, "TMA destinations, barriers");
static_assert(kGN == 32 && kGM / 2 == (kHelpers - 1) * 32, "a helper lane stages a token, the helper threads before it two rows each");
static_assert(kGroupedSmem > 114u * 1024u && kGroupedSmem <= 227u * 1024u, "one CTA per SM, within the shared memory of an SM");
// Polls of up to four microseconds: about a second. Fixed here: a limit out of the arguments cost the consumers' loop 2 % (512 rows of the dense block 1170 -> 1194 us a call).
constexpr u32 kWaitLimit = 1u << 18;
// Register split between whole warp groups, out of what the launch gives every thread (65,536 over the threads, by eights).
constexpr u32 kLaunchRegs = 65536u / kGThreads / 8u * 8u, kHelperRegs = 80;
constexpr u32 kConsumerRegs = (kGThreads * kLaunchRegs - kHelpers * 32u * kHelperRegs) / (kConsumers * 32u) / 8u * 8u;
static_assert(kConsumers * 32 * kConsumerRegs + kHelpers * 32 * kHelperRegs <= kGThreads * kLaunchRegs, "setmaxnreg split exceeds the launch's registers");

// 16 tokens x 8 weight rows x one group: signed codes times unsigned nibble bytes. d[z]: token lane / 4 + 8 z, weight rows
// 2 (lane % 4) and the next.
__device__ __forceinline__ void mma_dots(int2 (&d)[2], const u32 (&a)[4], u32 b0, u32 b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.u8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
        : "=r"(d[0].x), "=r"(d[0].y), "=r"(d[1].x), "=r"(d[1].y) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "r"(0));
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
    u32 n_row_tiles;         // row tiles of an expert: inter / 96 (gate/up) or hidden / 192 (down), rounded up
    u32 K;                   // hidden (gate/up) or inter (down)
    u32 es_vec;              // the input's deltas and sums lie in whole 16-byte units
    u32 raw_vec;             // raw lies on an 8-byte boundary
    u32 stall_stage;         // test hook: the helpers stop asking for stages before this one
};

// One super-block of the warp's 64 rows and chain against NMT 16-token tiles. rows: weight row lane / 4 of the stage at the pair's
// nibbles of the lane's k slice; codes: token lane / 4 at the pair's codes; es: the pair's {E, E', S, S'} from token lane / 4 on; fac: the
// pair's {D, D, D', D'} {-DM, -DM, -DM', -DM'} of two rows, from row pair lane % 4 on. acc[j][mt][z]: rows 8 j + 2 (lane % 4) and the
// next of token 16 mt + 8 z + lane / 4.
// SPLIT (gate/up): the warp's row tiles 4 to 7 are up rows, kOutRows behind the gate rows of the same outputs in tiles 0 to 3.
template <int NMT, bool SPLIT>
__device__ __forceinline__ void superblock(const unsigned char* rows, const unsigned char* codes, const float4* es, const float4* fac,
                                           float2 (&acc)[kRowTiles][kTokTiles][2]) {
    u32 cl[NMT][4], ch[NMT][4];
    float4 e[NMT][2];
#pragma unroll
    for (int mt = 0; mt < NMT; ++mt)
#pragma unroll
        for (int z = 0; z < 2; ++z) {
            const unsigned char* c = codes + (16 * mt + 8 * z) * kCodePitch;
            // word by word: an A fragment's registers alternate between its two tokens, and 64-bit loads would have to be moved apart
            // before every MMA (four moves each: 33.2 against 30.3 clocks an MMA)
            cl[mt][z] = *reinterpret_cast<const u32*>(c);
            cl[mt][z + 2] = *reinterpret_cast<const u32*>(c + 16);
            ch[mt][z] = *reinterpret_cast<const u32*>(c + 32);
            ch[mt][z + 2] = *reinterpret_cast<const u32*>(c + 48);
            e[mt][z] = es[16 * mt + 8 * z];
        }
#pragma unroll
    for (int j = 0; j < (int)kRowTiles; ++j) {
        const int row = 8 * j + (SPLIT && j >= (int)kRowTiles / 2 ? (int)kOutRows - 32 : 0);
        const u32 q0 = *reinterpret_cast<const u32*>(rows + row * kQ4KBlock), q1 = *reinterpret_cast<const u32*>(rows + row * kQ4KBlock + 16);
        const float4 d4 = fac[row], m4 = fac[row + 1];
        const float2 Dl = make_float2(d4.x, d4.y), Dh = make_float2(d4.z, d4.w), Ml = make_float2(m4.x, m4.y), Mh = make_float2(m4.z, m4.w);
#pragma unroll
        for (int mt = 0; mt < NMT; ++mt) {
            int2 l[2], h[2];
            mma_dots(l, cl[mt], q0 & 0x0f0f0f0fu, q1 & 0x0f0f0f0fu);
            mma_dots(h, ch[mt], q0 & 0xf0f0f0f0u, q1 & 0xf0f0f0f0u);
#pragma unroll
            for (int z = 0; z < 2; ++z) {
                // x = E * ((D * float(dot)) - (DM * S)) for the pair's two groups; M holds -DM, and (-DM) * S = -(DM * S) exactly
                const float2 sl = add2(mul2(Dl, to_float(l[z])), mul2(Ml, both(e[mt][z].z)));
                const float2 sh = add2(mul2(Dh, to_float(h[z])), mul2(Mh, both(e[mt][z].w)));
                acc[j][mt][z] = add2(add2(mul2(both(e[mt][z].x), sl), mul2(both(e[mt][z].y), sh)), acc[j][mt][z]);
            }
        }
    }
}

// SwiGLU + the A8 rule of kTasks (token, 32 outputs) tasks of one warp, step by step over them, so that their chains overlap. g, u: the
// lane's gate and up values; returns per task whether a value is not finite (code, delta and sum then mean nothing).
constexpr int kTasks = 2;
__device__ __forceinline__ u32 swiglu_a8(const float (&g)[kTasks], const float (&u)[kTasks], int (&code)[kTasks], float (&delta)[kTasks], int (&sum)[kTasks]) {
    float h[kTasks], x[kTasks];
    u32 bad = 0, amax[kTasks];
#pragma unroll
    for (int i = 0; i < kTasks; ++i) x[i] = gfx1151_expf(-g[i]);
#pragma unroll
    for (int i = 0; i < kTasks; ++i) {
        h[i] = __fmul_rn(__fdiv_rn(g[i], __fadd_rn(1.0f, x[i])), u[i]);  // swiglu_qwen (declared_math.cuh)
        bad |= __any_sync(0xffffffffu, !finite_f(g[i]) || !finite_f(u[i]) || !finite_f(h[i])) ? 1u << i : 0u;
        amax[i] = __reduce_max_sync(0xffffffffu, __float_as_uint(h[i]) & 0x7fffffffu);  // the bits of finite magnitudes order as they do
    }
#pragma unroll
    for (int i = 0; i < kTasks; ++i) {  // a8_quantize_lane (common.cuh)
        const float am = __uint_as_float(amax[i]);
        const bool tiny = am > 0.0f && am < 0x1p-119f;
        delta[i] = (am == 0.0f || tiny) ? 1.0f : over_127(am);
        const float r = tiny ? 0.0f : rintf(__fdiv_rn(h[i], delta[i]));
        const float lo = (-127.0f < r) ? r : -127.0f;
        code[i] = static_cast<int>((lo < 127.0f) ? lo : 127.0f);
        sum[i] = __reduce_add_sync(0xffffffffu, code[i]);
    }
    return bad;
}

// Factors of a row whose d and dmin are finite: sc / mn hold the 6-bit scales and mins of four groups a byte each. A byte goes behind
// the exponent of 2^23 and fma(d, 2^23 + s, -2^23 d) is d * s, exact as the product has 17 bits. f: per pair D, D' / 16 (the high nibbles'
// dots come as 16 * dot), -DM, -DM'.
__device__ __forceinline__ void fast_factors(u32 head, u32 sc, u32 mn, float (&f)[2][4]) {
    const float d = half_bits_to_float(head & 0xffffu), dm = -half_bits_to_float(head >> 16), dh = __fmul_rn(d, 0.0625f);
    const float nd = __fmul_rn(d, -8388608.0f), ndm = __fmul_rn(dm, -8388608.0f), ndh = __fmul_rn(dh, -8388608.0f);
#pragma unroll
    for (u32 i = 0; i < 2; ++i) {
        f[i][0] = __fmaf_rn(d, __uint_as_float(__byte_perm(sc, 0x4b000000u, 0x7440u + 2u * i)), nd);
        f[i][1] = __fmaf_rn(dh, __uint_as_float(__byte_perm(sc, 0x4b000000u, 0x7441u + 2u * i)), ndh);
        f[i][2] = __fmaf_rn(dm, __uint_as_float(__byte_perm(mn, 0x4b000000u, 0x7440u + 2u * i)), ndm);
        f[i][3] = __fmaf_rn(dm, __uint_as_float(__byte_perm(mn, 0x4b000000u, 0x7441u + 2u * i)), ndm);
    }
}

template <bool kDown>
__global__ void __launch_bounds__(kGThreads, 1) grouped_q4k_kernel(const __grid_constant__ CUtensorMap tm0, const __grid_constant__ CUtensorMap tm1,
                                                                   GroupedArgs a) {
    chain_begin();
    extern __shared__ __align__(128) unsigned char smem[];
    float2* s_fold = reinterpret_cast<float2*>(smem + kOffFold);       // [warp][kFoldCells][lane]
    u64* raw_full = reinterpret_cast<u64*>(smem + kOffBars);
    u64* ready = raw_full + kStages;
    u64* empty = ready + kStages;
    volatile u32* s_abort = reinterpret_cast<u32*>(empty + kStages);
    u32* s_tile = reinterpret_cast<u32*>(smem + kOffTile);             // [kTilePlaces][kTileWords]
    u32* cum = reinterpret_cast<u32*>(smem + kOffCum);                 // [2][kTileCounts]

    if (kDown && block_skips(a.summary)) return;  // a failed or aborted projection skips the stage (routed_expert.hpp:17-19)

    const u32 tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    const u32 n_union = min(a.routes.counts[0], kMaxUnion);
    if (tid == 0) {
        for (u32 i = 0; i < kStages; ++i) { mbar_init(&raw_full[i], 1); mbar_init(&ready[i], kHelpers); mbar_init(&empty[i], kConsumers); }
        *s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    const u32 n_tiles = count_tiles<kGN, false>(a.routes, n_union, cum) * a.n_row_tiles;
    const u32 I = a.shape.inter, H = a.shape.hidden;
    const u32 nblocks = a.K / 256;
    bool ok = true;
    const u32 my_tiles = n_tiles > blockIdx.x ? (n_tiles - blockIdx.x + gridDim.x - 1) / gridDim.x : 0u;
    const u32 total = my_tiles * nblocks;  // stages of this CTA

    if (warp >= kConsumers) {
        // ================================================================================================= helpers
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kHelperRegs));
        const u32 lt = tid - kConsumers * 32, hw = lt >> 5;
        const u32 in_stride = a.in.stride ? a.in.stride : a.in.width, in_gs = in_stride / 32;
        u32 ik = 0, ib = 0, cy = 0;                      // tile and super-block of the next stage to request; the tile's first weight row
        u32 slot_r = 0, lap_r = 0, asked = 0;            // its ring place and lap; stages requested
        const float* t_deltas = nullptr;                 // the last warp: of token `lane`
        const i32* t_sums = nullptr;
        const i8* t_codes[kGN / 8];                      // a half warp copies the 256 codes of one token
        // the next tile, looked up a tile ahead: what it needs is a chain of reads from memory
        Tile nx{};
        u32 nx_src = 0, nx_slot = 0;
        auto look_ahead = [&](u32 k) {
            if (k >= my_tiles) return;
            nx = find_tile<kGN, false>(a.routes, a.n_row_tiles, cum, n_union, blockIdx.x + k * gridDim.x);
            const u32 ent = nx.eb + min(lane, nx.nt - 1u);
            nx_slot = a.routes.slots[ent];
            nx_src = kDown ? nx_slot : a.routes.rows[ent];
        };
        // Requests the next stage: rows by TMA, codes and {E, S} by asynchronous copies.
        auto request = [&]() {
            unsigned char* st = smem + slot_r * kStageBytes;
            if (ib == 0) {  // a new tile: its tokens' A8 rows and slots are published
                u32* ti = s_tile + (ik % kTilePlaces) * kTileWords;
                const u32 first = kDown ? min(kGM * nx.c, H - kGM) : min(kOutRows * nx.c, I - kOutRows);
                if (hw == 0) { ti[4 + lane] = nx_src; ti[4 + kGN + lane] = nx_slot; }
                if (lt == 0) { ti[0] = first; ti[1] = nx.nt; ti[2] = nx.eb; }
                t_deltas = a.in.deltas + u64(nx_src) * in_gs;
                t_sums = a.in.sums + u64(nx_src) * in_gs;
                cy = nx.expert * (kDown ? H : I) + first;
                asm volatile("bar.sync 1, %0;" ::"n"(kHelpers * 32) : "memory");
#pragma unroll
                for (u32 i = 0; i < kGN / 8; ++i) t_codes[i] = a.in.codes + u64(ti[4 + (kGN / 4) * hw + 2u * i + (lane >> 4)]) * in_stride + 16u * (lane & 15u);
                look_ahead(ik + 1);
            }
            if (ok && lap_r) ok = mbar_wait(&empty[slot_r], (lap_r - 1u) & 1u, kWaitLimit, s_abort);
            if (ok) {
                if (lt == 0) {
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the consumers' reads precede the copies below
                    mbar_expect_tx(&raw_full[slot_r], kRawBytes);
                    tma_2d(st, &tm0, ib * (kQ4KBlock / 8), cy, &raw_full[slot_r]);
                    tma_2d(st + kOutRows * kQ4KBlock, kDown ? &tm0 : &tm1, ib * (kQ4KBlock / 8), kDown ? cy + kOutRows : cy, &raw_full[slot_r]);
                    ++asked;
                }
                unsigned char* sc = st + kOffCode + ((kGN / 4) * hw + (lane >> 4)) * kCodePitch + 16u * (lane & 15u);
#pragma unroll
                for (u32 i = 0; i < kGN / 8; ++i) { cp_async16(sc + 2u * i * kCodePitch, t_codes[i]); t_codes[i] += 256; }
                if (hw == kHelpers - 1u) {
                    unsigned char* pv = st + kOffPriv + 64u * lane;
                    if (a.es_vec) {
                        cp_async16(pv, t_deltas);
                        cp_async16(pv + 16, t_deltas + 4);
                        cp_async16(pv + 32, t_sums);
                        cp_async16(pv + 48, t_sums + 4);
                    } else {
#pragma unroll 1
                        for (u32 i = 0; i < 8; ++i) {
                            cp_async4(pv + 4u * i, t_deltas + i);
                            cp_async4(pv + 32u + 4u * i, t_sums + i);
                        }
                    }
                    t_deltas += 8; t_sums += 8;
                }
            }
            if (++ib == nblocks) { ib = 0; ++ik; }
            if (++slot_r == kStages) { slot_r = 0; ++lap_r; }
        };
        look_ahead(0);
        u32 slot = 0, lap = 0;
        for (u32 m = 0; m < total; ++m) {
            // decoded as soon as it has landed, up to two stages before the consumers need it
            if (m == a.stall_stage) break;
            request();
            unsigned char* st = smem + slot * kStageBytes;
            asm volatile("cp.async.wait_all;" ::: "memory");
            if (ok) ok = mbar_wait(&raw_full[slot], lap & 1u, kWaitLimit, s_abort);
            ok = __all_sync(0xffffffffu, ok);
            if (ok) {  // else no more requests or hand-overs; the tile barrier above is still met by every helper
                if (hw < kHelpers - 1u) {
                    // rows 2 lt and 2 lt + 1; which one is read first alternates, for the banks of the 128-bit reads
                    const u32 swap = (lt >> 2) & 1u;
                    const uint4 ha = *reinterpret_cast<const uint4*>(st + (2u * lt + swap) * kQ4KBlock), hb = *reinterpret_cast<const uint4*>(st + (2u * lt + 1u - swap) * kQ4KBlock);
                    auto special = [](u32 w) { return (w & 0x7c00u) == 0x7c00u || (w & 0x7c000000u) == 0x7c000000u; };
                    const bool slow = __any_sync(0xffffffffu, special(ha.x) || special(hb.x));
                    // [pair][row pair][D, D, D', D' | -DM, -DM, -DM', -DM']
                    float4* fac = reinterpret_cast<float4*>(st + kOffFac) + 2u * lt;
#pragma unroll
                    for (u32 half = 0; half < 2; ++half) {
                        float fa[2][4], fb[2][4];
                        auto decode = [&](const uint4& h, float (&f)[2][4]) {
                            if (slow) {  // an infinity or a NaN: the products themselves
#pragma unroll 1
                                for (u32 i = 0; i < 2; ++i) {
                                    const Factors x = q4k_factors(h, 2u * half + i);
                                    const float v[4] = {x.Dl, __fmul_rn(x.Dh, 0.0625f), -x.DMl, -x.DMh};
#pragma unroll
                                    for (u32 k = 0; k < 4; ++k) { if (i == 0) f[0][k] = v[k]; else f[1][k] = v[k]; }
                                }
                            } else if (half == 0) {
                                fast_factors(h.x, h.y & 0x3f3f3f3fu, h.z & 0x3f3f3f3fu, f);
                            } else {
                                fast_factors(h.x, (h.w & 0x0f0f0f0fu) | ((h.y >> 2) & 0x30303030u), ((h.w >> 4) & 0x0f0f0f0fu) | ((h.z >> 2) & 0x30303030u), f);
                            }
                        };
                        decode(swap ? hb : ha, fa);
                        decode(swap ? ha : hb, fb);
#pragma unroll
                        for (u32 i = 0; i < 2; ++i) {
                            fac[(2u * half + i) * kGM] = make_float4(fa[i][0], fb[i][0], fa[i][1], fb[i][1]);
                            fac[(2u * half + i) * kGM + 1] = make_float4(fa[i][2], fb[i][2], fa[i][3], fb[i][3]);
                        }
                    }
                } else {
                    const unsigned char* pv = st + kOffPriv + 64u * lane;
                    float4* es = reinterpret_cast<float4*>(st + kOffEs) + lane;  // [pair][token] {E, E', S, S'}
#pragma unroll
                    for (u32 i = 0; i < 2; ++i) {
                        const float4 e = reinterpret_cast<const float4*>(pv)[i];
                        const int4 sm = reinterpret_cast<const int4*>(pv + 32)[i];
                        es[2 * i * kGN] = make_float4(e.x, e.y, static_cast<float>(sm.x), static_cast<float>(sm.y));
                        es[(2 * i + 1) * kGN] = make_float4(e.z, e.w, static_cast<float>(sm.z), static_cast<float>(sm.w));
                    }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&ready[slot]);
            }
            if (++slot == kStages) { slot = 0; ++lap; }
        }
        if (!ok && lt == 0) drain(raw_full, kStages, asked, kWaitLimit);  // else it has seen every stage land
    } else {
        // ================================================================================================ consumers
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kConsumerRegs));
        const u32 p = warp & 3u, third = warp >> 2;     // chain, 64 rows of the tile: gate/up 32 gate rows and the up rows of the same outputs
        const u32 row_base = (kDown ? 64u : 32u) * third;
        float* s_out = reinterpret_cast<float*>(smem + kOffFold + third * (kFoldBytes / kThirds));  // [kGN][kOutPitch], the third's
        const u32 fr = lane >> 2, ft = lane & 3u;       // fragments: token fr (and fr + 8) of a token tile, rows 2 ft and 2 ft + 1 of a row tile
        const u32 act_stride = a.act.stride ? a.act.stride : a.act.width;
        u32 slot = 0, parity = 0;
        for (u32 ik = 0; ik < my_tiles; ++ik) {
            const u32* ti = s_tile + (ik % kTilePlaces) * kTileWords;
            u32 n_mt = 0;
            float2 acc[kRowTiles][kTokTiles][2];
#pragma unroll
            for (int i = 0; i < (int)(kRowTiles * kTokTiles * 2); ++i) (&acc[0][0][0])[i] = make_float2(0.0f, 0.0f);
            for (u32 b = 0; b < nblocks; ++b) {
                // the helpers have seen the rows' copies complete before they arrive
                if (ok) ok = mbar_wait(&ready[slot], parity, kWaitLimit, s_abort);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) continue;
                const u32 next = slot + 1u == kStages ? 0u : slot + 1u, next_parity = parity ^ (next == 0u ? 1u : 0u);
                if (b == 0) n_mt = (ti[1] + 15u) / 16u;
                const unsigned char* st = smem + slot * kStageBytes;
                const unsigned char* rows = st + (row_base + fr) * kQ4KBlock + 16u + 32u * p + 4u * ft;
                const unsigned char* codes = st + kOffCode + fr * kCodePitch + 64u * p + 4u * ft;
                const float4* es = reinterpret_cast<const float4*>(st + kOffEs) + p * kGN + fr;
                const float4* fac = reinterpret_cast<const float4*>(st + kOffFac) + p * kGM + row_base + 2u * ft;
                if (n_mt == 2) superblock<2, !kDown>(rows, codes, es, fac, acc);
                else superblock<1, !kDown>(rows, codes, es, fac, acc);
                __syncwarp();
                if (lane == 0) mbar_arrive(&empty[slot]);
                slot = next; parity = next_parity;
            }
            // (a0 + a1) + (a2 + a3). Warp p hands half of its row tiles to warp p ^ 1 of its third and adds what that hands over, then does the
            // same with half of what is left and warp p ^ 2. Buffer p is written by warp p, then by warp p ^ 1 (which alone has read it), then
            // read by warp p ^ 3. The barriers are met on every path.
            asm volatile("bar.sync %0, 128;" ::"r"(4u + third) : "memory");  // the previous tile's last reads of the buffers and of s_out
            float2* bufs = s_fold + 4u * third * (kFoldCells * 32) + lane;
            float2* mine = bufs + p * (kFoldCells * 32);
            float2* theirs = bufs + (p ^ 1u) * (kFoldCells * 32);
            const float2* last = bufs + (p ^ 3u) * (kFoldCells * 32);
            const bool odd = p & 1u, high = p >> 1;
            auto add = [](float2 x, float2 y) { return make_float2(__fadd_rn(x.x, y.x), __fadd_rn(x.y, y.y)); };
            constexpr int n = 2 * kTokTiles;  // cells of a row tile
            float2* cells = &acc[0][0][0];
#pragma unroll
            for (int i = 0; i < 4 * n; ++i) mine[32 * i] = pick(odd, cells[i], cells[4 * n + i]);
            asm volatile("bar.sync %0, 128;" ::"r"(4u + third) : "memory");
            float2 out[2][kTokTiles][2];
#pragma unroll
            for (int i = 0; i < 2 * n; ++i) {
                const float2 s0 = add(pick(odd, cells[4 * n + i], cells[i]), theirs[32 * i]), s1 = add(pick(odd, cells[6 * n + i], cells[2 * n + i]), theirs[32 * (2 * n + i)]);
                theirs[32 * i] = pick(high, s0, s1);
                (&out[0][0][0])[i] = pick(high, s1, s0);
            }
            asm volatile("bar.sync %0, 128;" ::"r"(4u + third) : "memory");
#pragma unroll
            for (int i = 0; i < 2 * n; ++i) (&out[0][0][0])[i] = add((&out[0][0][0])[i], last[32 * i]);
            const u32 row0 = 32u * (p & 1u) + 16u * (p >> 1) + 2u * ft;  // the lane's first of the third's 64 rows in the two row tiles that are left to it
            const u32 nt = ok ? ti[1] : 0u, first = ti[0], eb = ti[2];
            if (kDown) {
#pragma unroll
                for (int cz = 0; cz < n; ++cz) {
                    const u32 tk = 8u * cz + fr;
                    if (tk < nt) {
                        float* to = a.raw + u64(ti[4 + kGN + tk]) * H + first + row_base + row0;
#pragma unroll
                        for (int i = 0; i < 2; ++i) {
                            const float2 v = out[i][cz >> 1][cz & 1];
                            if (a.raw_vec) *reinterpret_cast<float2*>(to + 8 * i) = v;
                            else { to[8 * i] = v.x; to[8 * i + 1] = v.y; }
                        }
                    }
                }
            } else {
                asm volatile("bar.sync %0, 128;" ::"r"(4u + third) : "memory");  // the buffers have been read
#pragma unroll
                for (int cz = 0; cz < n; ++cz) {
                    float* to = s_out + (8u * cz + fr) * kOutPitch + row0;
#pragma unroll
                    for (int i = 0; i < 2; ++i) *reinterpret_cast<float2*>(to + 8 * i) = out[i][cz >> 1][cz & 1];
                }
                asm volatile("bar.sync %0, 128;" ::"r"(4u + third) : "memory");
                // SwiGLU + the A8 rule over the third's 32 outputs of every token. No barrier here is met by more than the third's four warps, which lie on four
                // schedulers: while one third is at its tile's end, the others keep the schedulers busy.
                const u32 group = first / 32u + third, o_col = 32u * group + lane;
                for (u32 k0 = kTasks * p; k0 < nt; k0 += kTasks * 4u) {
                    float g[kTasks], u[kTasks], delta[kTasks];
                    int code[kTasks], sum[kTasks];
#pragma unroll
                    for (int i = 0; i < kTasks; ++i) {
                        const float* src = s_out + min(k0 + i, nt - 1u) * kOutPitch + lane;
                        g[i] = src[0]; u[i] = src[32];
                    }
                    const u32 bad = swiglu_a8(g, u, code, delta, sum);
#pragma unroll
                    for (int i = 0; i < kTasks; ++i) {
                        const u32 tk = k0 + i;
                        if (tk >= nt) break;
                        const u32 slot_id = ti[4 + kGN + tk];
                        if (a.gate_out) { a.gate_out[u64(slot_id) * I + o_col] = g[i]; a.up_out[u64(slot_id) * I + o_col] = u[i]; }
                        if (bad >> i & 1u) {  // fail closed: nothing of the group is written (routed_expert.cpp:147-156)
                            if (lane == 0) {
                                if (a.row_status) atomicOr(&a.row_status[a.routes.rows[eb + tk]], B200MOE_ROW_PROJECTION_NONFINITE);
                                if (a.summary) atomicOr(a.summary, B200MOE_ROW_PROJECTION_NONFINITE);
                            }
                            continue;
                        }
                        a.act.codes[u64(slot_id) * act_stride + o_col] = static_cast<i8>(code[i]);
                        if (lane == 0) {
                            a.act.deltas[u64(slot_id) * (act_stride / 32) + group] = delta[i];
                            if (a.act.sums) a.act.sums[u64(slot_id) * (act_stride / 32) + group] = sum[i];
                        }
                    }
                }
            }
        }
    }
    if (!ok && lane == 0 && a.summary) atomicOr(a.summary, kAbortBit);
}

bool es_units(const b200moe_a8_rows& x) {
    const u32 stride = x.stride ? x.stride : x.width;
    return stride % 128 == 0 && aligned(x.deltas, 16) && aligned(x.sums, 16);
}

}  // namespace

// Each stage by itself: gate/up is the same kernel whatever the down's blocks are. An expert has at least a tile of rows, whole groups of outputs.
bool grouped_gate_up_fits(const b200moe_gate_up_view& v) {
    const b200moe_shape& s = v.shape;
    return v.x.sums && s.gate_type == B200MOE_TYPE_Q4_K && s.hidden % 256 == 0 && s.inter % 32 == 0 && s.inter >= kOutRows && s.experts <= kMaxUnion;
}
bool grouped_down_fits(const b200moe_down_view& v) {
    const b200moe_shape& s = v.shape;
    return v.act.sums && s.gate_type == B200MOE_TYPE_Q4_K && s.down_type == B200MOE_TYPE_Q4_K && s.hidden % 256 == 0 && s.inter % 256 == 0 && s.experts <= kMaxUnion;
}
u32 grouped_row_tiles(u32 outputs, bool down) { return (outputs + (down ? kGM : kOutRows) - 1) / (down ? kGM : kOutRows); }

int launch_gate_up_q4k_grouped(const b200moe_gate_up_view& v, cudaStream_t stream) {
    if (v.max_union == 0) return B200MOE_OK;
    GroupedArgs a{};
    a.shape = v.shape; a.routes = v.routes; a.in = v.x; a.act = v.act;
    a.gate_out = v.gate_out; a.up_out = v.up_out; a.row_status = v.row_status; a.summary = v.summary;
    a.n_row_tiles = grouped_row_tiles(v.shape.inter, false); a.K = v.shape.hidden; a.es_vec = es_units(v.x); a.stall_stage = debug_waits().stall_stage;
    CUtensorMap tm0, tm1;
    const u64 rb = u64(v.shape.hidden / 256) * kQ4KBlock, rows = u64(v.shape.experts) * v.shape.inter;
    if (int rc = wide::rows_map(v.weights.gate, rb, rows, kQ4KBlock, kOutRows, &tm0)) return rc;
    if (int rc = wide::rows_map(v.weights.up, rb, rows, kQ4KBlock, kOutRows, &tm1)) return rc;
    if (int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(grouped_q4k_kernel<false>), kGroupedSmem)) return rc;
    chain_launch(grouped_q4k_kernel<false>, device_sm_count(), kGThreads, kGroupedSmem, stream, tm0, tm1, a);
    return after_launch("gate_up_q4k_grouped");
}

int launch_down_q4k_grouped(const b200moe_down_view& v, cudaStream_t stream) {
    if (v.max_union == 0) return B200MOE_OK;
    GroupedArgs a{};
    a.shape = v.shape; a.routes = v.routes; a.in = v.act; a.raw = v.raw;
    a.summary = const_cast<u32*>(v.summary);
    a.n_row_tiles = grouped_row_tiles(v.shape.hidden, true); a.K = v.shape.inter; a.es_vec = es_units(v.act); a.raw_vec = aligned(v.raw, 8); a.stall_stage = debug_waits().stall_stage;
    CUtensorMap tm0;
    if (int rc = wide::rows_map(v.weights.down, u64(v.shape.inter / 256) * kQ4KBlock, u64(v.shape.experts) * v.shape.hidden, kQ4KBlock, kOutRows, &tm0)) return rc;
    if (int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(grouped_q4k_kernel<true>), kGroupedSmem)) return rc;
    chain_launch(grouped_q4k_kernel<true>, device_sm_count(), kGThreads, kGroupedSmem, stream, tm0, tm0, a);
    return after_launch("down_q4k_grouped");
}

}  // namespace b200moe
