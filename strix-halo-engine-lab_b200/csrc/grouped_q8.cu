// Q8_0 x A8 experts, GROUPED form for windows whose experts have many entries: the lane-class contract of
// src/ds41_formats.cpp:188-197 (product_q8_0), bit for bit that of gemv_q8.cu / gemv_q8_mma.cu, with the class sums in registers.
//
// The contract adds the terms float(dot_g) * (scale_g * delta_g) of a row into 32 lane classes (group g -> class g % 32) in ascending
// g, then folds the classes with the butterfly v[l] += v[l ^ d], d = 16 .. 1. A unit = 256 columns = 8 blocks = 8 neighbouring classes:
// consumer warp b of a row half owns block b of every unit. The units are taken in the order u % 4 = 0, 2, 1, 3, ascending inside: after
// each of the four sets a warp's sums are class sums, and the butterfly's steps 16 and 8 are ((set 0 + set 2) + (set 1 + set 3)) of
// its own registers; steps 4, 2 and 1 run between the eight warps, once per tile, each warp handing over half of what it has.
// Tile = (expert, 64 weight rows, 32 of its tokens): 32 gate and 32 up rows of the same outputs, or 64 down rows.
//
// What bounds it: issue slots (two thirds of them busy). A 16 x 8 MMA of a block is followed by six packed FP32 operations (scale times
// delta, times the dot, plus the sum) and four conversions: 17 instructions and 23 clocks of a scheduler with its loads on a loop of its own, 19
// and 27 for an even block; in the kernel 33 instructions and 49 clocks, the rest being waits and addresses of every second unit, the
// meeting of the sets and warps once per tile, and SwiGLU. Eight warps of all 64 rows had fewer instructions (27 an MMA) and were slower
// (399 against 353 us a call, 512 rows below): two warps a scheduler do not cover each other's latencies.
// Both instantiations spill a little at their 96 registers (52 bytes stored and 100 loaded in gate/up, 48 and 80 in down).
// 512 rows x 4 over 64 experts of 2048 -> 1024: gate/up 173, down 112 us (344 and 253 in gemv_q8_mma.cu); 8192 rows of a dense
// 7168 -> 2048 block 2530 and 1430 us (4960 and 3810).
//
// A persistent CTA per SM walks tiles round-robin. Producer warps (4): the unit's weight rows by tiled TMA (272 bytes x 32 rows: rows lie
// 4 (mod 32) words apart, the fragment loads are conflict free), the tokens' codes and deltas by 16-byte asynchronous copies, all counted on
// the stage's mbarrier. The places of absent tokens keep what an earlier tile left there (their cells are never stored): copies of the tile's last token
// in them had every CTA ask for the same lines again and again (gate/up of one expert of 2048 x 17408, 16 rows: 56.6 us, 32.9 without).
// Consumer warps (16): mma.sync m16n8k32 (tokens x weight rows, s8 x s8) straight from shared memory; a lane's two neighbouring cells are two weight rows of one token (packed FP32). Q8_0 blocks are 34 bytes: the quants of an even block start 2 (mod 4)
// bytes in (two words and a byte permute per register), those of an odd block on a word.
// Every wait is bounded; on a timeout the roles stop working, the producers wait (bounded) for the copies in flight and the launch sets
// B200MOE_JOB_WAIT_ABORTED in the job summary.
#include <type_traits>

#include "grouped_common.cuh"
#include "wide_common.cuh"

namespace b200moe {
namespace {
using namespace q4k;   // the mbarrier / copy wrappers
using namespace grouped;

constexpr u32 kRows = 64, kTokens = 32;          // tile
constexpr u32 kBlocks = 8;                       // of a unit
constexpr u32 kUnitBytes = kBlocks * kQ8Block;   // 272
constexpr u32 kConsumers = 2 * kBlocks, kProducers = 4;  // warps
constexpr u32 kGThreads = (kConsumers + kProducers) * 32;
constexpr u32 kStages = 5;
constexpr u32 kCodePitch = 256 + 16, kDeltaPitch = 48;  // bytes: 4 and 12 (mod 32) words
constexpr u32 kOffCode = kRows * kUnitBytes, kOffDelta = kOffCode + kTokens * kCodePitch, kStageBytes = kOffDelta + kTokens * kDeltaPitch;
constexpr u32 kCells = 16;                       // float2 cells of a lane: [row tile 4][token tile 2][2]
constexpr u32 kSumBytes = kConsumers * kCells * 32 * 8;
constexpr u32 kOutPitch = kRows + 8;             // floats: the 8-byte stores of a half warp (four tokens, four row pairs) meet every bank once
constexpr u32 kOutBytes = kTokens * kOutPitch * 4;
// What the consumers need of a tile: {row tile, tokens, first entry}, its tokens' A8 rows, its tokens' slots. The producers run at most
// kStages stages ahead, a tile has at least one: eight places.
constexpr u32 kTilePlaces = 8, kTileWords = 4 + 2 * kTokens;
constexpr u32 kOffSum = kStages * kStageBytes, kOffOut = kOffSum + kSumBytes, kOffBars = kOffOut + kOutBytes, kOffTile = kOffBars + 2 * kStages * 8 + 8,
              kOffCum = kOffTile + kTilePlaces * kTileWords * 4, kSmem = kOffCum + 2 * kTileCounts * 4;
static_assert(kStageBytes % 128 == 0 && (32 * kUnitBytes) % 128 == 0 && kOffBars % 8 == 0, "TMA destinations, barriers");
static_assert(kSmem > 114u * 1024u && kSmem <= 227u * 1024u, "one CTA per SM, within the shared memory of an SM");
constexpr u32 kLaunchRegs = 65536u / kGThreads / 8u * 8u, kProducerRegs = 64;
constexpr u32 kConsumerRegs = (kGThreads * kLaunchRegs - kProducers * 32u * kProducerRegs) / (kConsumers * 32u) / 8u * 8u;
static_assert(kConsumers * 32 * kConsumerRegs + kProducers * 32 * kProducerRegs <= kGThreads * kLaunchRegs, "setmaxnreg split exceeds the launch's registers");

struct Q8Args {
    b200moe_shape shape;
    b200moe_routes routes;
    b200moe_a8_rows in;      // x (gate/up: indexed by row) or act (down: indexed by slot)
    b200moe_a8_rows act;     // gate/up output
    float* gate_out;
    float* up_out;
    float* raw;              // down output [slots][hidden]
    u32* summary;
    u32 n_row_tiles;         // inter / 32 (gate/up) or hidden / 64 (down)
    u32 K;                   // hidden (gate/up) or inter (down)
    u32 delta_vec;           // the input's deltas lie in whole 16-byte units
    u32 raw_vec;             // raw lies on an 8-byte boundary
    Waits waits;
};

// 16 tokens x 8 weight rows x one block. d[z]: token lane / 4 + 8 z, weight rows 2 (lane % 4) and the next.
__device__ __forceinline__ void mma_dots(int2 (&d)[2], const u32 (&a)[4], u32 b0, u32 b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
        : "=r"(d[0].x), "=r"(d[0].y), "=r"(d[1].x), "=r"(d[1].y) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "r"(0));
}

// One block of one unit: the warp's 32 rows against NMT 16-token tiles. rows: block of weight row lane / 4; scales: block of weight row
// 2 (lane % 4); codes / deltas: token lane / 4 at this block, the codes at the lane's k slice. acc[j][mt][z]: rows 8 j + 2 (lane % 4)
// and the next of token 16 mt + 8 z + lane / 4. ODD: the block's position in the unit is odd (quants on a word).
template <bool ODD, int NMT>
__device__ __forceinline__ void unit_step(const unsigned char* rows, const unsigned char* scales, const unsigned char* codes, const unsigned char* deltas, u32 t4,
                                          float2 (&acc)[4][2][2]) {
    u32 a[NMT][4];
    float dl[NMT][2];
#pragma unroll
    for (int mt = 0; mt < NMT; ++mt)
#pragma unroll
        for (int z = 0; z < 2; ++z) {
            const unsigned char* c = codes + (16 * mt + 8 * z) * kCodePitch;
            a[mt][z] = *reinterpret_cast<const u32*>(c);
            a[mt][z + 2] = *reinterpret_cast<const u32*>(c + 16);
            dl[mt][z] = *reinterpret_cast<const float*>(deltas + (16 * mt + 8 * z) * kDeltaPitch);
        }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const u32* q = reinterpret_cast<const u32*>(rows + 8 * j * kUnitBytes + (ODD ? 2u : 0u) + 4u * t4);
        const u32 b0 = ODD ? q[0] : __byte_perm(q[0], q[1], 0x5432u), b1 = ODD ? q[4] : __byte_perm(q[4], q[5], 0x5432u);
        const unsigned char* sc = scales + 8 * j * kUnitBytes;
        const float2 s = make_float2(half_bits_to_float(*reinterpret_cast<const unsigned short*>(sc)), half_bits_to_float(*reinterpret_cast<const unsigned short*>(sc + kUnitBytes)));
#pragma unroll
        for (int mt = 0; mt < NMT; ++mt) {
            int2 d[2];
            mma_dots(d, a[mt], b0, b1);
#pragma unroll
            for (int z = 0; z < 2; ++z) acc[j][mt][z] = add2(mul2(to_float(d[z]), mul2(s, both(dl[mt][z]))), acc[j][mt][z]);
        }
    }
}

template <bool kDown>
__global__ void __launch_bounds__(kGThreads, 1) grouped_q8_kernel(const __grid_constant__ CUtensorMap tm0, const __grid_constant__ CUtensorMap tm1, Q8Args a) {
    chain_begin();
    extern __shared__ __align__(128) unsigned char smem[];
    float2* s_sum = reinterpret_cast<float2*>(smem + kOffSum);         // [row half][block][cell][lane]
    float* s_out = reinterpret_cast<float*>(smem + kOffOut);           // [kTokens][kOutPitch]
    u64* full = reinterpret_cast<u64*>(smem + kOffBars);
    u64* empty = full + kStages;
    volatile u32* s_abort = reinterpret_cast<u32*>(empty + kStages);   // and the stages that the first producer has asked for
    u32* s_tile = reinterpret_cast<u32*>(smem + kOffTile);             // [kTilePlaces][kTileWords]
    u32* cum = reinterpret_cast<u32*>(smem + kOffCum);                 // [2][kTileCounts]

    if (kDown && block_skips(a.summary)) return;  // an aborted projection skips the stage

    const u32 tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    const u32 n_union = min(a.routes.counts[0], kMaxUnion);
    if (tid == 0) {
        for (u32 i = 0; i < kStages; ++i) { mbar_init(&full[i], kProducers * 32 + 1); mbar_init(&empty[i], kConsumers); }
        *s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    const u32 n_tiles = count_tiles<kTokens, true>(a.routes, n_union, cum) * a.n_row_tiles;
    const u32 I = a.shape.inter, H = a.shape.hidden;
    const u32 units = a.K / 256;
    bool ok = true;
    const u32 my_tiles = n_tiles > blockIdx.x ? (n_tiles - blockIdx.x + gridDim.x - 1) / gridDim.x : 0u;
    const u32 total = my_tiles * units;  // stages of this CTA

    if (warp >= kConsumers) {
        // =============================================================================================== producers
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kProducerRegs));
        const u32 lt = tid - kConsumers * 32, hw = lt >> 5;
        const u32 in_stride = a.in.stride ? a.in.stride : a.in.width, in_gs = in_stride / 32;
        u32 ring = 0, lap = 0, ik = 0, u = 0, cy = 0;    // u: unit of the next stage; cy: the tile's first weight row
        u32 fed = 0, t_nt = 0;                           // stages that this warp has asked for; tokens of the tile
        bool fresh = true;                               // the next stage begins a tile
        const i8* t_codes[kTokens / 8];                  // a half warp copies the 256 codes of one token
        const float* t_deltas = nullptr;                 // two threads copy the 8 deltas of one token
        // the next tile, looked up a tile ahead: what it needs is a chain of reads from memory
        Tile nx{};
        u32 nx_src = 0, nx_slot = 0;
        auto look_ahead = [&](u32 k) {
            if (k >= my_tiles) return;
            nx = find_tile<kTokens, true>(a.routes, a.n_row_tiles, cum, n_union, blockIdx.x + k * gridDim.x);
            const u32 ent = nx.eb + min(lane, nx.nt - 1u);
            nx_slot = a.routes.slots[ent];
            nx_src = kDown ? nx_slot : a.routes.rows[ent];
        };
        look_ahead(0);
        for (u32 m = 0; m < total; ++m) {
            if (fresh) {  // a new tile: its tokens' A8 rows and slots are published
                u32* ti = s_tile + (ik % kTilePlaces) * kTileWords;
                if (hw == 0) { ti[4 + lane] = nx_src; ti[4 + kTokens + lane] = nx_slot; }
                if (lt == 0) { ti[0] = nx.c; ti[1] = nx.nt; ti[2] = nx.eb; }
                cy = kDown ? nx.expert * H + kRows * nx.c : nx.expert * I + 32u * nx.c;
                asm volatile("bar.sync 1, %0;" ::"n"(kProducers * 32) : "memory");
#pragma unroll
                for (u32 i = 0; i < kTokens / 8; ++i) t_codes[i] = a.in.codes + u64(ti[4 + (kTokens / 4) * hw + 2u * i + (lane >> 4)]) * in_stride + 16u * (lane & 15u);
                t_deltas = a.in.deltas + u64(ti[4 + ((lt & 63u) >> 1)]) * in_gs + 4u * (lt & 1u);
                t_nt = nx.nt;
                look_ahead(ik + 1);
                fresh = false;
            }
            const bool feed = m < a.waits.stall_stage;
            if (ok && feed && lap) ok = mbar_wait(&empty[ring], (lap - 1u) & 1u, a.waits.limit, s_abort);
            ok = __all_sync(0xffffffffu, ok);
            if (ok && feed) {
                ++fed;
                unsigned char* st = smem + ring * kStageBytes;
                if (lt == 0) {
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the consumers' reads precede the copies below
                    mbar_expect_tx(&full[ring], kRows * kUnitBytes);
                    tma_2d(st, &tm0, u * (kUnitBytes / 8), cy, &full[ring]);
                    tma_2d(st + 32u * kUnitBytes, kDown ? &tm0 : &tm1, u * (kUnitBytes / 8), kDown ? cy + 32u : cy, &full[ring]);
                }
                unsigned char* sc = st + kOffCode + ((kTokens / 4) * hw + (lane >> 4)) * kCodePitch + 16u * (lane & 15u);
#pragma unroll
                for (u32 i = 0; i < kTokens / 8; ++i)
                    if ((kTokens / 4) * hw + 2u * i + (lane >> 4) < t_nt) cp_async16(sc + 2u * i * kCodePitch, t_codes[i] + 256u * u);
                if (lt < 2 * t_nt) {
                    unsigned char* sd = st + kOffDelta + (lt >> 1) * kDeltaPitch + 16u * (lt & 1u);
                    if (a.delta_vec) cp_async16(sd, t_deltas + 8u * u);
                    else
#pragma unroll
                        for (u32 i = 0; i < 4; ++i) cp_async4(sd + 4u * i, t_deltas + 8u * u + i);
                }
                asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(saddr(&full[ring])) : "memory");
            }
            if (++ring == kStages) { ring = 0; ++lap; }
            // the order of the units: u % 4 = 0, 2, 1, 3, ascending inside; a set may be empty
            u += 4;
            while (u >= units) {
                const u32 set = u & 3u;
                if (set == 3u) { u = 0; ++ik; fresh = true; break; }
                u = set == 0u ? 2u : set == 2u ? 1u : 3u;
            }
        }
        // The last producer to leave has seen every copy land, on every path: a consumer's wait may run out after the last stage was asked for.
        // A warp that gave up earlier than the first one makes up for its arrivals, so that the stages' phases complete.
        asm volatile("cp.async.wait_all;" ::: "memory");
        if (lt == 0) s_abort[1] = fed;
        asm volatile("bar.sync 1, %0;" ::"n"(kProducers * 32) : "memory");
        const u32 asked = s_abort[1];
        for (; fed < asked; ++fed) mbar_arrive(&full[fed % kStages]);
        if (lt == 0) drain(full, kStages, asked, a.waits.limit);
    } else {
        // =============================================================================================== consumers
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kConsumerRegs));
        // even blocks cost more instructions: every scheduler (warp % 4) gets two of each
        const u32 half = warp >> 3, b = (warp & 7u) ^ ((warp >> 2) & 1u);
        const u32 g = lane >> 2, t = lane & 3u;          // fragments: token g (and g + 8) of a token tile, rows 2 t and 2 t + 1 of a row tile
        const u32 act_stride = a.act.stride ? a.act.stride : a.act.width;
        const u32 off_rows = (32u * half + g) * kUnitBytes + kQ8Block * b, off_scales = (32u * half + 2u * t) * kUnitBytes + kQ8Block * b;
        const u32 off_codes = kOffCode + g * kCodePitch + 32u * b + 4u * t, off_deltas = kOffDelta + g * kDeltaPitch + 4u * b;
        float2* sums = s_sum + (8u * half) * (kCells * 32) + lane;  // + block * kCells * 32: of the warps of this row half
        float2* mine = sums + b * (kCells * 32);
        u32 ring = 0, parity = 0;
        for (u32 ik = 0; ik < my_tiles; ++ik) {
            const u32* ti = s_tile + (ik % kTilePlaces) * kTileWords;
            u32 nt = 0;
            float2 acc[4][2][2], sum[4][2][2];
            float2 *cells = &acc[0][0][0], *pair = &sum[0][0][0];
            // the units first, first + 4, ... on top of c, two at a time: a wait, its vote and the addresses are a third of a unit's instructions
            auto run_set = [&](u32 first_unit, float2 (&c)[4][2][2]) {
#pragma unroll
                for (int i = 0; i < (int)kCells; ++i) (&c[0][0][0])[i] = make_float2(0.0f, 0.0f);
                u32 left = units > first_unit ? (units - first_unit + 3u) / 4u : 0u;
#pragma unroll 1
                while (left) {
                    const bool two = left > 1u;
                    const u32 next = ring + 1u == kStages ? 0u : ring + 1u, next_parity = parity ^ (next == 0u ? 1u : 0u);
                    if (ok) ok = mbar_wait(&full[ring], parity, a.waits.limit, s_abort);
                    if (ok && two) ok = mbar_wait(&full[next], next_parity, a.waits.limit, s_abort);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                    if (nt == 0) nt = ti[1];
                    const unsigned char *st = smem + ring * kStageBytes, *st2 = smem + next * kStageBytes;
                    auto step = [&](auto odd, auto nmt) {
                        constexpr bool kOdd = decltype(odd)::value;
                        constexpr int kNmt = decltype(nmt)::value;
                        unit_step<kOdd, kNmt>(st + off_rows, st + off_scales, st + off_codes, st + off_deltas, t, c);
                        if (two) unit_step<kOdd, kNmt>(st2 + off_rows, st2 + off_scales, st2 + off_codes, st2 + off_deltas, t, c);
                    };
                    using Odd = std::true_type;
                    using Even = std::false_type;
                    if (nt > 16u) {
                        if (b & 1u) step(Odd{}, std::integral_constant<int, 2>{});
                        else step(Even{}, std::integral_constant<int, 2>{});
                    } else {
                        if (b & 1u) step(Odd{}, std::integral_constant<int, 1>{});
                        else step(Even{}, std::integral_constant<int, 1>{});
                    }
                    __syncwarp();
                    if (lane == 0) {
                        mbar_arrive(&empty[ring]);
                        if (two) mbar_arrive(&empty[next]);
                    }
                    ring = next; parity = next_parity;
                    if (two && ++ring == kStages) { ring = 0; parity ^= 1u; }
                    left -= two ? 2u : 1u;
                }
            };
            // steps 16 and 8 of the butterfly: (set 0 + set 2) + (set 1 + set 3), the first pair kept in shared memory
#pragma unroll 1
            for (u32 h = 0; h < 2; ++h) {
                run_set(h, sum);
                run_set(h + 2u, acc);
#pragma unroll
                for (int i = 0; i < (int)kCells; ++i) pair[i] = add2(pair[i], cells[i]);
                if (h == 0) {
#pragma unroll
                    for (int i = 0; i < (int)kCells; ++i) mine[32 * i] = pair[i];  // a barrier since the last reads at the previous tile's end
                } else {
#pragma unroll
                    for (int i = 0; i < (int)kCells; ++i) cells[i] = add2(mine[32 * i], pair[i]);
                }
            }
            // steps 4, 2 and 1: half of the cells go to the other warp each time, the barriers are met on every path
            float2 s8[8], s4[4], out[2];
            {
                const bool up = b & 4u;
                const float2* theirs = sums + (b ^ 4u) * (kCells * 32);
#pragma unroll
                for (int i = 0; i < 8; ++i) mine[32 * i] = pick(up, cells[i], cells[8 + i]);
                if (kDown) asm volatile("bar.sync %0, 256;" ::"r"(4u + half) : "memory");
                else asm volatile("bar.sync 2, %0;" ::"n"(kConsumers * 32) : "memory");  // every warp: the previous tile's reads of s_out too
#pragma unroll
                for (int i = 0; i < 8; ++i) s8[i] = add2(pick(up, cells[8 + i], cells[i]), theirs[32 * i]);
            }
            {
                const bool up = b & 2u;
                const float2* theirs = sums + (b ^ 2u) * (kCells * 32);
#pragma unroll
                for (int i = 0; i < 4; ++i) mine[32 * (8 + i)] = pick(up, s8[i], s8[4 + i]);
                asm volatile("bar.sync %0, 256;" ::"r"(4u + half) : "memory");
#pragma unroll
                for (int i = 0; i < 4; ++i) s4[i] = add2(pick(up, s8[4 + i], s8[i]), theirs[32 * (8 + i)]);
            }
            {
                const bool up = b & 1u;
                const float2* theirs = sums + (b ^ 1u) * (kCells * 32);
#pragma unroll
                for (int i = 0; i < 2; ++i) mine[32 * (12 + i)] = pick(up, s4[i], s4[2 + i]);
                asm volatile("bar.sync %0, 256;" ::"r"(4u + half) : "memory");
#pragma unroll
                for (int i = 0; i < 2; ++i) out[i] = add2(pick(up, s4[2 + i], s4[i]), theirs[32 * (12 + i)]);
            }
            // what is left to the lane: rows row, row + 1 of tokens tk, tk + 8
            const u32 row = 32u * half + 16u * (b >> 2) + 8u * ((b >> 1) & 1u) + 2u * t, tk = 16u * (b & 1u) + g;
            if (!ok) nt = 0;
            if (kDown) {
                asm volatile("bar.sync %0, 256;" ::"r"(4u + half) : "memory");  // the sums have been read
#pragma unroll
                for (u32 z = 0; z < 2; ++z) {
                    if (tk + 8u * z >= nt) break;
                    float* to = a.raw + u64(ti[4 + kTokens + tk + 8u * z]) * H + kRows * ti[0] + row;
                    if (a.raw_vec) *reinterpret_cast<float2*>(to) = out[z];
                    else { to[0] = out[z].x; to[1] = out[z].y; }
                }
            } else {
#pragma unroll
                for (u32 z = 0; z < 2; ++z) *reinterpret_cast<float2*>(s_out + (tk + 8u * z) * kOutPitch + row) = out[z];
                asm volatile("bar.sync 2, %0;" ::"n"(kConsumers * 32) : "memory");  // the outputs are there, the sums have been read
                // swiglu_clamped + the A8 rule over the 32 outputs of a token (src/ds41_moe.cpp:134-146)
                for (u32 k = warp; k < nt; k += kConsumers) {
                    const float gv = s_out[k * kOutPitch + lane], uv = s_out[k * kOutPitch + 32u + lane];
                    const u32 slot_id = ti[4 + kTokens + k], group = ti[0], o_col = 32u * group + lane;
                    if (a.gate_out) { a.gate_out[u64(slot_id) * I + o_col] = gv; a.up_out[u64(slot_id) * I + o_col] = uv; }
                    const float h = swiglu_ds41(gv, uv, a.shape.limit);  // NaN propagates: this family has no status rule
                    float delta;
                    int sum;
                    const int code = a8_quantize_lane(h, &delta, &sum);
                    a.act.codes[u64(slot_id) * act_stride + o_col] = static_cast<i8>(code);
                    if (lane == 0) {
                        a.act.deltas[u64(slot_id) * (act_stride / 32) + group] = delta;
                        if (a.act.sums) a.act.sums[u64(slot_id) * (act_stride / 32) + group] = sum;
                    }
                }
            }
        }
    }
    if (!ok && lane == 0 && a.summary) atomicOr(a.summary, kAbortBit);
}

bool shape_ok(const b200moe_shape& s, u32 K, u32 row_multiple, u32 rows) {
    return s.gate_type == B200MOE_TYPE_Q8_0 && s.down_type == B200MOE_TYPE_Q8_0 && K % 256 == 0 && rows % row_multiple == 0 && s.experts <= kMaxUnion;
}
bool delta_units(const b200moe_a8_rows& x) { return (x.stride ? x.stride : x.width) % 128 == 0 && aligned(x.deltas, 16); }

}  // namespace

bool grouped_q8_gate_up_fits(const b200moe_gate_up_view& v) {
    return shape_ok(v.shape, v.shape.hidden, 32, v.shape.inter) && aligned(v.weights.gate, 16) && aligned(v.weights.up, 16);
}
bool grouped_q8_down_fits(const b200moe_down_view& v) { return shape_ok(v.shape, v.shape.inter, kRows, v.shape.hidden) && aligned(v.weights.down, 16); }

int launch_gate_up_q8_grouped(const b200moe_gate_up_view& v, cudaStream_t stream) {
    if (v.max_union == 0) return B200MOE_OK;
    Q8Args a{};
    a.shape = v.shape; a.routes = v.routes; a.in = v.x; a.act = v.act; a.gate_out = v.gate_out; a.up_out = v.up_out; a.summary = v.summary;
    a.n_row_tiles = v.shape.inter / 32; a.K = v.shape.hidden; a.delta_vec = delta_units(v.x); a.waits = debug_waits();
    CUtensorMap tm0, tm1;
    const u64 rb = u64(v.shape.hidden / 32) * kQ8Block, rows = u64(v.shape.experts) * v.shape.inter;
    if (int rc = wide::rows_map(v.weights.gate, rb, rows, kUnitBytes, 32, &tm0)) return rc;
    if (int rc = wide::rows_map(v.weights.up, rb, rows, kUnitBytes, 32, &tm1)) return rc;
    if (int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(grouped_q8_kernel<false>), kSmem)) return rc;
    chain_launch(grouped_q8_kernel<false>, device_sm_count(), kGThreads, kSmem, stream, tm0, tm1, a);
    return after_launch("gate_up_q8_grouped");
}

int launch_down_q8_grouped(const b200moe_down_view& v, cudaStream_t stream) {
    if (v.max_union == 0) return B200MOE_OK;
    Q8Args a{};
    a.shape = v.shape; a.routes = v.routes; a.in = v.act; a.raw = v.raw; a.summary = const_cast<u32*>(v.summary);
    a.n_row_tiles = v.shape.hidden / kRows; a.K = v.shape.inter; a.delta_vec = delta_units(v.act); a.raw_vec = aligned(v.raw, 8); a.waits = debug_waits();
    CUtensorMap tm0;
    if (int rc = wide::rows_map(v.weights.down, u64(v.shape.inter / 32) * kQ8Block, u64(v.shape.experts) * v.shape.hidden, kUnitBytes, 32, &tm0)) return rc;
    if (int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(grouped_q8_kernel<true>), kSmem)) return rc;
    chain_launch(grouped_q8_kernel<true>, device_sm_count(), kGThreads, kSmem, stream, tm0, tm0, a);
    return after_launch("down_q8_grouped");
}

}  // namespace b200moe
