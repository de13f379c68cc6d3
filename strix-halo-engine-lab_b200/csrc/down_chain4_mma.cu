// Q8_0 / Q5_1 down in the four-chain rule (routed_expert.cpp:110-144) for windows whose experts have several entries: the integer dots on the tensor cores, bit for
// bit the forms of gemv_q4k.cu. Chain c = g % 4 adds E_g * (d * float(dot) [+ m * float(S_g)]) in ascending g; value = (acc0 + acc1) + (acc2 + acc3).
//
// Item = (expert, 64 or 32 weight rows), which lie one behind the other in memory: untiled copies, two items in flight. A step = an item against up to 32 (or 16) of its
// entries, whose A8 rows come by asynchronous copies a step ahead; the weights stay for the item's further steps. A warp has one chain of 16 weight rows (the MMA's rows)
// against the step's entries, eight an MMA (mma.sync m16n8k32, s8 x s8, one block); the chains meet in shared memory at the step's end, and a warp an entry stores the sums.
// One CTA of 16 warps an SM: two items and two steps of long rows fill its shared memory.
// What bounds it: latency with four warps a scheduler (issue slots 47 to 59 % busy; a warp's wait between dependent instructions and, with few entries, a step's ends - two barriers,
// the entries' copies, the meeting - are the top stalls) and the instructions beside the MMAs: 67 of all warps an MMA at 8 entries an expert (95 of Q5_1), 41 at 64. More items in flight
// and two CTAs of 8 warps an SM gave nothing; a k order that reads 8 Q8_0 quants as three words cost bank conflicts (1024 rows below 182 -> 186 us).
// 64 experts of 768 -> 2560, top 4, Q8_0, us a launch, the dp4a form and this: 64 rows 69 and 43, 128 111 and 48, 1024 686 and 164.
// Q8_0 blocks are 34 bytes: a lane reads two words and a byte permute puts its quants together where they do not lie on one.
// Every wait is bounded; where one runs out B200MOE_JOB_WAIT_ABORTED is set in the job summary once the copies in flight have landed.
#include <algorithm>
#include <type_traits>

#include "grouped_common.cuh"
#include "kernels.cuh"
#include "q4k_row.cuh"

namespace b200moe {
namespace {
using namespace q4k;
using namespace grouped;

constexpr u32 kChainThreads = 512, kChainWarps = kChainThreads / 32;

struct ChainMmaPlan {
    u32 n_chunks, stage_bytes;
    u32 copy_rows, row_gap;              // rows of a copy, bytes left free behind them
    u32 form, max_union;
    u32 early, wait_limit, stall_stage;  // test hook: item `stall_stage` of a CTA's items and those behind it are not asked for
};
// An entry's block of a step in shared memory: its codes, delta and sum, 12 words, so that eight entries' word reads meet every bank once and every offset is known when the
// loop is compiled. Apart, with pitches out of the plan, their addresses were a third of the instructions.
constexpr u32 kCell = 48, kCellDelta = 32, kCellSum = 36;

__device__ __forceinline__ void mma_s8(int (&d)[4], const u32 (&a)[4], u32 b0, u32 b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "r"(0));
}

__device__ __forceinline__ u32 lds16(u32 a) { u16 v; asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a)); return v; }

// A row's blocks of one chain, for one lane: its quants 4 t .. 4 t + 3 and 16 + 4 t .., the factor and the minimum. Four Q8_0 blocks are whole words, so all of a chain's blocks
// of a row begin alike, on a word or between two. A word past the block's end may be read, of which nothing is used.
template <bool Q51>
struct ChainRow {
    u32 at, quants, sel;
    __device__ ChainRow(u32 first, u32 t) : at(first), quants(Q51 ? first + 8u + 4u * t : (first & 2u ? first + 2u : first) + 4u * t), sel(first & 2u ? 0x3210u : 0x5432u), bits(4u * t) {}
    u32 bits;
    __device__ __forceinline__ void next() { constexpr u32 step = 4u * (Q51 ? kQ51Block : kQ8Block); at += step; quants += step; }
    __device__ __forceinline__ void read(u32& lo, u32& hi, float& d, float& m) const {
        if (Q51) {
            const uint2 head = lds64(at);
            const u32 q = lds32(quants);
            d = half_bits_to_float(head.x & 0xffffu);
            m = half_bits_to_float(head.x >> 16);
            auto spread = [](u32 x) { return ((x & 15u) * 0x02040810u) & 0x10101010u; };  // bit k of four to bit 4 of byte k
            lo = (q & 0x0f0f0f0fu) | spread(head.y >> bits);
            hi = ((q >> 4) & 0x0f0f0f0fu) | spread(head.y >> (16u + bits));
        } else {
            d = half_bits_to_float(lds16(at));
            m = 0.0f;
            lo = __byte_perm(lds32(quants), lds32(quants + 4u), sel);
            hi = __byte_perm(lds32(quants + 16u), lds32(quants + 20u), sel);
        }
    }
};

// RT: row tiles of 16 of an item; EG: shares of the entries; NT: entry tiles of 8 of a warp. 4 chains x RT x EG = 16 warps.
template <bool Q51, u32 RT, u32 EG, u32 NT>
__global__ void __launch_bounds__(kChainThreads, 1) down_chain4_mma_kernel(b200moe_down_view v, ChainMmaPlan plan) {
    static_assert(4 * RT * EG == kChainWarps);
    extern __shared__ __align__(128) unsigned char smem[];
    constexpr u32 R = 16 * RT, kCap = 8 * EG * NT, block = Q51 ? kQ51Block : kQ8Block, kMeet = R + 4;
    const u32 H = v.shape.hidden, I = v.shape.inter, groups = I / 32, row_bytes = groups * block, a8_bytes = groups * kCap * kCell;
    __shared__ u64 full[2];
    __shared__ u32 s_abort, s_slots[2][32];
    unsigned char* a8 = smem + 2 * plan.stage_bytes;                 // [2][group][entry] cells
    float* s_meet = reinterpret_cast<float*>(a8 + 2 * a8_bytes);     // [chain][entry][kMeet]
    u32* s_begins = reinterpret_cast<u32*>(s_meet + 4 * kCap * kMeet);
    u32* s_experts = s_begins + plan.max_union + 1;
    const u32 tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    if (tid == 0) {
        mbar_init(&full[0], kChainWarps); mbar_init(&full[1], kChainWarps);
        s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (!plan.early) chain_begin();
    const u32 n_union = min(load_l2(v.routes.counts), plan.max_union), n_items = n_union * plan.n_chunks;
    for (u32 j = tid; j <= n_union; j += kChainThreads) {
        s_begins[j] = load_l2(v.routes.begins + j);
        if (j < n_union) s_experts[j] = load_l2(v.routes.experts + j);
    }
    __syncthreads();
    struct Item { u32 id, j, chunk; };  // j: place of its expert in the union. The CTA's items are gridDim.x apart
    const u32 dj = gridDim.x / plan.n_chunks, dc = gridDim.x - dj * plan.n_chunks;
    auto onward = [&](Item& x) {
        x.id += gridDim.x; x.j += dj; x.chunk += dc;
        if (x.chunk >= plan.n_chunks) { x.chunk -= plan.n_chunks; ++x.j; }
    };
    const Item first_item{blockIdx.x, blockIdx.x / plan.n_chunks, blockIdx.x % plan.n_chunks};
    const u32 copies = R / plan.copy_rows, copy_bytes = plan.copy_rows * row_bytes, my_copies = warp < copies ? (copies - warp + kChainWarps - 1u) / kChainWarps : 0u;
    auto ask = [&](u32 n, const Item& x) {  // lane 0 of every warp: its share of the item's copies
        const unsigned char* from = v.weights.down + (u64(s_experts[x.j]) * H + R * x.chunk) * row_bytes;
        unsigned char* to = smem + (n & 1u) * plan.stage_bytes;
        if (my_copies) mbar_expect_tx(&full[n & 1u], my_copies * copy_bytes);
        else mbar_arrive(&full[n & 1u]);
        for (u32 k = warp; k < copies; k += kChainWarps) bulk_g2s(to + k * (copy_bytes + plan.row_gap), from + k * copy_bytes, copy_bytes, &full[n & 1u]);
    };
    u32 asked = 0;
    Item to_ask = first_item;
    const u32 n_ask = plan.stall_stage == 0xffffffffu ? n_items : min(n_items, blockIdx.x + plan.stall_stage * gridDim.x);
    for (; asked < 2 && to_ask.id < n_ask; ++asked, onward(to_ask))
        if (lane == 0) ask(asked, to_ask);
    if (plan.early) chain_begin();
    auto drain_asked = [&](u32 from) {  // one thread: the copies asked for land (the wait is bounded) before the CTA retires
        for (u32 n = from; n < asked; ++n)
            for (u32 i = 0; i < (plan.wait_limit >> 4) + 64u; ++i)
                if (mbar_try_wait(&full[n & 1u], (n >> 1) & 1u, kWaitHintNs)) break;
    };
    if (block_skips(v.summary)) {  // a failed projection skips the whole down stage (routed_expert.hpp:17-19)
        if (tid == 0) drain_asked(0);
        return;
    }
    const u32 stride = v.act.stride ? v.act.stride : v.act.width;
    struct Step { Item item; u32 first, nr, last; };  // entries first .. first + nr; whether they are the item's last
    auto step_at = [&](const Item& x, u32 first) {
        const u32 end = s_begins[x.j + 1], nr = min(kCap, end - first);
        return Step{x, first, nr, first + nr == end ? 1u : 0u};
    };
    auto item_begin = [&](const Item& x) { return x.id < n_items ? step_at(x, s_begins[x.j]) : Step{x, 0, 0, 1}; };
    auto after = [&](const Step& s) {
        if (!s.last) return step_at(s.item, s.first + s.nr);
        Item x = s.item;
        onward(x);
        return item_begin(x);
    };
    // the step's slots, two entries a warp, asked for a step ahead of their rows
    auto slots_of = [&](const Step& s, u32 (&mine)[2]) {
#pragma unroll
        for (u32 k = 0; k < 2; ++k)
            if (warp + kChainWarps * k < s.nr) mine[k] = load(v.routes.slots + s.first + warp + kChainWarps * k);
    };
    auto stage = [&](u32 b, const Step& s, const u32 (&mine)[2]) {
#pragma unroll
        for (u32 k = 0; k < 2; ++k) {
            const u32 r = warp + kChainWarps * k;
            if (r >= s.nr) break;
            if (lane == 0) s_slots[b][r] = mine[k];
            unsigned char* to = a8 + b * a8_bytes + r * kCell;
            const i8* c = v.act.codes + u64(mine[k]) * stride;
            for (u32 i = lane; i < 2u * groups; i += 32) cp_async16(to + (i >> 1) * (kCap * kCell) + 16u * (i & 1u), c + 16u * i);
            const float* deltas = v.act.deltas + u64(mine[k]) * (stride / 32);
            const i32* sums = v.act.sums + u64(mine[k]) * (stride / 32);
            for (u32 i = lane; i < groups; i += 32) {
                cp_async4(to + i * (kCap * kCell) + kCellDelta, deltas + i);
                if (Q51) cp_async4(to + i * (kCap * kCell) + kCellSum, sums + i);
            }
        }
    };
    const u32 chain = warp & 3u, rt = (warp >> 2) % RT, eg = (warp >> 2) / RT, g = lane >> 2, t = lane & 3u;
    const u32 my_row = 16u * rt + g, at_row = my_row * row_bytes + my_row / plan.copy_rows * plan.row_gap;
    const u32 eight_on = 8u * row_bytes + ((my_row + 8u) / plan.copy_rows - my_row / plan.copy_rows) * plan.row_gap;
    Step cur = item_begin(first_item), next = after(cur);
    u32 slots[2] = {0, 0};
    slots_of(cur, slots);
    stage(0, cur, slots);
    slots_of(next, slots);
    bool ok = true, begins = true;
    u32 n = 0, b = 0;  // the CTA's item, the step's buffer
    while (cur.item.id < n_items) {
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();  // the step's rows are there, the other buffer and the meeting place have been read
        stage(b ^ 1u, next, slots);
        const Step then = after(next);
        slots_of(then, slots);
        if (begins) {
            ok = mbar_wait(&full[n & 1u], (n >> 1) & 1u, plan.wait_limit, &s_abort);
            if (__syncthreads_or(!ok)) { ok = false; break; }
        }
        const u32 rows = saddr(smem) + (n & 1u) * plan.stage_bytes + at_row + chain * block;
        const u32 cells = saddr(a8) + b * a8_bytes + (chain * kCap + 8u * eg) * kCell, codes = cells + g * kCell + 4u * t, es = cells + 2u * t * kCell;
        const u32 tiles = cur.nr > 8u * eg ? (cur.nr - 8u * eg + 8u * EG - 1u) / (8u * EG) : 0u;  // of this warp
        float2 acc[NT][2];
#pragma unroll
        for (u32 e = 0; e < NT; ++e) acc[e][0] = acc[e][1] = make_float2(0.0f, 0.0f);
        auto run = [&](auto some, auto unroll) {  // blocks at a time: a block's chain of reads, MMA and sums is some 200 clocks long
            constexpr u32 T = decltype(some)::value, U = decltype(unroll)::value;
            ChainRow<Q51> r0(rows, t), r1(rows + eight_on, t);
            u32 at_codes = codes, at_es = es;
#pragma unroll U
            for (u32 gi = chain; gi < groups; gi += 4) {
                u32 a[4];
                float d0, d1, m0, m1;
                r0.read(a[0], a[2], d0, m0);
                r1.read(a[1], a[3], d1, m1);
#pragma unroll
                for (u32 e = 0; e < T; ++e) {
                    if (T > 2 && e >= tiles) break;
                    constexpr u32 tile = 8u * EG * kCell;
                    int dot[4];
                    mma_s8(dot, a, lds32(at_codes + e * tile), lds32(at_codes + e * tile + 16u));
                    const u32 x = at_es + e * tile;
                    float2 x0 = mul2(both(d0), to_float(make_int2(dot[0], dot[1]))), x1 = mul2(both(d1), to_float(make_int2(dot[2], dot[3]))), E;
                    if (Q51) {
                        const uint2 p = lds64(x + kCellDelta), q = lds64(x + kCell + kCellDelta);
                        E = make_float2(__uint_as_float(p.x), __uint_as_float(q.x));
                        const float2 S = to_float(make_int2(static_cast<int>(p.y), static_cast<int>(q.y)));
                        x0 = add2(x0, mul2(both(m0), S));
                        x1 = add2(x1, mul2(both(m1), S));
                    } else {
                        E = make_float2(__uint_as_float(lds32(x + kCellDelta)), __uint_as_float(lds32(x + kCell + kCellDelta)));
                    }
                    acc[e][0] = add2(acc[e][0], mul2(E, x0));
                    acc[e][1] = add2(acc[e][1], mul2(E, x1));
                }
                r0.next(); r1.next();
                at_codes += 4u * kCap * kCell; at_es += 4u * kCap * kCell;
            }
        };
        using std::integral_constant;
        if (tiles == 1u) run(integral_constant<u32, 1>{}, integral_constant<u32, 2>{});
        else if (NT > 1 && tiles == 2u) run(integral_constant<u32, (NT > 1 ? 2 : 1)>{}, integral_constant<u32, 2>{});
        else if (NT > 2 && tiles) run(integral_constant<u32, NT>{}, integral_constant<u32, 1>{});
#pragma unroll
        for (u32 e = 0; e < NT; ++e) {
            if (e >= tiles) break;
            float* to = s_meet + (chain * kCap + 8u * (eg + EG * e) + 2u * t) * kMeet + 16u * rt + g;
            to[0] = acc[e][0].x; to[kMeet] = acc[e][0].y;
            to[8] = acc[e][1].x; to[kMeet + 8] = acc[e][1].y;
        }
        __syncthreads();
        for (u32 r = warp; r < cur.nr; r += kChainWarps)
#pragma unroll
            for (u32 o = lane; o < R; o += 32) {
                const float* c = s_meet + r * kMeet + o;
                const u32 p = kCap * kMeet;
                v.raw[u64(s_slots[b][r]) * H + R * cur.item.chunk + o] = __fadd_rn(__fadd_rn(c[0], c[p]), __fadd_rn(c[2 * p], c[3 * p]));
            }
        begins = cur.last;
        if (cur.last) {
            if (to_ask.id < n_ask) {  // the stage has been read
                if (lane == 0) {
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    ask(n + 2, to_ask);
                }
                ++asked;
                onward(to_ask);
            }
            ++n;
        }
        cur = next; next = then; b ^= 1u;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    if (!ok && tid == 0) {
        drain_asked(n);
        if (v.summary) atomicOr(const_cast<u32*>(v.summary), kAbortBit);
    }
}

// Rows of an item and entries of a step: 64 x 32, 64 x 16 (a step's rows come out of L2 once an item), 32 x 32 (Q8_0; a group of Q5_1 takes in it what it takes in 64 x 16) or
// 32 x 16, as shared memory allows; false where rows are too long for that. H is whole blocks of a K-quant gate/up, a multiple of 256.
bool chain_mma_plan(const b200moe_down_view& v, ChainMmaPlan* p, u32* smem) {
    const u32 H = v.shape.hidden, groups = v.shape.inter / 32, row_bytes = groups * (v.shape.down_type == B200MOE_TYPE_Q5_1 ? kQ51Block : kQ8Block);
    const u32 limit = debug_value(B200MOE_DEBUG_WAIT_LIMIT), stall = debug_value(B200MOE_DEBUG_STALL_STAGE);
    p->wait_limit = limit ? limit : 1u << 18;  // about a second
    p->stall_stage = stall ? stall - 1u : 0xffffffffu;
    p->max_union = v.max_union;
    // Eight rows' word reads meet every bank once if the rows lie an odd multiple of 4 (mod 32) words apart, about so at other odd distances. Rows whose length is a multiple of
    // 8 words come by copies of as many as fall on different banks, 16 bytes left free between the copies (60 experts of 2560, 1536 wide, Q5_1, 960 rows of top 4: 641 -> 410 us).
    const u32 words = row_bytes % 32 ? 1u : row_bytes / 4u % 32u;
    p->copy_rows = words == 0 ? 1u : words == 16 ? 2u : words % 8 == 0 ? 4u : 16u;
    p->row_gap = p->copy_rows == 16u ? 0u : 16u;
    constexpr u32 forms[4][2] = {{64, 32}, {64, 16}, {32, 32}, {32, 16}};
    for (u32 i = 0; i < 4; ++i) {
        const u32 R = forms[i][0], cap = forms[i][1];
        p->form = i;
        p->n_chunks = H / R;
        p->stage_bytes = (R * row_bytes + R / p->copy_rows * p->row_gap + 127u) / 128u * 128u;
        const u64 total = 2 * u64(p->stage_bytes) + 2 * u64(groups) * cap * kCell + 4 * u64(cap) * (R + 4) * 4 + (2 * u64(v.max_union) + 1) * 4;
        if (total > 226u * 1024u || (i == 2 && v.shape.down_type == B200MOE_TYPE_Q5_1)) continue;
        *smem = static_cast<u32>(total);
        return u64(p->n_chunks) * v.max_union < (1u << 30);
    }
    return false;
}

}  // namespace

u32 chain4_mma_chunks(const b200moe_down_view& v) {
    ChainMmaPlan p{};
    u32 smem;
    const bool q51 = v.shape.down_type == B200MOE_TYPE_Q5_1;
    const bool fits = (q51 || v.shape.down_type == B200MOE_TYPE_Q8_0) && (!q51 || v.act.sums) && aligned(v.weights.down, 16) && chain_mma_plan(v, &p, &smem);
    return fits ? p.n_chunks : 0u;
}

int launch_down_chain4_mma(const b200moe_down_view& v, const ChainHints& hints, cudaStream_t stream) {
    if (v.max_union == 0) return B200MOE_OK;
    ChainMmaPlan p{};
    u32 smem = 0;
    if (!chain_mma_plan(v, &p, &smem)) return fail(B200MOE_ERR_UNSUPPORTED, "down: the tensor-core four-chain form does not apply to this shape");
    p.early = hints.routes_done;
    const bool q51 = v.shape.down_type == B200MOE_TYPE_Q5_1;
    const auto kernel = p.form == 0 ? (q51 ? down_chain4_mma_kernel<true, 4, 1, 4> : down_chain4_mma_kernel<false, 4, 1, 4>)
                      : p.form == 1 ? (q51 ? down_chain4_mma_kernel<true, 4, 1, 2> : down_chain4_mma_kernel<false, 4, 1, 2>)
                      : p.form == 2 ? down_chain4_mma_kernel<false, 2, 2, 2>
                                    : (q51 ? down_chain4_mma_kernel<true, 2, 2, 1> : down_chain4_mma_kernel<false, 2, 2, 1>);
    const u32 grid = static_cast<u32>(std::min<u64>(static_cast<u32>(device_sm_count()), u64(p.n_chunks) * v.max_union));
    if (int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), smem)) return rc;
    chain_launch(kernel, grid, kChainThreads, smem, stream, v, p);
    return after_launch("down_chain4_mma");
}

}  // namespace b200moe
