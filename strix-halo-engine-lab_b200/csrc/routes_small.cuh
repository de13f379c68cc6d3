// Routes of a decode window (up to 1024 slots, up to 1024 experts) built by ONE block of any size, or by one warp: device code of
// the stand-alone routes kernels (routes.cu); the launch that selects too has a build of its own.
// Contract: strix::ds41::build_window_routes + restrict_routes (src/ds41_moe.cpp:11-61), see routes.cu.
#pragma once
#include "common.cuh"

namespace b200moe {
namespace routes_detail {

constexpr u32 kChunk = 1024;
constexpr u32 kRankedTopK = 8;  // row_order: up to so many slots of a row are ranked in registers

// Exclusive scan of one value per thread over the block (blockDim a multiple of 32, at most 1024); `total` gets the
// sum. warp_tot: 32 words of shared memory.
__device__ __forceinline__ u32 block_exclusive_scan(u32 v, u32* warp_tot, u32* total) {
    const u32 lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    u32 inc = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) { const u32 o = __shfl_up_sync(0xffffffffu, inc, d); if (lane >= (u32)d) inc += o; }
    if (lane == 31) warp_tot[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        u32 t = lane < nwarps ? warp_tot[lane] : 0u, ti = t;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) { const u32 o = __shfl_up_sync(0xffffffffu, ti, d); if (lane >= (u32)d) ti += o; }
        warp_tot[lane] = ti - t;
        if (lane == 31) *total = ti;
    }
    __syncthreads();
    const u32 r = warp_tot[warp] + inc - v;
    __syncthreads();
    return r;
}

// Per row: the slots sorted by expert id (stable), the low count and the route check. One thread a row, in the middle of a call's chain
// of launches. Up to kRankedTopK slots are ranked in registers, all ids requested at once; more go through the insertion sort, whose
// arrays live in local memory. The routes of 64 rows x 8 over 256 experts take 9.5 us ranked, 11.7 sorted, those of 1024 x 8 over 128
// 24.4 and 30.2. RANKED: any top_k, by a test; a kernel for more slots holds the sort alone (100 rows x 10: 21.4 us, 21.7 with the
// test), while ranking alone gained nothing (32 rows x 8: 9.4 us, 9.2 with the test).
template <bool RANKED>
__device__ inline void row_order(const u32* ids, u32 row, u32 top_k, u32 experts, u32 split, u32* order, u32* low_counts, u32* row_status) {
    if (RANKED && top_k <= kRankedTopK) {
        u32 id[kRankedTopK], low = 0;
        bool bad = false;
#pragma unroll
        for (u32 k = 0; k < kRankedTopK; ++k) id[k] = k < top_k ? ids[row * top_k + k] : 0xffffffffu;
#pragma unroll
        for (u32 k = 0; k < kRankedTopK; ++k)
            if (k < top_k) {
                u32 rank = 0;
#pragma unroll
                for (u32 j = 0; j < kRankedTopK; ++j)
                    if (j != k && j < top_k) {
                        rank += (id[j] < id[k] || (id[j] == id[k] && j < k)) ? 1u : 0u;
                        bad |= id[j] == id[k];
                    }
                bad |= id[k] >= experts;
                low += id[k] < split ? 1u : 0u;
                order[row * top_k + rank] = row * top_k + k;
            }
        low_counts[row] = low;
        if (bad && row_status) atomicOr(&row_status[row], B200MOE_ROW_INVALID_ROUTE);
        return;
    }
    u32 key[32], slot[32];
    u32 low = 0;
    bool bad = false;
    for (u32 k = 0; k < top_k; ++k) {
        const u32 s = row * top_k + k, e = ids[s];
        bad |= e >= experts;
        low += e < split ? 1u : 0u;
        u32 j = k;
        while (j > 0 && key[j - 1] > e) { key[j] = key[j - 1]; slot[j] = slot[j - 1]; --j; }
        bad |= (j > 0 && key[j - 1] == e);
        key[j] = e; slot[j] = s;
    }
    for (u32 k = 0; k < top_k; ++k) order[row * top_k + k] = slot[k];
    low_counts[row] = low;
    if (bad && row_status) atomicOr(&row_status[row], B200MOE_ROW_INVALID_ROUTE);
}

__device__ __forceinline__ bool owned(u32 e, u32 experts, u32 first, u32 end) { return e < experts && e >= first && e < end; }
// The expert id slot s contributes an entry for, or 0xffffffff for none: the id must lie in the owned range and must not
// repeat an earlier slot of the same row. (The host builder throws on a repeated id, src/ds41_moe.cpp:22-23; here the row
// is flagged INVALID_ROUTE and only the first occurrence keeps its entry, so no expert ever has more entries than the
// window has rows and a flagged row cannot disturb the entries of a valid one.)
__device__ __forceinline__ u32 entry_id(const u32* ids, u32 s, u32 top_k, u32 experts, u32 first, u32 end) {
    const u32 e = ids[s];
    if (!owned(e, experts, first, end)) return 0xffffffffu;
    bool repeats = false;
    for (u32 i = s - s % top_k; i < s; ++i) repeats |= ids[i] == e;  // no early way out: the loads overlap
    return repeats ? 0xffffffffu : e;
}

// What the first launch of a call that owns its status words clears on the way (all optional).
struct Clear {
    u32* row_status;  // rows words
    u32* summary4;    // 4 words
    u32* summary;     // 1 word
};
__device__ __forceinline__ void clear_words(const Clear& c, u32 rows) {
    if (c.row_status) for (u32 r = threadIdx.x; r < rows; r += blockDim.x) c.row_status[r] = 0u;
    if (c.summary4 && threadIdx.x < 4) c.summary4[threadIdx.x] = 0u;
    if (c.summary && threadIdx.x == 0) *c.summary = 0u;
}

// The rank of a slot among the slots of its expert: within the slot's warp by a match, over the warps before by counts that each run of 32 slots
// leaves in shared memory, [runs][experts] 16-bit words. A thread's own walk over the slots before took 14 us for 1024 slots, 6 for 64.
__device__ __forceinline__ void clear_counts(u16* counts, u32 runs, u32 experts) {
    for (u32 i = threadIdx.x; i < (runs * experts + 1u) / 2u; i += blockDim.x) reinterpret_cast<u32*>(counts)[i] = 0u;
}
__device__ __forceinline__ u32 count_run(u16* counts, u32 run, u32 experts, u32 e) {  // a whole warp; e: 0xffffffff for none. The lanes with the same expert
    const u32 peers = __match_any_sync(0xffffffffu, e);
    if (e != 0xffffffffu && (threadIdx.x & 31u) == __ffs(peers) - 1u) counts[run * experts + e] = static_cast<u16>(__popc(peers));
    return peers;
}
__device__ __forceinline__ u32 sum_runs(u16* counts, u32 runs, u32 experts, u32 e) {  // exclusive sums in place; the total
    u32 n = 0;
#pragma unroll 4
    for (u32 w = 0; w < runs; ++w) { const u32 c = counts[w * experts + e]; counts[w * experts + e] = static_cast<u16>(n); n += c; }
    return n;
}
__device__ __forceinline__ u32 rank_of(const u16* counts, u32 run, u32 experts, u32 e, u32 peers) {
    return counts[run * experts + e] + __popc(peers & ((1u << (threadIdx.x & 31u)) - 1u));
}
__host__ __device__ constexpr u32 counts_bytes(u32 slots, u32 experts) { return (((slots + 31u) / 32u * experts * 2u) + 15u) / 16u * 16u; }

// The build of a window of a few slots (kWarpSlots, 32 at most) by one warp: a slot a lane, every count from the other lanes' ids. No scan over the experts and no barrier, which
// cost the form below more than the walk over the other slots costs here: over 64 and 1024 experts 1 slot 2.5 and 3.2 us a launch, here
// 1.7 and 1.6, 8 slots 2.8 and 3.3, 2.2 both, 16 slots 2.7 and 3.4, 2.8 both, 32 slots 2.9 and 3.6, 3.8 both.
constexpr u32 kWarpSlots = 16;
__device__ __forceinline__ void routes_one_warp(const b200moe_routes_view& v, u32 end, const u32* ids) {
    const u32 s = threadIdx.x, n = v.rows * v.top_k, K = v.top_k, row = s / K, first = row * K;
    const u32 id = s < n ? ids[s] : 0xffffffffu;
    u32 pos = 0, low = 0;
    bool bad = id >= v.experts, repeats = false;
    for (u32 i = 0; i < n; ++i) {
        const u32 o = __shfl_sync(0xffffffffu, id, i);
        const bool mine = i - first < K, same = mine && o == id && i != s;
        pos += mine && (o < id || (same && i < s)) ? 1u : 0u;
        low += mine && o < v.split ? 1u : 0u;
        bad |= same;
        repeats |= same && i < s;
    }
    const u32 e = s < n && !repeats && owned(id, v.experts, v.first, end) ? id : 0xffffffffu;
    const u32 peers = __match_any_sync(0xffffffffu, e), rank = __popc(peers & ((1u << s) - 1u));
    const bool entry = e != 0xffffffffu, head = entry && rank == 0;
    const u32 heads = __ballot_sync(0xffffffffu, head), entries = __ballot_sync(0xffffffffu, entry), most = __reduce_max_sync(0xffffffffu, entry ? __popc(peers) : 0u);
    u32 before = 0, uidx = 0;  // entries of the experts below, and how many these are
    for (u32 i = 0; i < n; ++i) {
        const bool below = __shfl_sync(0xffffffffu, e, i) < e;  // no entry is above every expert
        before += below ? 1u : 0u;
        uidx += below && (heads >> i & 1u) ? 1u : 0u;
    }
    if (s < n) {
        v.out.order[first + pos] = s;
        if (s == first) v.out.low_counts[row] = low;
        if (bad && v.row_status) atomicOr(&v.row_status[row], B200MOE_ROW_INVALID_ROUTE);
    }
    if (entry) {
        v.out.rows[before + rank] = row;
        v.out.slots[before + rank] = s;
        if (head) { v.out.experts[uidx] = e - v.base; v.out.begins[uidx + 1] = before + __popc(peers); }
    }
    if (s == 0) {
        v.out.begins[0] = 0;
        v.out.counts[0] = __popc(heads); v.out.counts[1] = most; v.out.counts[2] = __popc(entries); v.out.counts[3] = 0;
    }
}

// The whole build of a window of up to kChunk slots by one block. ids: the slots' experts; counts: counts_bytes(slots, experts) of shared memory. A slot's place in its row, the row's low count and check come from the row's ids in
// shared memory, its place among its expert's entries from the ranks above and one scan over the experts: five block barriers.
__device__ inline void routes_small_body(const b200moe_routes_view& v, u32 end, const u32* ids, u16* counts) {
    __shared__ u32 sid[kChunk], ent[kChunk], ebegin[1024], warp_tot[32], total_s, maxc;
    const u32 t = threadIdx.x, nt = blockDim.x, lane = t & 31u, n = v.rows * v.top_k, K = v.top_k, E = v.experts, runs = (n + 31u) / 32u;
    clear_counts(counts, runs, E);
    for (u32 s = t; s < n; s += nt) sid[s] = ids[s];
    if (t == 0) maxc = 0;
    __syncthreads();
    for (u32 s = t; s - lane < n; s += nt) {
        u32 e = 0xffffffffu;
        if (s < n) {
            const u32 row = s / K, first = row * K, id = sid[s];
            u32 pos = 0, low = 0;
            bool bad = id >= E, repeats = false;  // an earlier slot of the row has the id: no entry (entry_id)
            for (u32 i = first; i < first + K; ++i) {
                const u32 o = sid[i];
                const bool same = o == id && i != s, before = i < s;
                pos += (o < id || (same && before)) ? 1u : 0u;
                low += o < v.split ? 1u : 0u;
                bad |= same;
                repeats |= same && before;
            }
            v.out.order[first + pos] = s;
            if (s == first) v.out.low_counts[row] = low;
            if (bad && v.row_status) atomicOr(&v.row_status[row], B200MOE_ROW_INVALID_ROUTE);
            if (!repeats && owned(id, E, v.first, end)) e = id;
            ent[s] = e;
        }
        count_run(counts, s / 32u, E, e);
    }
    __syncthreads();
    const u32 per = (E + nt - 1) / nt, e0 = min(t * per, E), e1 = min(e0 + per, E);  // a thread's experts
    u32 sum = 0, most = 0;  // entries, and experts that have some in the upper half (up to 1024 each)
    for (u32 e = e0; e < e1; ++e) {
        const u32 c = sum_runs(counts, runs, E, e);
        ebegin[e] = c;
        sum += c + (c ? 0x10000u : 0u);
        most = max(most, c);
    }
    most = __reduce_max_sync(0xffffffffu, most);
    if (lane == 0 && most) atomicMax(&maxc, most);
    const u32 at = block_exclusive_scan(sum, warp_tot, &total_s);
    u32 begin = at & 0xffffu, uidx = at >> 16;
    for (u32 e = e0; e < e1; ++e) {
        const u32 c = ebegin[e];
        ebegin[e] = begin;
        if (c) { v.out.experts[uidx] = e - v.base; v.out.begins[uidx + 1] = begin + c; ++uidx; }
        begin += c;
    }
    __syncthreads();
    if (t == 0) {
        v.out.begins[0] = 0;
        v.out.counts[0] = total_s >> 16; v.out.counts[1] = maxc; v.out.counts[2] = total_s & 0xffffu; v.out.counts[3] = 0;
    }
    for (u32 s = t; s - lane < n; s += nt) {
        const u32 e = s < n ? ent[s] : 0xffffffffu, peers = __match_any_sync(0xffffffffu, e);
        if (e == 0xffffffffu) continue;
        const u32 pos = ebegin[e] + rank_of(counts, s / 32u, E, e, peers);
        v.out.rows[pos] = s / K;
        v.out.slots[pos] = s;
    }
}

}  // namespace routes_detail
}  // namespace b200moe
