// Window routes: the expert-major CSR of (row, slot) entries that every expert kernel gathers through. Activations
// are never permuted in memory.
//
// Contract: strix::ds41::build_window_routes + restrict_routes (src/ds41_moe.cpp:11-61; device mirror
// include/strix/cuda/ds41_moe.hpp:41-72): union experts ascending, the entries of an expert in ascending row,
// slots[i] = row * top_k + k, order[row][*] = the row's slots in ascending expert id, low_counts[row] = ids < split.
// All integer work; results are exact and independent of the launch shape.
//
// Two forms: up to 1024 slots (decode windows) one block does everything; above that three launches over chunks of
// 1024 slots (per-chunk histograms, a scan over chunks and experts, then the stable fill).
#include <algorithm>

#include "kernels.cuh"
#include "router_select.cuh"
#include "routes_small.cuh"

namespace b200moe {
namespace {

constexpr u32 kChunk = routes_detail::kChunk;
constexpr u32 kFusedExperts = 256;  // of the launch that selects too

using routes_detail::block_exclusive_scan;
using routes_detail::entry_id;
using routes_detail::kRankedTopK;
using routes_detail::row_order;
using routes_detail::routes_small_body;

using routes_detail::Clear;
using routes_detail::counts_bytes;

__global__ void __launch_bounds__(1024) routes_small_kernel(b200moe_routes_view v, u32 end, Clear clear) {
    extern __shared__ __align__(16) u16 counts[];
    chain_begin();
    routes_detail::clear_words(clear, v.rows);  // in front of the body's first barrier
    routes_small_body(v, end, v.ids, counts);
}

// Windows of a few slots.
__global__ void __launch_bounds__(32) routes_one_warp_kernel(b200moe_routes_view v, u32 end, Clear clear) {
    chain_begin();
    routes_detail::clear_words(clear, v.rows);
    __syncwarp();  // the rows' status is cleared before it is set
    routes_detail::routes_one_warp(v, end, v.ids);
}

// Decode windows: the router's selection (one warp per row) and the routes of the selected ids in ONE block, so the
// layer prologue costs one launch less. Up to 256 experts (their keys fit the 64 registers that a block of 1024 threads has) and 8 rows in the form of 256 threads.
// What bounds it: a chain of latencies on cold instruction caches. A row's slots are ordered, checked and counted by its own warp, out of registers; the rows
// of an expert are bits of one word (32 rows at most), so that an entry's place among its expert's is a count of bits and the rest one scan over the experts. With the
// general build behind the selection (routes_small_body), and the selection's other paths between its steps, the kernel took 19,400 clocks behind its wait with 8 rows x 8 over 128
// experts and 12,000 with 1 row, 10,100 and 4,450 of them the routes'; 9,800 and 9,500 now, 2,300 both. A call 49.6 -> 45.3 and 22.8 -> 21.4 us.
template <u32 THREADS, int EPL>
__global__ void __launch_bounds__(THREADS) select_routes_small_kernel(const float* logits, float* scores_out, const float* bias,
                                                                      const __grid_constant__ b200moe_route_policy p, u32 rows, u32* ids, float* weights,
                                                                      b200moe_routes_view rv, u32 end, Clear clear) {
    extern __shared__ __align__(16) float sel_smem[];
    __shared__ u32 s_rows[kFusedExperts], s_begin[kFusedExperts], s_total[32], s_most[32];
    const u32 t = threadIdx.x, lane = t & 31u, warp = t >> 5, E = rv.experts, K = rv.top_k;
    for (u32 i = t; i < kFusedExperts; i += blockDim.x) s_rows[i] = 0u;
    chain_begin();
    routes_detail::clear_words(clear, rows);
    __syncthreads();  // the rows' status is cleared before it is set
    u32 e = 0xffffffffu;  // the expert that the lane's slot is an entry of
    if (warp < rows) {
        const u32 id = select_detail::select_row<EPL>(logits, scores_out, bias, p, warp, lane, sel_smem + warp * select_detail::scratch_floats(p.experts), ids, weights);
        u32 pos = 0;  // the slot's place in ascending expert id
        bool bad = id >= E, repeats = false;
#pragma unroll 1
        for (u32 k0 = 0; k0 < K; k0 += 8) {
            u32 o[8];
#pragma unroll
            for (u32 i = 0; i < 8; ++i) o[i] = __shfl_sync(0xffffffffu, id, k0 + i);
#pragma unroll
            for (u32 i = 0; i < 8; ++i) {
                const u32 k = k0 + i;
                const bool slot = k < K, same = slot && o[i] == id && k != lane, before = k < lane;
                pos += (slot && o[i] < id) || (same && before) ? 1u : 0u;
                bad |= same;
                repeats |= same && before;
            }
        }
        const u32 low = __popc(__ballot_sync(0xffffffffu, lane < K && id < rv.split));
        if (lane < K) {
            rv.out.order[warp * K + pos] = warp * K + lane;
            if (lane == 0) rv.out.low_counts[warp] = low;
            if (bad && rv.row_status) atomicOr(&rv.row_status[warp], B200MOE_ROW_INVALID_ROUTE);
            if (!repeats && routes_detail::owned(id, E, rv.first, end)) {
                e = id;
                atomicOr(&s_rows[e], 1u << warp);
            }
        }
    }
    __syncthreads();
    const u32 own = t < E ? s_rows[t] : 0u, c = __popc(own), sum = c + (c ? 0x10000u : 0u);  // entries, and experts that have some in the upper half
    u32 upto = sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) { const u32 o = __shfl_up_sync(0xffffffffu, upto, d); if (lane >= (u32)d) upto += o; }
    const u32 most = __reduce_max_sync(0xffffffffu, c);
    if (lane == 31u) { s_total[warp] = upto; s_most[warp] = most; }
    __syncthreads();
    const u32 others = lane < blockDim.x / 32u ? s_total[lane] : 0u, total = __reduce_add_sync(0xffffffffu, others);
    const u32 at = __reduce_add_sync(0xffffffffu, lane < warp ? others : 0u) + upto - sum, begin = at & 0xffffu, uidx = at >> 16;
    if (t < E) {
        s_begin[t] = begin;
        if (c) { rv.out.experts[uidx] = t - rv.base; rv.out.begins[uidx + 1] = begin + c; }
    }
    if (warp == 0) {
        const u32 maxc = __reduce_max_sync(0xffffffffu, lane < blockDim.x / 32u ? s_most[lane] : 0u);
        if (lane == 0) {
            rv.out.begins[0] = 0;
            rv.out.counts[0] = total >> 16; rv.out.counts[1] = maxc; rv.out.counts[2] = total & 0xffffu; rv.out.counts[3] = 0;
        }
    }
    __syncthreads();
    if (e != 0xffffffffu) {
        const u32 to = s_begin[e] + __popc(s_rows[e] & ((1u << warp) - 1u));
        rv.out.rows[to] = warp;
        rv.out.slots[to] = warp * K + lane;
    }
}

// ---- chunked form --------------------------------------------------------------------------------------------------
// scratch: hist[chunks][experts], then ebegin[experts].
template <bool RANKED>
__global__ void __launch_bounds__(1024) routes_count_kernel(b200moe_routes_view v, u32 end, u32 chunks, Clear clear) {
    chain_begin();
    __shared__ u32 cnt[1024];
    const u32 t = threadIdx.x, n = v.rows * v.top_k, s = blockIdx.x * kChunk + t;
    cnt[t] = 0;
    __syncthreads();
    if (s < n) { const u32 e = entry_id(v.ids, s, v.top_k, v.experts, v.first, end); if (e != 0xffffffffu) atomicAdd(&cnt[e], 1u); }
    __syncthreads();
    if (t < v.experts) v.scratch[u64(blockIdx.x) * v.experts + t] = cnt[t];
    if (blockIdx.x == 0) {
        if (clear.summary4 && t < 4) clear.summary4[t] = 0u;
        if (clear.summary && t == 0) *clear.summary = 0u;
    }
    // Rows that are ranked in registers go to neighbouring threads; those that are sorted, in arrays of local memory, to the blocks in turn, so that a
    // multiprocessor's L1 holds the arrays of its few (129 rows x 32: 63 us with all of them in one block, 246 when the carve-out
    // left that block 28 KB of L1, 51 here).
    for (u32 r = RANKED ? blockIdx.x * blockDim.x + t : t * gridDim.x + blockIdx.x; r < v.rows; r += gridDim.x * blockDim.x) {
        if (clear.row_status) clear.row_status[r] = 0u;  // the row's status is this thread's alone in this launch
        row_order<RANKED>(v.ids, r, v.top_k, v.experts, v.split, v.out.order, v.out.low_counts, v.row_status);
    }
}
__global__ void __launch_bounds__(1024) routes_scan_kernel(b200moe_routes_view v, u32 chunks) {
    chain_begin();
    __shared__ u32 warp_tot[32], total_s, union_s, maxc;
    const u32 t = threadIdx.x;
    if (t == 0) maxc = 0;
    u32 c = 0;
    if (t < v.experts)
        for (u32 k0 = 0; k0 < chunks; k0 += 8) {  // eight chunks' counts asked for at once
            u32 x[8];
#pragma unroll
            for (u32 k = 0; k < 8; ++k) x[k] = k0 + k < chunks ? v.scratch[u64(k0 + k) * v.experts + t] : 0u;
#pragma unroll
            for (u32 k = 0; k < 8; ++k) {
                if (k0 + k < chunks) v.scratch[u64(k0 + k) * v.experts + t] = c;
                c += x[k];
            }
        }
    __syncthreads();
    const u32 begin = block_exclusive_scan(c, warp_tot, &total_s);
    const u32 uidx = block_exclusive_scan(c ? 1u : 0u, warp_tot, &union_s);
    if (t < v.experts) v.scratch[u64(chunks) * v.experts + t] = begin;
    if (c) { v.out.experts[uidx] = t - v.base; v.out.begins[uidx + 1] = begin + c; atomicMax(&maxc, c); }
    __syncthreads();
    if (t == 0) {
        v.out.begins[0] = 0;
        v.out.counts[0] = union_s; v.out.counts[1] = maxc; v.out.counts[2] = total_s; v.out.counts[3] = 0;
    }
}
__global__ void __launch_bounds__(1024) routes_fill_kernel(b200moe_routes_view v, u32 end, u32 chunks) {
    extern __shared__ __align__(16) u16 counts[];  // [32][experts]
    const u32 t = threadIdx.x, n = v.rows * v.top_k, s = blockIdx.x * kChunk + t;
    routes_detail::clear_counts(counts, 32, v.experts);
    chain_begin();
    u32 e = 0xffffffffu;
    if (s < n) e = entry_id(v.ids, s, v.top_k, v.experts, v.first, end);
    const u32 base = e == 0xffffffffu ? 0u : v.scratch[u64(chunks) * v.experts + e] + v.scratch[u64(blockIdx.x) * v.experts + e];
    __syncthreads();
    const u32 peers = routes_detail::count_run(counts, t / 32u, v.experts, e);
    __syncthreads();
    if (t < v.experts) routes_detail::sum_runs(counts, 32, v.experts, t);
    __syncthreads();
    if (e == 0xffffffffu) return;
    const u32 pos = base + routes_detail::rank_of(counts, t / 32u, v.experts, e, peers);
    v.out.rows[pos] = s / v.top_k;
    v.out.slots[pos] = s;
}


// The routes of a dense block (one expert, top-1: every row is one entry of expert 0, slot = row) written directly, with
// the job's status words cleared in the same launch: what build_window_routes (src/ds41_moe.cpp:11-43) gives for ids = 0,
// without the sort and without the memsets in front of it.
__global__ void __launch_bounds__(256) dense_routes_kernel(b200moe_routes out, u32 rows, u32* row_status, u32* summary4, float* zero, u64 count) {
    chain_begin();
    const u32 i = blockIdx.x * blockDim.x + threadIdx.x, threads = gridDim.x * blockDim.x;
    if (zero) {
        const u64 whole = reinterpret_cast<uintptr_t>(zero) % 16 == 0 ? count / 4 : 0;
        for (u64 k = i; k < whole; k += threads) reinterpret_cast<float4*>(zero)[k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        for (u64 k = 4 * whole + i; k < count; k += threads) zero[k] = 0.0f;
    }
    if (i < rows) {
        out.rows[i] = i;
        out.slots[i] = i;
        if (out.order) out.order[i] = i;
        if (out.low_counts) out.low_counts[i] = 1u;  // id 0 < split 1
        if (row_status) row_status[i] = 0u;
    }
    if (i == 0) {
        out.experts[0] = 0u;
        out.begins[0] = 0u;
        out.begins[1] = rows;
        out.counts[0] = 1u; out.counts[1] = rows; out.counts[2] = rows; out.counts[3] = 0u;
        if (summary4) { summary4[0] = 0u; summary4[1] = 0u; summary4[2] = 0u; summary4[3] = 0u; }
    }
}

}  // namespace

u64 routes_scratch_words(u32 rows, u32 top_k, u32 experts) {
    const u64 n = u64(rows) * top_k, chunks = (n + kChunk - 1) / kChunk;
    return (chunks + 1) * experts + 4;
}

u32 small_threads(u32 slots, u32 experts) { return std::min(1024u, std::max(256u, (std::max(slots, experts) + 31u) / 32u * 32u)); }

bool select_routes_fusable(const b200moe_router_view& r, u32 top_k) {
    return r.rows <= 32 && u64(r.rows) * top_k <= kChunk && r.policy.experts <= kFusedExperts && u64(r.rows) * select_detail::scratch_floats(r.policy.experts) * 4u <= 96u * 1024u;
}
int launch_select_routes(const b200moe_router_view& r, const b200moe_routes_view& v, const RoutesClear& clear, cudaStream_t stream) {
    if (r.rows == 0) return B200MOE_OK;
    const u32 smem = r.rows * select_detail::scratch_floats(r.policy.experts) * 4u, threads = std::max(32u * r.rows, 256u);  // a thread an expert
    const bool few = r.policy.experts <= 128u;
    const auto kernel = threads <= 256u ? (few ? select_routes_small_kernel<256, 4> : select_routes_small_kernel<256, 8>) : few ? select_routes_small_kernel<1024, 4> : select_routes_small_kernel<1024, 8>;
    if (int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), smem)) return rc;
    small_launch(kernel, 1, threads, smem, stream, r.logits, r.scores, r.bias, r.policy, r.rows, r.ids, r.weights, v, v.end ? v.end : v.experts,
                 Clear{clear.row_status, clear.summary4, clear.summary});
    return after_launch("select_routes_small");
}

int launch_dense_routes(const b200moe_routes& out, u32 rows, u32* row_status, u32* summary4, float* zero, u64 count, cudaStream_t stream) {
    const u64 most = std::max<u64>(rows, zero ? std::min<u64>((count + 3) / 4, 256ull * 8ull * static_cast<u32>(device_sm_count())) : 0);
    small_launch(dense_routes_kernel, static_cast<u32>((most + 255) / 256), 256, 0, stream, out, rows, row_status, summary4, zero, count);
    return after_launch("dense_routes");
}

int launch_routes(const b200moe_routes_view& v, const RoutesClear& clear, cudaStream_t stream) {
    const u64 n = u64(v.rows) * v.top_k;
    if (n == 0) return B200MOE_OK;
    const u32 end = v.end ? v.end : v.experts;
    const Clear c{clear.row_status, clear.summary4, clear.summary};
    const u32 smem = counts_bytes(static_cast<u32>(std::min<u64>(n, kChunk)), v.experts);
    if (n <= routes_detail::kWarpSlots) {
        small_launch(routes_one_warp_kernel, 1, 32, 0, stream, v, end, c);
        return after_launch("routes_small");
    }
    if (n <= kChunk) {
        if (int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(routes_small_kernel), smem)) return rc;
        small_launch(routes_small_kernel, 1, small_threads(static_cast<u32>(n), v.experts), smem, stream, v, end, c);
        return after_launch("routes_small");
    }
    const u32 chunks = static_cast<u32>((n + kChunk - 1) / kChunk);
    if (int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(routes_fill_kernel), smem)) return rc;
    small_launch((v.top_k <= kRankedTopK ? routes_count_kernel<true> : routes_count_kernel<false>), chunks, 1024, 0, stream, v, end, chunks, c);
    if (int rc = after_launch("routes_count")) return rc;
    small_launch(routes_scan_kernel, 1, 1024, 0, stream, v, chunks);
    if (int rc = after_launch("routes_scan")) return rc;
    small_launch(routes_fill_kernel, chunks, 1024, smem, stream, v, end, chunks);
    return after_launch("routes_fill");
}

}  // namespace b200moe
