// Weighted combine of the raw slot vectors, plus the small elementwise helpers of the layer.
//
// Forms (include/b200moe.h):
//   PARTS     y = ((shared + S_0) + S_1) + ...; S_p over the row's slots of expert range p in ascending expert id from
//             +0, one product then one add per step (src/ds41_moe.cpp:99-115, :152-163; device twin
//             include/strix/cuda/ds41_moe.hpp:109-134).
//   FMA_SLOTS acc = fma(w[k], raw[k], acc) in slot order (src/cuda/models/qwen/qwen_moe.cu:298-306;
//             include/strix/moe/combine.hpp:36-59), y = acc (+ shared), optional bfloat16 RNE commit (:330-335).
// HBM: rows * top_k * hidden * 4 B read, rows * hidden * 4 B written; elementwise over hidden, coalesced.
#include <algorithm>

#include "kernels.cuh"

namespace b200moe {
namespace {

constexpr u32 kMaxTopK = 32;

// skip_bits: with one of them in the job summary raw holds nothing of this job for some slots or for all, and no row is combined.
// grid (ceil(hidden / 256), min(rows, 65535)); 256 threads; a block walks rows blockIdx.y, blockIdx.y + gridDim.y, ...
__global__ void __launch_bounds__(256) combine_kernel(b200moe_combine_view v, u32 skip_bits, bool zero_skipped) {
    chain_begin();
    const u32 o = blockIdx.x * blockDim.x + threadIdx.x;
    const bool skipped = v.summary && (*v.summary & skip_bits);
    if (skipped && !zero_skipped) return;
    __shared__ float s_w[kMaxTopK];
    __shared__ u32 s_slot[kMaxTopK], s_part[kMaxTopK];
    for (u32 row = blockIdx.y; row < v.rows; row += gridDim.y) {
        __syncthreads();  // the previous row's readers are done with the shared arrays
        if (skipped || (v.row_status && v.row_status[row])) {  // fail closed (qwen_moe.cu:291); uniform over the block
            if (zero_skipped && !v.y_blocks && o < v.hidden) {
                for (u32 i = 0; i < max(v.only_part_count, 1u); ++i) v.y[i * v.part_stride + u64(row) * v.hidden + o] = 0.0f;  // every destination of the row
                if (v.y_bf16) v.y_bf16[u64(row) * v.hidden + o] = 0;
            }
            continue;
        }
        if (threadIdx.x < v.top_k) {
            const u32 k = threadIdx.x;
            if (v.form == B200MOE_COMBINE_PARTS) {
                const u32 slot = v.order[row * v.top_k + k];
                s_slot[k] = slot;
                s_w[k] = v.weights[slot];
                s_part[k] = v.low_counts ? (k < v.low_counts[row] ? 0u : 1u) : min(v.ids[slot] / v.part_experts, v.parts - 1);
            } else {
                s_slot[k] = row * v.top_k + k;
                s_w[k] = v.weights[row * v.top_k + k];
            }
        }
        __syncthreads();
        if (o >= v.hidden) continue;
        float out;
        if (v.form == B200MOE_COMBINE_FMA_SLOTS) {
            float acc = 0.0f;
            for (u32 k = 0; k < v.top_k; ++k) acc = __fmaf_rn(s_w[k], v.raw[u64(s_slot[k]) * v.hidden + o], acc);
            out = v.shared ? __fadd_rn(acc, v.shared[u64(row) * v.hidden + o]) : acc;
        } else {
            float total = v.shared ? v.shared[u64(row) * v.hidden + o] : 0.0f, single = 0.0f;
            const u32 first_part = v.only_part >= 0 ? static_cast<u32>(v.only_part) : 0u, n_parts = v.only_part_count > 1 ? v.only_part_count : 1u;
            u32 k = 0;
            for (u32 p = 0; p < v.parts; ++p) {  // the slots are sorted by expert id, so each part is one run
                float sum = 0.0f;
                while (k < v.top_k && s_part[k] == p) {
                    sum = __fadd_rn(sum, __fmul_rn(s_w[k], v.raw[u64(s_slot[k]) * v.hidden + o]));
                    ++k;
                }
                if (static_cast<int>(p) == v.only_part) single = sum;
                else if (v.only_part >= 0 && p > first_part && p < first_part + n_parts) {  // the further sums of a rank that owns several ranges
                    const u64 at = u64(p - first_part) * v.part_stride;
                    if (v.y_blocks) { const u32 blk = row / v.y_block_rows; v.y_blocks[blk][at + u64(row - blk * v.y_block_rows) * v.hidden + o] = sum; }
                    else v.y[at + u64(row) * v.hidden + o] = sum;
                }
                total = __fadd_rn(total, sum);
            }
            out = v.only_part >= 0 ? single : total;
        }
        if (v.y_blocks) {  // the row's home rank's buffer: a peer store
            const u32 blk = row / v.y_block_rows;
            v.y_blocks[blk][u64(row - blk * v.y_block_rows) * v.hidden + o] = out;
            continue;
        }
        v.y[u64(row) * v.hidden + o] = out;
        if (v.y_bf16) v.y_bf16[u64(row) * v.hidden + o] = bf16_rne_bits(out);
    }
}

// The PARTS form over whole rows with up to kVecTopK slots and 16-byte rows: four outputs a thread, every slot's values requested before the
// first is used and no block-wide step, so that a block's loads overlap. Bound by HBM (raw read once, y written once): the
// one-output form above, with one load in flight a thread, took 1441 us for 8192 rows x 8 x 7168, this one 444 us. The additions
// and their order are those of combine_kernel. A small window is a chain of two memory latencies: the row's order, then all that the order leads to and
// the row's status and the job's summary with it. 64 registers a thread, so that eight CTAs share a multiprocessor and cover the first of them (4096 rows
// x 8 x 2048 80 us, 100 with five CTAs; 114 while weights and ids were asked for between the two). The order comes through L1: from L2 every warp of a row's CTAs asks
// one 32-byte sector for it (53 rows x 8 x 7168 6.9 us, 5.0 through L1; the 4096 rows 62).
// EARLY: order, weights, ids and low_counts were complete before the launch in front was admitted (ChainHints): what the order leads to is known before the
// wait but for the values. An instance of its own: with a branch between the two, 1 row x 8 x 1024 took 4.4 us, 3.3 without.
constexpr u32 kVecTopK = 8;
template <bool CHAIN, bool EARLY>
__global__ void __launch_bounds__(128, EARLY ? 1 : 8) combine_vec_kernel(b200moe_combine_view v, u32 skip_bits, bool zero_skipped) {
    if (!EARLY) chain_begin_if<CHAIN>();
    const u32 o = 4u * (blockIdx.x * 128u + threadIdx.x);
    for (u32 row = blockIdx.y; row < v.rows; row += gridDim.y) {
        u32 slot[kVecTopK], part[kVecTopK], low = 0;  // part: the expert's id until the slot's turn comes, unless EARLY
        float w[kVecTopK];
        float4 x[kVecTopK];
        auto part_of = [&](u32 k, u32 e) { return v.low_counts ? (k < low ? 0u : 1u) : min(e / v.part_experts, v.parts - 1); };
        if (EARLY && v.low_counts) low = load_l2(v.low_counts + row);
#pragma unroll
        for (u32 k = 0; k < kVecTopK; ++k)
            if (k < v.top_k) slot[k] = EARLY ? load_l2(v.order + row * v.top_k + k) : load(v.order + row * v.top_k + k);
#pragma unroll
        for (u32 k = 0; k < kVecTopK; ++k)
            if (k < v.top_k) {
                slot[k] = min(slot[k], v.rows * v.top_k - 1u);  // the order of a row whose status is not zero may mean nothing
                if (EARLY) {
                    w[k] = __uint_as_float(load_l2(reinterpret_cast<const u32*>(v.weights) + slot[k]));
                    part[k] = part_of(k, v.low_counts ? 0u : load_l2(v.ids + slot[k]));
                }
            }
        if (EARLY && row == blockIdx.y) chain_begin();
        if (o >= v.hidden) return;
        const bool skipped = v.summary && (load(v.summary) & skip_bits);
        const u32 status = v.row_status ? load(v.row_status + row) : 0u;
#pragma unroll
        for (u32 k = 0; k < kVecTopK; ++k)
            if (k < v.top_k) {
                const float4* at = reinterpret_cast<const float4*>(v.raw + u64(slot[k]) * v.hidden + o);
                x[k] = EARLY ? load(at) : __ldcs(at);
                if (!EARLY) {
                    w[k] = load(v.weights + slot[k]);
                    part[k] = v.low_counts ? 0u : load(v.ids + slot[k]);
                }
            }
        if (!EARLY && v.low_counts) low = load(v.low_counts + row);
        const float4 sh = v.shared ? load(reinterpret_cast<const float4*>(v.shared + u64(row) * v.hidden + o)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        float4 y = sh, sum = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        u32 p = 0;
        bool run = true;  // a slot out of order ends the walk, as it does in combine_kernel
        auto flush = [&]() {
            y = make_float4(__fadd_rn(y.x, sum.x), __fadd_rn(y.y, sum.y), __fadd_rn(y.z, sum.z), __fadd_rn(y.w, sum.w));
            sum = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        };
#pragma unroll
        for (u32 k = 0; k < kVecTopK; ++k)
            if (run && k < v.top_k) {
                const u32 to = EARLY ? part[k] : part_of(k, part[k]);
                for (; p < to; ++p) flush();
                run = to == p;
                if (run) {
                    sum.x = __fadd_rn(sum.x, __fmul_rn(w[k], x[k].x)); sum.y = __fadd_rn(sum.y, __fmul_rn(w[k], x[k].y));
                    sum.z = __fadd_rn(sum.z, __fmul_rn(w[k], x[k].z)); sum.w = __fadd_rn(sum.w, __fmul_rn(w[k], x[k].w));
                }
            }
        for (; p < v.parts; ++p) flush();
        if (skipped || status) {
            if (!zero_skipped) continue;
            y = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
        *reinterpret_cast<float4*>(v.y + u64(row) * v.hidden + o) = y;
        if (v.y_bf16)
            *reinterpret_cast<uint2*>(v.y_bf16 + u64(row) * v.hidden + o) =
                make_uint2(bf16_rne_bits(y.x) | (u32(bf16_rne_bits(y.y)) << 16), bf16_rne_bits(y.z) | (u32(bf16_rne_bits(y.w)) << 16));
    }
}

// The slot-order form over whole rows with up to kVecTopK slots and even rows: two outputs a thread, and every word that the thread reads - the
// row's status, the job's summary, weights, values - is asked for before any of them is looked at: a small window is a chain of
// memory latencies (three in the general form, with two block barriers between them), a large one wants bytes in flight.
// 4096 rows x 8 x 2048: 79 us in the general form, 60 here (5.0 TB/s); 8 rows 3.1 and 2.2; 37 rows 4.0 and 2.8.
template <bool CHAIN>
__global__ void __launch_bounds__(128) combine_slots_kernel(b200moe_combine_view v, u32 skip_bits, bool zero_skipped) {
    chain_begin_if<CHAIN>();
    const u32 o = 2u * (blockIdx.x * 128u + threadIdx.x);
    if (o >= v.hidden) return;
    const u32 job = v.summary ? load(v.summary) : 0u;
    for (u32 row = blockIdx.y; row < v.rows; row += gridDim.y) {
        const u32 status = v.row_status ? load(v.row_status + row) : 0u;
        float2 x[kVecTopK];
        float w[kVecTopK];
#pragma unroll
        for (u32 k = 0; k < kVecTopK; ++k)
            if (k < v.top_k) {
                x[k] = load(reinterpret_cast<const float2*>(v.raw + (u64(row) * v.top_k + k) * v.hidden + o));
                w[k] = load(v.weights + row * v.top_k + k);
            }
        const float2 sh = v.shared ? load(reinterpret_cast<const float2*>(v.shared + u64(row) * v.hidden + o)) : make_float2(0.0f, 0.0f);
        float2 y = make_float2(0.0f, 0.0f);
#pragma unroll
        for (u32 k = 0; k < kVecTopK; ++k)
            if (k < v.top_k) y = make_float2(__fmaf_rn(w[k], x[k].x, y.x), __fmaf_rn(w[k], x[k].y, y.y));
        if (v.shared) y = make_float2(__fadd_rn(y.x, sh.x), __fadd_rn(y.y, sh.y));
        if ((job & skip_bits) || status) {  // fail closed (qwen_moe.cu:291)
            if (!zero_skipped) continue;
            y = make_float2(0.0f, 0.0f);
        }
        *reinterpret_cast<float2*>(v.y + u64(row) * v.hidden + o) = y;
        if (v.y_bf16) *reinterpret_cast<u32*>(v.y_bf16 + u64(row) * v.hidden + o) = bf16_rne_bits(y.x) | (u32(bf16_rne_bits(y.y)) << 16);
    }
}
__global__ void __launch_bounds__(256) canonical_sum_kernel(const float* a, const float* b, const float* c, u64 count, float* y) {
    const u64 i = u64(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const float ab = __fadd_rn(a[i], b[i]);
    y[i] = c ? __fadd_rn(ab, c[i]) : ab;
}

__global__ void __launch_bounds__(256) fill_u32_kernel(u32* p, u32 value, u64 count) {
    chain_begin();
    const u64 i = u64(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < count) p[i] = value;
}

__global__ void __launch_bounds__(256) row_order_kernel(const u32* ids, u32 rows, u32 top_k, u32* order) {
    chain_begin();
    const u32 row = blockIdx.x * blockDim.x + threadIdx.x;
    if (row >= rows) return;
    u32 key[kMaxTopK], slot[kMaxTopK];
    for (u32 k = 0; k < top_k; ++k) {
        const u32 s = row * top_k + k, e = ids[s];
        u32 j = k;
        while (j > 0 && key[j - 1] > e) { key[j] = key[j - 1]; slot[j] = slot[j - 1]; --j; }
        key[j] = e; slot[j] = s;
    }
    for (u32 k = 0; k < top_k; ++k) order[row * top_k + k] = slot[k];
}

// The complete first non-zero summary stays (include/strix/deferred_moe_status.hpp:19-28); one thread, stream ordered.
__global__ void merge_first_error_kernel(b200moe_first_error* record, const u32* summary, u32 domain) {
    const u32 bits = *summary;
    if (bits != 0u && record->domain == 0u) {
        record->bits = bits;
        record->domain = domain;
    }
}

}  // namespace

int launch_merge_first_error(b200moe_first_error* record, const u32* summary, u32 domain, cudaStream_t stream) {
    merge_first_error_kernel<<<1, 1, 0, stream>>>(record, summary, domain);
    return after_launch("merge_first_error");
}
int launch_combine(const b200moe_combine_view& v, cudaStream_t stream, u32 skip_bits, bool zero_skipped, const ChainHints& hints) {
    if (v.rows == 0) return B200MOE_OK;
    // PARTS in one row: a whole call 37.2 us in the general form, 35.5 in the wide one; 32 rows x 8 x 2048 of 8 parts 5.0 and 4.2 us.
    const bool whole = v.y && !v.y_blocks && v.top_k <= kVecTopK;
    const u32 rows = std::min<u32>(v.rows, 65535u);
    if (v.form == B200MOE_COMBINE_PARTS && whole && v.only_part < 0 && v.hidden % 4 == 0 && aligned(v.raw, 16) && aligned(v.y, 16) && aligned(v.shared, 16) && aligned(v.y_bf16, 8)) {
        const dim3 grid((v.hidden + 511) / 512, rows);
        if (!chain_pays(u64(grid.x) * rows)) plain_launch(combine_vec_kernel<false, false>, grid, 128, 0, stream, v, skip_bits, zero_skipped);
        else small_launch(hints.routes_done ? combine_vec_kernel<true, true> : combine_vec_kernel<true, false>, grid, 128, 0, stream, v, skip_bits, zero_skipped);
        return after_launch("combine");
    }
    if (v.form == B200MOE_COMBINE_FMA_SLOTS && whole && v.hidden % 2 == 0 && aligned(v.raw, 8) && aligned(v.y, 8) && aligned(v.shared, 8) && aligned(v.y_bf16, 4)) {
        const dim3 grid((v.hidden + 255) / 256, rows);
        if (chain_pays(u64(grid.x) * rows)) small_launch(combine_slots_kernel<true>, grid, 128, 0, stream, v, skip_bits, zero_skipped);
        else plain_launch(combine_slots_kernel<false>, grid, 128, 0, stream, v, skip_bits, zero_skipped);
        return after_launch("combine");
    }
    if (int rc = prefer_max_shared(reinterpret_cast<const void*>(combine_kernel))) return rc;
    const dim3 grid((v.hidden + 255) / 256, rows);
    if (chain_pays(u64(grid.x) * rows)) chain_launch(combine_kernel, grid, 256, 0, stream, v, skip_bits, zero_skipped);
    else plain_launch(combine_kernel, grid, 256, 0, stream, v, skip_bits, zero_skipped);
    return after_launch("combine");
}
int launch_canonical_sum(const float* a, const float* b, const float* c, u64 count, float* y, cudaStream_t stream) {
    if (count == 0) return B200MOE_OK;
    canonical_sum_kernel<<<static_cast<u32>((count + 255) / 256), 256, 0, stream>>>(a, b, c, count, y);
    return after_launch("canonical_sum");
}
int launch_fill_u32(u32* p, u32 value, u64 count, cudaStream_t stream) {
    if (count == 0) return B200MOE_OK;
    chain_launch(fill_u32_kernel, static_cast<u32>((count + 255) / 256), 256, 0, stream, p, value, count);
    return after_launch("fill_u32");
}
int launch_row_order(const u32* ids, u32 rows, u32 top_k, u32* order, cudaStream_t stream) {
    if (rows == 0) return B200MOE_OK;
    chain_launch(row_order_kernel, (rows + 255) / 256, 256, 0, stream, ids, rows, top_k, order);
    return after_launch("row_order");
}

}  // namespace b200moe
