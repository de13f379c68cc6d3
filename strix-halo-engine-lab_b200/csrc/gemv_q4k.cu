// Routed experts, Qwen A8 family, decode form: dequant-fused GEMVs over Q4_K super-blocks kept in their GGUF bytes.
//
// Contract (src/cpu/core/routed_expert.hpp:9-15, routed_expert.cpp:73-170): per super-block b of 256 weights and
// group j of 32 (g = 8b + j):  x_j = E_g * ((d * sc_j) * float(dot_j) - (dmin * m_j) * float(S_g)),
// pair_p = x_2p + x_2p+1, acc_p += pair_p over ascending b, value = (acc0 + acc1) + (acc2 + acc3); then
// h = (g / (1 + exp(-g))) * u and the A8 rule per 32 outputs. Q4_K down = the same row rule over K = inter
// (src/moe_a8_down_contract.cpp:141-146); Q8_0 down = four chains by g % 4 (routed_expert.cpp:110-144).
// Integer dots are exact (dp4a), every FP32 step is one IEEE operation, so results equal the host's bit for bit.
// The same kernels read the executor's other stored formats (routed_expert.hpp:27-28): Q5_K gate / up (176-byte
// super-blocks, the Q4_K rule with a fifth bit per weight) and Q5_1 down (24-byte blocks on the four chains,
// d * float(dot) + m * float(S_g)).
//
// Mapping: 4 lanes per super-block (lane = pair p: 32 B of nibbles serve groups 2p (low) and 2p+1 (high)), LPR lanes
// per weight row (8 / 16 / 32 by row length), so a warp streams 32 / LPR rows at once with 16-byte loads: per
// super-block one 16 B header (broadcast to its 4 lanes) + 4 x 32 B = 144 B, fully coalesced. The serial chain over b
// is rebuilt with shuffles. Up to 8 entries (tokens routed to the expert) share one pass over the weights.
//
// Roofline: HBM. Algorithmic bytes per (expert, call) = 2 * inter * hidden / 256 * 144 (gate, up) and
// hidden * inter / 256 * 144 (down), read once however many of the <= 8 staged rows use the expert.
#include <type_traits>

#include "declared_math.cuh"
#include "grouped_common.cuh"
#include "kernels.cuh"

namespace b200moe {
namespace {

constexpr int kR = 8;  // entries staged per pass

struct A8Smem {
    const i8* codes;    // [kR][width]
    const float* deltas;  // [kR][width / 32]
    const i32* sums;    // [kR][width / 32]
    u32 width;
};

__device__ __forceinline__ void q4k_factor(const uint4& hdr, u32 j, float d, float dm, float* D, float* DM) {
    const u32 shift = 8u * (j & 3u);
    const u32 a = (hdr.y >> shift) & 255u, b = (hdr.z >> shift) & 255u, c = (hdr.w >> shift) & 255u;
    const u32 sc = j < 4u ? (a & 63u) : ((c & 15u) | ((a >> 6) << 4));
    const u32 mn = j < 4u ? (b & 63u) : ((c >> 4) | ((b >> 6) << 4));
    *D = __fmul_rn(d, static_cast<float>(sc));
    *DM = __fmul_rn(dm, static_cast<float>(mn));
}

// 32 weights of one group against 32 codes: nibbles at `shift` (0 = low, 4 = high) of the 32 bytes wa | wb. Q5_K adds
// bit j of the 32 high-bit bytes ha | hb as bit 4 of each weight (routed_expert.cpp:88-95).
template <bool Q5K>
__device__ __forceinline__ int dot8(const uint4& wa, const uint4& wb, const uint4& ha, const uint4& hb, u32 j, const uint4& ca, const uint4& cb, u32 shift) {
    auto w = [&](u32 q, u32 h) -> int {
        u32 v = (q >> shift) & 0x0f0f0f0fu;
        if (Q5K) v |= ((h >> j) & 0x01010101u) << 4;
        return static_cast<int>(v);
    };
    int s = 0;
    s = __dp4a(w(wa.x, ha.x), static_cast<int>(ca.x), s);
    s = __dp4a(w(wa.y, ha.y), static_cast<int>(ca.y), s);
    s = __dp4a(w(wa.z, ha.z), static_cast<int>(ca.z), s);
    s = __dp4a(w(wa.w, ha.w), static_cast<int>(ca.w), s);
    s = __dp4a(w(wb.x, hb.x), static_cast<int>(cb.x), s);
    s = __dp4a(w(wb.y, hb.y), static_cast<int>(cb.y), s);
    s = __dp4a(w(wb.z, hb.z), static_cast<int>(cb.z), s);
    s = __dp4a(w(wb.w, hb.w), static_cast<int>(cb.w), s);
    return s;
}

// One Q4_K weight row (nblocks super-blocks at wrow) against nr <= kR staged A8 rows. LPR lanes cooperate on the row
// (lane-in-row li: super-block li / 4 of each step, pair li % 4); `base` is the first lane of the row's lane group.
// Every lane of the group returns the row values in out[].
template <int LPR, bool Q5K = false>
__device__ __forceinline__ void q4k_row(const u8* __restrict__ wrow, u32 nblocks, const A8Smem& x, int nr, u32 li, u32 base, float* out) {
    constexpr u32 BPI = LPR / 4;
    const u32 p = li & 3u, bsub = li >> 2;
    float acc[kR];
#pragma unroll
    for (int r = 0; r < kR; ++r) acc[r] = 0.0f;
    // The loads of step b0 + BPI are issued before the arithmetic of step b0 (one step of register prefetch): the row walk
    // is otherwise a chain of load -> dot -> shuffle with nothing in flight.
    struct Blk { uint4 hdr, q0, q1, h0, h1; };
    auto load_blk = [&](u32 b) {
        Blk k;
        k.hdr = make_uint4(0, 0, 0, 0); k.q0 = k.hdr; k.q1 = k.hdr; k.h0 = k.hdr; k.h1 = k.hdr;
        if (b < nblocks) {
            const uint4* blk = reinterpret_cast<const uint4*>(wrow + u64(b) * (Q5K ? kQ5KBlock : kQ4KBlock));
            k.hdr = load(blk);
            if (Q5K) { k.h0 = load(blk + 1); k.h1 = load(blk + 2); }  // Q5_K: 32 bytes of high bits between header and nibbles
            k.q0 = load(blk + (Q5K ? 3 : 1) + 2 * p);
            k.q1 = load(blk + (Q5K ? 4 : 2) + 2 * p);
        }
        return k;
    };
    Blk nxt = load_blk(bsub);
    for (u32 b0 = 0; b0 < nblocks; b0 += BPI) {
        const u32 b = b0 + bsub;
        const bool valid = b < nblocks;
        const Blk cur = nxt;
        nxt = load_blk(b + BPI);
        const uint4 hdr = cur.hdr, q0 = cur.q0, q1 = cur.q1, h0 = cur.h0, h1 = cur.h1;
        const float d = half_bits_to_float(hdr.x & 0xffffu), dm = half_bits_to_float(hdr.x >> 16);
        float Dl, DMl, Dh, DMh;
        q4k_factor(hdr, 2 * p, d, dm, &Dl, &DMl);
        q4k_factor(hdr, 2 * p + 1, d, dm, &Dh, &DMh);
        const u32 nb = min(BPI, nblocks - b0);
#pragma unroll
        for (int r = 0; r < kR; ++r) {
            if (r < nr) {
                float pair = 0.0f;
                if (valid) {
                    const uint4* c = reinterpret_cast<const uint4*>(x.codes + u64(r) * x.width + 256u * b + 64u * p);
                    const uint4 c0 = c[0], c1 = c[1], c2 = c[2], c3 = c[3];
                    const int dl = dot8<Q5K>(q0, q1, h0, h1, 2 * p, c0, c1, 0), dh = dot8<Q5K>(q0, q1, h0, h1, 2 * p + 1, c2, c3, 4);
                    const u32 g = r * (x.width / 32) + 8u * b + 2u * p;
                    const float2 e = *reinterpret_cast<const float2*>(x.deltas + g);
                    const int2 s = *reinterpret_cast<const int2*>(x.sums + g);
                    const float xl = __fmul_rn(e.x, __fsub_rn(__fmul_rn(Dl, static_cast<float>(dl)), __fmul_rn(DMl, static_cast<float>(s.x))));
                    const float xh = __fmul_rn(e.y, __fsub_rn(__fmul_rn(Dh, static_cast<float>(dh)), __fmul_rn(DMh, static_cast<float>(s.y))));
                    pair = __fadd_rn(xl, xh);
                }
                // acc_p += pair_p over ascending super-blocks: the serial chain, rebuilt across the row's lanes
#pragma unroll
                for (u32 bb = 0; bb < BPI; ++bb) {
                    const float t = __shfl_sync(0xffffffffu, pair, base + 4u * bb + p);
                    if (bb < nb) acc[r] = __fadd_rn(acc[r], t);
                }
            }
        }
    }
#pragma unroll
    for (int r = 0; r < kR; ++r) {
        const float a0 = __shfl_sync(0xffffffffu, acc[r], base + 0), a1 = __shfl_sync(0xffffffffu, acc[r], base + 1);
        const float a2 = __shfl_sync(0xffffffffu, acc[r], base + 2), a3 = __shfl_sync(0xffffffffu, acc[r], base + 3);
        out[r] = __fadd_rn(__fadd_rn(a0, a1), __fadd_rn(a2, a3));
    }
}

// Stage nr A8 rows (row ids from idx[]) of `width` into shared memory. All threads of the block take part.
__device__ __forceinline__ void stage_a8(const b200moe_a8_rows& src, const u32* idx, int nr, u32 width, i8* s_codes, float* s_deltas, i32* s_sums) {
    const u32 stride = src.stride ? src.stride : src.width, groups = width / 32;
    for (int r = 0; r < nr; ++r) {
        const u64 row = idx[r];
        const uint4* c = reinterpret_cast<const uint4*>(src.codes + row * stride);
        uint4* dc = reinterpret_cast<uint4*>(s_codes + u64(r) * width);
        for (u32 i = threadIdx.x; i < width / 16; i += blockDim.x) dc[i] = c[i];
        for (u32 i = threadIdx.x; i < groups; i += blockDim.x) {
            s_deltas[r * groups + i] = src.deltas[row * (stride / 32) + i];
            s_sums[r * groups + i] = src.sums ? src.sums[row * (stride / 32) + i] : 0;
        }
    }
}

// grid (inter / 32, max_union); 256 threads. One CTA = one expert x one 32-output group (= one A8 group of h).
template <int LPR, bool Q5K>
__global__ void __launch_bounds__(256) gate_up_q4k_kernel(b200moe_gate_up_view v) {
    chain_begin();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const u32 j = blockIdx.y;
    if (j >= v.routes.counts[0]) return;
    const u32 H = v.shape.hidden, I = v.shape.inter, groups = H / 32, nblocks = H / 256;
    i8* s_codes = reinterpret_cast<i8*>(smem_raw);
    float* s_deltas = reinterpret_cast<float*>(smem_raw + u64(kR) * H);
    i32* s_sums = reinterpret_cast<i32*>(s_deltas + kR * groups);
    float* s_g = reinterpret_cast<float*>(s_sums + kR * groups);  // [kR][32]
    float* s_u = s_g + kR * 32;
    __shared__ u32 s_rows[kR], s_slots[kR];

    const u32 expert = v.routes.experts[j], eb = v.routes.begins[j], ee = v.routes.begins[j + 1];
    const u32 lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    constexpr u32 RPW = 32 / LPR;
    const u32 sub = lane / LPR, li = lane % LPR, base = sub * LPR;
    const u64 row_bytes = u64(nblocks) * (Q5K ? kQ5KBlock : kQ4KBlock);
    const u8* gate = v.weights.gate + (u64(expert) * I + 32u * blockIdx.x) * row_bytes;
    const u8* up = v.weights.up + (u64(expert) * I + 32u * blockIdx.x) * row_bytes;
    const A8Smem xs{s_codes, s_deltas, s_sums, H};
    const u32 act_stride = v.act.stride ? v.act.stride : v.act.width;

    for (u32 p0 = eb; p0 < ee; p0 += kR) {
        const int nr = static_cast<int>(min(u32(kR), ee - p0));
        __syncthreads();
        if (threadIdx.x < (u32)nr) { s_rows[threadIdx.x] = v.routes.rows[p0 + threadIdx.x]; s_slots[threadIdx.x] = v.routes.slots[p0 + threadIdx.x]; }
        __syncthreads();
        stage_a8(v.x, s_rows, nr, H, s_codes, s_deltas, s_sums);
        __syncthreads();
        // 64 weight rows (gate 0..31, up 32..63): 8 warps x RPW rows per step
        for (u32 t0 = warp * RPW; t0 < 64; t0 += 8 * RPW) {
            const u32 t = t0 + sub;
            const u8* wrow = (t < 32 ? gate : up) + u64(t & 31u) * row_bytes;
            float val[kR];
            q4k_row<LPR, Q5K>(wrow, nblocks, xs, nr, li, base, val);
            if (li == 0) {
                float* dst = t < 32 ? s_g : s_u;
#pragma unroll
                for (int r = 0; r < kR; ++r) if (r < nr) dst[r * 32 + (t & 31u)] = val[r];
            }
        }
        __syncthreads();
        // epilogue: one warp per entry: SwiGLU, then the A8 rule over the 32 outputs
        for (int r = warp; r < nr; r += 8) {
            const float g = s_g[r * 32 + lane], u = s_u[r * 32 + lane];
            const u32 slot = s_slots[r];
            const u32 o = 32u * blockIdx.x + lane;
            if (v.gate_out) { v.gate_out[u64(slot) * I + o] = g; v.up_out[u64(slot) * I + o] = u; }
            const float h = swiglu_qwen(g, u);
            const bool bad = __any_sync(0xffffffffu, !finite_f(g) || !finite_f(u) || !finite_f(h));
            if (bad) {  // fail closed: nothing of the group is written (routed_expert.cpp:147-156)
                if (lane == 0) {
                    if (v.row_status) atomicOr(&v.row_status[s_rows[r]], B200MOE_ROW_PROJECTION_NONFINITE);
                    if (v.summary) atomicOr(v.summary, B200MOE_ROW_PROJECTION_NONFINITE);
                }
                continue;
            }
            float delta;
            int sum;
            const int code = a8_quantize_lane(h, &delta, &sum);
            v.act.codes[u64(slot) * act_stride + o] = static_cast<i8>(code);
            if (lane == 0) {
                v.act.deltas[u64(slot) * (act_stride / 32) + blockIdx.x] = delta;
                if (v.act.sums) v.act.sums[u64(slot) * (act_stride / 32) + blockIdx.x] = sum;
            }
        }
    }
}

// grid (hidden / rows_per_cta, max_union); 256 threads: rows_per_cta (64, or fewer when that grid would leave SMs idle:
// the dense block has one "expert") down rows per CTA, Q4_K rows over K = inter.
template <int LPR>
__global__ void __launch_bounds__(256) down_q4k_kernel(b200moe_down_view v, u32 rows_per_cta) {
    chain_begin();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    if (block_skips(v.summary)) return;  // a failed projection skips the whole down stage (routed_expert.hpp:17-19)
    const u32 j = blockIdx.y;
    if (j >= v.routes.counts[0]) return;
    const u32 H = v.shape.hidden, I = v.shape.inter, groups = I / 32, nblocks = I / 256;
    i8* s_codes = reinterpret_cast<i8*>(smem_raw);
    float* s_deltas = reinterpret_cast<float*>(smem_raw + u64(kR) * I);
    i32* s_sums = reinterpret_cast<i32*>(s_deltas + kR * groups);
    __shared__ u32 s_slots[kR];
    const u32 expert = v.routes.experts[j], eb = v.routes.begins[j], ee = v.routes.begins[j + 1];
    const u32 lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    constexpr u32 RPW = 32 / LPR;
    const u32 sub = lane / LPR, li = lane % LPR, base = sub * LPR;
    const u64 row_bytes = u64(nblocks) * kQ4KBlock;
    const u32 o0 = rows_per_cta * blockIdx.x;
    const u8* down = v.weights.down + (u64(expert) * H + o0) * row_bytes;
    const A8Smem xs{s_codes, s_deltas, s_sums, I};

    for (u32 p0 = eb; p0 < ee; p0 += kR) {
        const int nr = static_cast<int>(min(u32(kR), ee - p0));
        __syncthreads();
        if (threadIdx.x < (u32)nr) s_slots[threadIdx.x] = v.routes.slots[p0 + threadIdx.x];
        __syncthreads();
        stage_a8(v.act, s_slots, nr, I, s_codes, s_deltas, s_sums);
        __syncthreads();
        for (u32 t0 = warp * RPW; t0 < rows_per_cta; t0 += 8 * RPW) {
            const u32 t = t0 + sub;
            float val[kR];
            q4k_row<LPR>(down + u64(t) * row_bytes, nblocks, xs, nr, li, base, val);
            if (li == 0) {
#pragma unroll
                for (int r = 0; r < kR; ++r) if (r < nr) v.raw[u64(s_slots[r]) * H + o0 + t] = val[r];
            }
        }
    }
}

// One 32-weight block of the four-chain down tensors: the 32 weights as bytes, the factor and (Q5_1) the minimum.
template <bool Q51>
struct ChainBlock { u32 q[8]; float d, mn; };
template <bool Q51>
__device__ __forceinline__ void load_chain_block(const u8* b, ChainBlock<Q51>& o) {
    if (Q51) {
        // Q5_1 (routed_expert.cpp:124-133): 24-byte blocks, 8-byte aligned. Weight k < 16 = low nibble of byte k, k >= 16 = high
        // nibble of byte k - 16, bit k of the 32 high bits on top: unsigned 0..31. Kept raw here, spread when used.
        const uint2* b8 = reinterpret_cast<const uint2*>(b);
        const uint2 hd = load(b8), qa = load(b8 + 1), qb = load(b8 + 2);
        o.q[0] = qa.x; o.q[1] = qa.y; o.q[2] = qb.x; o.q[3] = qb.y; o.q[4] = hd.x; o.q[5] = hd.y;
    } else {  // 34-byte blocks are 2-byte aligned: whole words where the quants lie on one, else words and a byte permute
        const bool odd = (reinterpret_cast<uintptr_t>(b) & 2u) != 0;
        o.d = half_bits_to_float(load(reinterpret_cast<const u16*>(b)));
        if (odd) {
            const u32* w = reinterpret_cast<const u32*>(b + 2);
#pragma unroll
            for (int i = 0; i < 8; ++i) o.q[i] = load(w + i);
        } else {
            const u32* w = reinterpret_cast<const u32*>(b);
            u32 r[9];
#pragma unroll
            for (int i = 0; i < 8; ++i) r[i] = load(w + i);
            r[8] = load(reinterpret_cast<const u16*>(b + 32));  // nothing is read past the block
#pragma unroll
            for (int i = 0; i < 8; ++i) o.q[i] = __byte_perm(r[i], r[i + 1], 0x5432u);
        }
    }
}
template <bool Q51>
__device__ __forceinline__ void spread_chain_block(ChainBlock<Q51>& o) {
    if (!Q51) return;
    const u32 qs[4] = {o.q[0], o.q[1], o.q[2], o.q[3]}, hd = o.q[4], hb = o.q[5];
    o.d = half_bits_to_float(hd & 0xffffu);
    o.mn = half_bits_to_float(hd >> 16);
    auto spread = [](u32 x) { return ((x & 15u) * 0x02040810u) & 0x10101010u; };  // bit k of four to bit 4 of byte k
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        o.q[i] = (qs[i] & 0x0f0f0f0fu) | spread(hb >> (4 * i));
        o.q[4 + i] = ((qs[i] >> 4) & 0x0f0f0f0fu) | spread(hb >> (16 + 4 * i));
    }
}

// Q8_0 / Q5_1 down in the four-chain rule (routed_expert.cpp:110-144): chain c = g % 4 adds E_g * (d * float(dot)) in
// ascending g; value = (acc0 + acc1) + (acc2 + acc3). A lane IS one chain of one row (lane = 4 * row + chain), so the chain is a
// plain register sum and the four lanes of a row read neighbouring blocks. (The form before this one gave a row to a warp
// with a lane per group and handed every term round by shuffles: with 20 groups a row, 12 lanes idled and a term cost eight
// shuffles.) What bounds it: the latency of the weight loads, so a lane asks for kChainBatch blocks at once, the first batch
// before the entries' A8 rows are staged. 4 rows over 128 experts of 640 -> 2560, top 8, Q5_1: 43.6 -> 23.1 us.
// grid (hidden / 64, max_union); 256 threads, 8 rows a warp.
constexpr u32 kChainBatch = 3;
template <bool Q51>
__global__ void __launch_bounds__(256) down_q8_chain4_kernel(b200moe_down_view v) {
    chain_begin();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    if (block_skips(v.summary)) return;
    const u32 j = blockIdx.y;
    if (j >= v.routes.counts[0]) return;
    const u32 H = v.shape.hidden, I = v.shape.inter, groups = I / 32;
    i8* s_codes = reinterpret_cast<i8*>(smem_raw);
    float* s_deltas = reinterpret_cast<float*>(smem_raw + u64(kR) * I);
    i32* s_sums = reinterpret_cast<i32*>(s_deltas + kR * groups);
    __shared__ u32 s_slots[kR];
    const u32 expert = v.routes.experts[j], eb = v.routes.begins[j], ee = v.routes.begins[j + 1];
    const u32 lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, chain = lane & 3u;
    constexpr u32 block = Q51 ? kQ51Block : kQ8Block;
    const u32 o = 64u * blockIdx.x + 8u * warp + (lane >> 2);
    const u8* wrow = v.weights.down + (u64(expert) * H + o) * (u64(groups) * block);

    for (u32 p0 = eb; p0 < ee; p0 += kR) {
        const int nr = static_cast<int>(min(u32(kR), ee - p0));
        ChainBlock<Q51> w[kChainBatch];
        auto load_batch = [&](u32 g0) {
#pragma unroll
            for (u32 i = 0; i < kChainBatch; ++i)
                if (g0 + 4u * i < groups) load_chain_block<Q51>(wrow + u64(g0 + 4u * i) * block, w[i]);
        };
        load_batch(chain);
        __syncthreads();
        if (threadIdx.x < (u32)nr) s_slots[threadIdx.x] = v.routes.slots[p0 + threadIdx.x];
        __syncthreads();
        stage_a8(v.act, s_slots, nr, I, s_codes, s_deltas, s_sums);
        __syncthreads();
        float acc[kR];
#pragma unroll
        for (int r = 0; r < kR; ++r) acc[r] = 0.0f;
        for (u32 g0 = chain; g0 < groups; g0 += 4u * kChainBatch) {
#pragma unroll
            for (u32 i = 0; i < kChainBatch; ++i) {
                const u32 g = g0 + 4u * i;
                if (g >= groups) break;
                ChainBlock<Q51>& b = w[i];
                spread_chain_block<Q51>(b);
#pragma unroll
                for (int r = 0; r < kR; ++r) {
                    if (r < nr) {
                        const uint4* c = reinterpret_cast<const uint4*>(s_codes + u64(r) * I + 32u * g);
                        const uint4 c0 = c[0], c1 = c[1];
                        int dot = 0;
                        dot = __dp4a((int)b.q[0], (int)c0.x, dot); dot = __dp4a((int)b.q[1], (int)c0.y, dot);
                        dot = __dp4a((int)b.q[2], (int)c0.z, dot); dot = __dp4a((int)b.q[3], (int)c0.w, dot);
                        dot = __dp4a((int)b.q[4], (int)c1.x, dot); dot = __dp4a((int)b.q[5], (int)c1.y, dot);
                        dot = __dp4a((int)b.q[6], (int)c1.z, dot); dot = __dp4a((int)b.q[7], (int)c1.w, dot);
                        float combined = __fmul_rn(b.d, static_cast<float>(dot));
                        if (Q51) combined = __fadd_rn(combined, __fmul_rn(b.mn, static_cast<float>(s_sums[r * groups + g])));
                        acc[r] = __fadd_rn(acc[r], __fmul_rn(s_deltas[r * groups + g], combined));
                    }
                }
            }
            load_batch(g0 + 4u * kChainBatch);
        }
#pragma unroll
        for (int r = 0; r < kR; ++r) {
            if (r < nr) {  // uniform over the block
                const float pair = __fadd_rn(acc[r], __shfl_xor_sync(0xffffffffu, acc[r], 1));
                const float y = __fadd_rn(pair, __shfl_xor_sync(0xffffffffu, pair, 2));
                if (chain == 0) v.raw[u64(s_slots[r]) * H + o] = y;
            }
        }
    }
}

// The same rule with the weight rows brought in by bulk copies: rows_per_item rows of an expert lie one behind the other in memory, so an item = (expert, that
// many rows) is ONE copy. A CTA of 4 threads a row walks its items round-robin over two stages: an item's weights are asked for two items ahead,
// its entries' A8 rows (up to `cap` of them, the rest in further passes) one item ahead by asynchronous copies. An early launch (ChainHints) asks for its
// first two items' weights before it waits for the launch in front.
// What bounds it: the trip to HBM and the start, for the few items a CTA has in a decode window. The form above, whose 1280 CTAs (4 rows over 128 experts of
// 640 -> 2560, top 8, Q5_1) each made that trip twice from registers, eight a multiprocessor and a second wave of 96, took 20 us.
struct ChainPlan {
    u32 rows_per_item, n_chunks, cap, stage_bytes, a8_bytes;  // a8_bytes: of `cap` entries
    u32 early, wait_limit, stall_stage;  // test hook: item `stall_stage` of a CTA's items and those behind it are not asked for
};
template <bool Q51>
__global__ void __launch_bounds__(256, 4) down_chain4_stream_kernel(b200moe_down_view v, ChainPlan plan) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const u32 H = v.shape.hidden, I = v.shape.inter, groups = I / 32, R = plan.rows_per_item;
    constexpr u32 block = Q51 ? kQ51Block : kQ8Block;
    const u64 row_bytes = u64(groups) * block;
    __shared__ u64 full[2];
    __shared__ u32 s_abort, s_slots[2][kR];
    const u32 tid = threadIdx.x, chain = tid & 3u, my_row = tid >> 2;
    if (tid == 0) {
        q4k::mbar_init(&full[0], 1); q4k::mbar_init(&full[1], 1);
        s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (!plan.early) chain_begin();
    const u32 n_items = load_l2(v.routes.counts) * plan.n_chunks;
    struct Item { u32 id, j, chunk; };  // j: place of its expert in the union. The CTA's items are gridDim.x apart
    const u32 dj = gridDim.x / plan.n_chunks, dc = gridDim.x - dj * plan.n_chunks;
    auto onward = [&](Item x) {
        x.id += gridDim.x; x.j += dj; x.chunk += dc;
        if (x.chunk >= plan.n_chunks) { x.chunk -= plan.n_chunks; ++x.j; }
        return x;
    };
    const Item first_item{blockIdx.x, blockIdx.x / plan.n_chunks, blockIdx.x % plan.n_chunks};
    auto ask = [&](u32 n, const Item& x) {  // one thread
        unsigned char* st = smem_raw + (n & 1u) * plan.stage_bytes;
        const u32 bytes = R * static_cast<u32>(row_bytes);
        q4k::mbar_expect_tx(&full[n & 1u], bytes);
        q4k::bulk_g2s(st, v.weights.down + (u64(load_l2(v.routes.experts + x.j)) * H + R * x.chunk) * row_bytes, bytes, &full[n & 1u]);
    };
    u32 asked = 0;
    Item to_ask = first_item;
    const u32 n_ask = plan.stall_stage == 0xffffffffu ? n_items : min(n_items, blockIdx.x + plan.stall_stage * gridDim.x);
    if (tid == 0)
        for (; asked < 2 && to_ask.id < n_ask; ++asked, to_ask = onward(to_ask)) ask(asked, to_ask);
    if (plan.early) chain_begin();
    auto drain = [&](u32 from) {  // one thread: the copies asked for land (the wait is bounded) before the CTA retires
        for (u32 n = from; n < asked; ++n)
            for (u32 i = 0; i < (plan.wait_limit >> 4) + 64u; ++i)
                if (q4k::mbar_try_wait(&full[n & 1u], (n >> 1) & 1u, q4k::kWaitHintNs)) break;
    };
    if (block_skips(v.summary)) {  // a failed projection skips the whole down stage (routed_expert.hpp:17-19)
        if (tid == 0) drain(0);
        return;
    }
    unsigned char* a8 = smem_raw + 2 * plan.stage_bytes;
    const u32 stride = v.act.stride ? v.act.stride : v.act.width;
    // entries [first, first + nr) into buffer b: codes[nr][I], deltas[cap][groups], sums[cap][groups]
    auto stage = [&](u32 b, u32 first, u32 nr) {
        unsigned char* to = a8 + b * plan.a8_bytes;
        float* deltas = reinterpret_cast<float*>(to + plan.cap * I);
        i32* sums = reinterpret_cast<i32*>(deltas + plan.cap * groups);
        for (u32 r = 0; r < nr; ++r) {
            const u32 slot = load(v.routes.slots + first + r);
            if (tid == 0) s_slots[b][r] = slot;
            const i8* c = v.act.codes + u64(slot) * stride;
            for (u32 i = tid; i < I / 16; i += blockDim.x) grouped::cp_async16(to + r * I + 16u * i, c + 16u * i);
            const float* d = v.act.deltas + u64(slot) * (stride / 32);
            const i32* sm = v.act.sums ? v.act.sums + u64(slot) * (stride / 32) : nullptr;
            for (u32 i = tid; i < groups; i += blockDim.x) {
                grouped::cp_async4(deltas + r * groups + i, d + i);
                if (Q51) grouped::cp_async4(sums + r * groups + i, sm + i);
            }
        }
    };
    auto entries = [&](const Item& x, u32& first, u32& count) {
        first = load(v.routes.begins + x.j);
        count = load(v.routes.begins + x.j + 1) - first;
    };
    u32 first = 0, count = 0;
    if (blockIdx.x < n_items) {
        entries(first_item, first, count);
        stage(0, first, min(plan.cap, count));
    }
    bool ok = true;
    u32 n = 0;
    for (Item item = first_item; item.id < n_items; item = onward(item), ++n) {
        const u32 b = n & 1u, o = R * item.chunk + my_row;
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        u32 next_first = 0, next_count = 0;
        const Item next = onward(item);
        if (next.id < n_items) {
            entries(next, next_first, next_count);
            stage(b ^ 1u, next_first, min(plan.cap, next_count));
        }
        ok = q4k::mbar_wait(&full[b], (n >> 1) & 1u, plan.wait_limit, &s_abort);
        if (__syncthreads_or(!ok)) { ok = false; break; }
        const unsigned char* wrow = smem_raw + b * plan.stage_bytes + u64(my_row) * row_bytes;
        const unsigned char* from = a8 + b * plan.a8_bytes;
        const float* deltas = reinterpret_cast<const float*>(from + plan.cap * I);
        const i32* sums = reinterpret_cast<const i32*>(deltas + plan.cap * groups);
        for (u32 p0 = 0; p0 < count; p0 += plan.cap) {
            const u32 nr = min(plan.cap, count - p0);
            if (p0) {  // an expert of more entries: the passes after the first
                __syncthreads();
                stage(b, first + p0, nr);
                asm volatile("cp.async.wait_all;" ::: "memory");
                __syncthreads();
            }
            // Up to so many entries; one and two, the common counts of a window that keeps this form, have code of their own: a launch fetches its instructions cold, and the checks
            // of eight entries were a third of them. 4 rows over 128 experts of 640 -> 2560, top 8, Q5_1: 18.8 -> 12.1 us a launch, with the items' divisions gone, the fifth bits spread by a product
            // and four blocks of an only entry at once (two, and of more entries too, 14.5: more registers, fewer CTAs).
            auto run = [&](auto most) {
                constexpr int kMost = decltype(most)::value;
                float acc[kMost];
#pragma unroll
                for (int r = 0; r < kMost; ++r) acc[r] = 0.0f;
#pragma unroll (kMost == 1 ? 4 : 1)
                for (u32 g = chain; g < groups; g += 4) {
                    ChainBlock<Q51> w;
                    load_chain_block<Q51>(wrow + g * block, w);
                    spread_chain_block<Q51>(w);
#pragma unroll
                    for (int r = 0; r < kMost; ++r) {
                        if (kMost <= 2 || r < (int)nr) {
                            const uint4* c = reinterpret_cast<const uint4*>(from + r * I + 32u * g);
                            const uint4 c0 = c[0], c1 = c[1];
                            int da = __dp4a((int)w.q[0], (int)c0.x, 0), db = __dp4a((int)w.q[4], (int)c1.x, 0);
                            da = __dp4a((int)w.q[1], (int)c0.y, da); db = __dp4a((int)w.q[5], (int)c1.y, db);
                            da = __dp4a((int)w.q[2], (int)c0.z, da); db = __dp4a((int)w.q[6], (int)c1.z, db);
                            da = __dp4a((int)w.q[3], (int)c0.w, da); db = __dp4a((int)w.q[7], (int)c1.w, db);
                            float combined = __fmul_rn(w.d, static_cast<float>(da + db));
                            if (Q51) combined = __fadd_rn(combined, __fmul_rn(w.mn, static_cast<float>(sums[r * groups + g])));
                            acc[r] = __fadd_rn(acc[r], __fmul_rn(deltas[r * groups + g], combined));
                        }
                    }
                }
#pragma unroll
                for (int r = 0; r < kMost; ++r) {
                    if (kMost <= 2 || r < (int)nr) {  // uniform over the block
                        const float pair = __fadd_rn(acc[r], __shfl_xor_sync(0xffffffffu, acc[r], 1));
                        const float y = __fadd_rn(pair, __shfl_xor_sync(0xffffffffu, pair, 2));
                        if (chain == 0) v.raw[u64(s_slots[b][r]) * H + o] = y;
                    }
                }
            };
            if (nr == 1u) run(std::integral_constant<int, 1>{});
            else if (nr == 2u) run(std::integral_constant<int, 2>{});
            else run(std::integral_constant<int, kR>{});
        }
        __syncthreads();  // the stage and the buffer have been read
        if (tid == 0 && to_ask.id < n_ask) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            ask(n + 2, to_ask);
            ++asked;
            to_ask = onward(to_ask);
        }
        first = next_first; count = next_count;
    }
    if (!ok) {
        asm volatile("cp.async.wait_all;" ::: "memory");
        if (tid == 0) {
            drain(n);
            if (v.summary) atomicOr(const_cast<u32*>(v.summary), q4k::kAbortBit);
        }
    }
}

// Rows of an item and entries of a pass: as many rows (64, 32 or 16) as let three CTAs share a multiprocessor, fewer CTAs for rows so long that not even 16
// do. False where the form above is the better one: rows too long for two stages, and windows of more than four rounds of items (over the experts that are met) whose long rows leave
// a multiprocessor no more than 128 threads (four a row and CTA), for Q5_1 with its longer decoding fewer than 512. Layers of Q4_K gate/up, this form and the one above, us:
// 60 experts of 2560, top 4, Q5_1: 768 wide 1 row 15.1 and 17.7, 30 rows 74.7 and 79.2; 1536 wide 1 row 17.2 and 22.6, 4 rows 40.9 and 44.7, 8 rows 64.0 and 65.8, 15 rows 96 and 91,
// 60 rows 236 and 176; 2816 wide 1 row 23.5 and 32.2, 2 rows 36.7 and 42.0, 4 rows 60 and 66, 8 rows 137 and 95; Q8_0: 1536 wide 8 rows 74 and 82, 15 rows 115 and 121; 2816 wide
// 1 row 29.3 and 48.6, 2 rows 45.0 and 66.6, 4 rows 108 and 94, 8 rows 174 and 142. Over 527 random layers that keep the dp4a forms the choice takes 0.7 % more than the better of the two.
bool chain_plan(const b200moe_down_view& v, u32 rows, ChainPlan* p, u32* smem, u32* per_sm) {
    const u32 I = v.shape.inter, H = v.shape.hidden, block = v.shape.down_type == B200MOE_TYPE_Q5_1 ? kQ51Block : kQ8Block;
    const u64 row_bytes = u64(I / 32) * block;
    p->cap = std::min<u32>(kR, std::max(1u, rows));
    p->a8_bytes = (p->cap * (I + I / 32 * 8) + 15u) / 16u * 16u;
    const u32 limit = debug_value(B200MOE_DEBUG_WAIT_LIMIT), stall = debug_value(B200MOE_DEBUG_STALL_STAGE);
    p->wait_limit = limit ? limit : 1u << 18;  // about a second
    p->stall_stage = stall ? stall - 1u : 0xffffffffu;
    for (u32 R = 64; R >= 16; R /= 2) {
        const u64 stage = (R * row_bytes + 127) / 128 * 128, total = 2 * (stage + p->a8_bytes);
        if (total > 75u * 1024u && !(R == 16 && total <= 226u * 1024u)) continue;
        p->rows_per_item = R; p->n_chunks = H / R; p->stage_bytes = static_cast<u32>(stage);
        *smem = static_cast<u32>(total);
        *per_sm = std::max(1u, std::min(2048u / (4u * R), 227u * 1024u / (*smem + 1024u)));
        const u64 at_once = u64(*per_sm) * static_cast<u32>(device_sm_count());
        if (4u * R * *per_sm < (block == kQ51Block ? 512u : 129u) && u64(p->n_chunks) * experts_met(v.shape, u64(rows) * v.shape.top_k, v.max_union) > 4 * at_once) return false;
        return u64(p->n_chunks) * v.max_union < (1u << 30);
    }
    return false;
}

template <class K>
int set_smem(K kernel, u32 bytes) {
    return ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), bytes);
}
inline int lanes_per_row(u32 nblocks) { return nblocks > 4 ? 32 : (nblocks > 2 ? 16 : 8); }

}  // namespace

int launch_gate_up_q4k(const b200moe_gate_up_view& v, cudaStream_t stream) {
    const u32 H = v.shape.hidden, I = v.shape.inter;
    if (v.max_union == 0) return B200MOE_OK;
    const u32 smem = kR * (H + H / 32 * 8) + 2 * kR * 32 * 4;
    const dim3 grid(I / 32, v.max_union);
#define B200_GU(L)                                                                   \
    {                                                                                \
        if (v.shape.gate_type == B200MOE_TYPE_Q5_K) {                                \
            if (int rc = set_smem(gate_up_q4k_kernel<L, true>, smem)) return rc;     \
            chain_launch(gate_up_q4k_kernel<L, true>, grid, 256, smem, stream, v);             \
        } else {                                                                     \
            if (int rc = set_smem(gate_up_q4k_kernel<L, false>, smem)) return rc;    \
            chain_launch(gate_up_q4k_kernel<L, false>, grid, 256, smem, stream, v);            \
        }                                                                            \
    }
    switch (lanes_per_row(H / 256)) {
        case 32: B200_GU(32) break;
        case 16: B200_GU(16) break;
        default: B200_GU(8) break;
    }
#undef B200_GU
    return after_launch("gate_up_q4k");
}

int launch_down_q4k(const b200moe_down_view& v, cudaStream_t stream) {
    const u32 H = v.shape.hidden, I = v.shape.inter;
    if (v.max_union == 0) return B200MOE_OK;
    const u32 smem = kR * (I + I / 32 * 8);
    u32 rpc = 64;  // rows per CTA: halved while the grid would not give every SM two CTAs (H is a multiple of 256)
    while (rpc > 8 && u64(H / rpc) * v.max_union < 2u * static_cast<u32>(device_sm_count())) rpc /= 2;  // at least two CTAs per SM
    const dim3 grid(H / rpc, v.max_union);
#define B200_DN(L)                                                     \
    {                                                                  \
        if (int rc = set_smem(down_q4k_kernel<L>, smem)) return rc;    \
        chain_launch(down_q4k_kernel<L>, grid, 256, smem, stream, v, rpc);       \
    }
    switch (lanes_per_row(I / 256)) {
        case 32: B200_DN(32) break;
        case 16: B200_DN(16) break;
        default: B200_DN(8) break;
    }
#undef B200_DN
    return after_launch("down_q4k");
}

int launch_down_q8_chain4(const b200moe_down_view& v, u32 rows, const ChainHints& hints, cudaStream_t stream) {
    const u32 H = v.shape.hidden, I = v.shape.inter;
    if (v.max_union == 0) return B200MOE_OK;
    const bool q51 = v.shape.down_type == B200MOE_TYPE_Q5_1;
    ChainPlan p{};
    u32 smem = 0, per_sm = 0;
    if (debug_value(B200MOE_DEBUG_DECODE_FORM) != 3 && aligned(v.weights.down, 16) && chain_plan(v, rows, &p, &smem, &per_sm)) {
        p.early = hints.routes_done;
        const u32 grid = static_cast<u32>(std::min<u64>(u64(per_sm) * static_cast<u32>(device_sm_count()), u64(p.n_chunks) * v.max_union));
        const auto kernel = q51 ? down_chain4_stream_kernel<true> : down_chain4_stream_kernel<false>;
        if (int rc = set_smem(kernel, smem)) return rc;
        chain_launch(kernel, grid, 4 * p.rows_per_item, smem, stream, v, p);
        return after_launch("down_chain4_stream");
    }
    const u32 bytes = kR * (I + I / 32 * 8);
    const auto kernel = q51 ? down_q8_chain4_kernel<true> : down_q8_chain4_kernel<false>;
    if (int rc = set_smem(kernel, bytes)) return rc;
    chain_launch_l1(kernel, dim3(H / 64, v.max_union), 256, bytes, stream, v);  // one expert of 5120 -> 512, Q8_0, 90 rows behind gate/up: 1200 -> 620 us
    return after_launch("down_q8_chain4");
}

}  // namespace b200moe
