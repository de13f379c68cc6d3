// Score transform, k-pass top-k selection and weights of one router row by one warp: device code shared by the
// stand-alone select kernel (router.cu) and the fused select + routes kernel of decode windows (routes.cu).
// Contracts: include/strix/moe/route_policy.hpp:80-156 (see router.cu).
#pragma once
#include "declared_math.cuh"

namespace b200moe {
namespace select_detail {

__device__ __forceinline__ u32 ordered_key(float v) {  // route_policy.hpp:84-88
    u32 u = __float_as_uint(v);
    if (u == 0x80000000u) u = 0;
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
// True when candidate (a, ai) beats the current pick (b, bi) in a reduction over disjoint ascending scans: the
// serial scan keeps the lower id on equal keys, so the parallel form orders by (key desc, id asc).
__device__ __forceinline__ bool beats(u32 key, float a, u32 ai, float b, u32 bi) {
    if (key == B200MOE_KEY_FLOAT_SERIAL) return a > b || (a == b && ai < bi);
    const u32 ka = ordered_key(a), kb = ordered_key(b);
    return ka > kb || (ka == kb && ai < bi);
}

constexpr u32 kNone = 0xffffffffu;

// The serial scan of one selection pass (route_policy.hpp:104-114) over a short candidate list, skipping `skip`.
__device__ __forceinline__ u32 serial_pick(u32 key, const float* c, u32 n, u32 skip) {
    u32 pick = kNone;
    float best = 0.0f;
    for (u32 e = 0; e < n; ++e) {
        if (e == skip) continue;
        const bool better = key == B200MOE_KEY_FLOAT_SERIAL ? c[e] > best : ordered_key(c[e]) > ordered_key(best);
        if (pick == kNone || better) { pick = e; best = c[e]; }
    }
    return pick;
}

// One k-pass over `n` candidates c[] (shared memory), lane-strided; `taken` holds this lane's taken candidates (bit j
// = candidate lane + 32 j), `allowed_groups` masks candidates by group (per = candidates per group; all ones = no
// mask). Returns the pick (kNone when nothing is left) to every lane and marks it taken.
__device__ __forceinline__ u32 k_pass(u32 key, const float* c, u32 n, u32 lane, u32& taken, u32 allowed_groups, u32 per) {
    // the serial scan's first candidate: lowest untaken allowed id
    u32 first = kNone, pick = kNone;
    float best = 0.0f;
    for (u32 j = 0, e = lane; e < n; ++j, e += 32) {
        if ((taken >> j) & 1u) continue;
        if (!((allowed_groups >> (e / per)) & 1u)) continue;
        if (first == kNone) first = e;
        const float v = c[e];
        if (key == B200MOE_KEY_FLOAT_SERIAL && v != v) continue;  // a NaN never replaces a pick
        if (pick == kNone || beats(key, v, e, best, pick)) { pick = e; best = v; }
    }
#pragma unroll
    for (int d = 16; d; d >>= 1) {
        const u32 of = __shfl_xor_sync(0xffffffffu, first, d);
        first = min(first, of);
        const u32 op = __shfl_xor_sync(0xffffffffu, pick, d);
        const float ob = __shfl_xor_sync(0xffffffffu, best, d);
        if (op != kNone && (pick == kNone || beats(key, ob, op, best, pick))) { pick = op; best = ob; }
    }
    if (first == kNone) return kNone;
    if (key == B200MOE_KEY_FLOAT_SERIAL) {
        const float fv = c[first];
        if (fv != fv) pick = first;  // a NaN taken as the first candidate stays (route_policy.hpp:11-12)
    }
    if (pick != kNone && (pick & 31u) == lane) taken |= 1u << (pick >> 5);
    return pick;
}

// The value whose key it is (a zero's sign is gone).
__device__ __forceinline__ float key_value(u32 k) { return __uint_as_float((k & 0x80000000u) ? k & 0x7fffffffu : ~k); }

// Fast path of one row, one warp: the row's choices live in registers (EPL per lane, expert lane + 32 j) as ordered keys, none of them a NaN:
// the contract's serial scans are then "largest choice, lowest id on ties" under either key rule, which two warp reductions a pass give (the
// largest key, then the lowest id that has it; 0 is no candidate's key). Groups are runs of 2^i lanes or whole runs of 32 experts: a group's two
// best are merged by shuffles or reductions. Returns false - with nothing stored - when the row needs the general path. `s` = this warp's
// scratch of scratch_floats(experts) floats on a 16-byte boundary (shared memory); holds the scores afterwards.
// The work is a chain of latencies in one warp, mostly run once a call on cold instruction caches, so the long steps (exp, quotient) are
// rolled loops of four values a lane: 8 rows of 128 took 12,800 clocks with a shuffle tree a pass and everything unrolled.
template <int EPL>
__device__ __forceinline__ bool select_row_fast(const float* logits, float* scores_out, const float* bias, const b200moe_route_policy& p, u32 row, u32 lane, float* s, u32* picked) {
    const u32 E = p.experts, per = E / p.n_group;
    const float* z = logits + u64(row) * E;
    const float ninf = -__uint_as_float(0x7f800000u);
    float m = ninf;
#pragma unroll
    for (int j = 0; j < EPL; ++j) {
        const u32 e = lane + 32u * j;
        if (e < E) { const float v = z[e]; s[e] = v; m = v > m ? v : m; }
    }
    if (p.score == B200MOE_SCORE_SOFTMAX) {  // route_policy.hpp:135-144
#pragma unroll
        for (int d = 16; d; d >>= 1) { const float o = __shfl_xor_sync(0xffffffffu, m, d); m = o > m ? o : m; }
#pragma unroll 1
        for (u32 e0 = lane; e0 < E; e0 += 128) {
            float v[4];
#pragma unroll
            for (u32 i = 0; i < 4; ++i) v[i] = e0 + 32u * i < E ? s[e0 + 32u * i] : ninf;
#pragma unroll
            for (u32 i = 0; i < 4; ++i) v[i] = declared_exp(__fsub_rn(v[i], m));
#pragma unroll
            for (u32 i = 0; i < 4; ++i) if (e0 + 32u * i < E) s[e0 + 32u * i] = v[i];
        }
        __syncwarp();
        float sum = 0.0f;  // ascending serial sum (the declared order), every lane alike
#pragma unroll 1
        for (u32 e = 0; e + 32 <= E; e += 32) {  // 32 values asked for at once: an addition is four clocks, a read thirty
            float4 v[8];
#pragma unroll
            for (u32 i = 0; i < 8; ++i) v[i] = *reinterpret_cast<const float4*>(s + e + 4u * i);
#pragma unroll
            for (u32 i = 0; i < 8; ++i) sum = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(sum, v[i].x), v[i].y), v[i].z), v[i].w);
        }
        for (u32 e = E & ~31u; e < E; ++e) sum = __fadd_rn(sum, s[e]);
        __syncwarp();
#pragma unroll 1
        for (u32 e0 = lane; e0 < E; e0 += 128)
#pragma unroll
            for (u32 i = 0; i < 4; ++i) if (e0 + 32u * i < E) s[e0 + 32u * i] = __fdiv_rn(s[e0 + 32u * i], sum);
    } else {
#pragma unroll 1
        for (u32 e0 = lane; e0 < E; e0 += 128) {
            float v[4];
#pragma unroll
            for (u32 i = 0; i < 4; ++i) v[i] = e0 + 32u * i < E ? s[e0 + 32u * i] : 0.0f;
            if (p.score == B200MOE_SCORE_SIGMOID) {
#pragma unroll
                for (u32 i = 0; i < 4; ++i) v[i] = sigmoid_score(v[i]);
            } else {
#pragma unroll
                for (u32 i = 0; i < 4; ++i) v[i] = sqrt_softplus_score(v[i]);
            }
#pragma unroll
            for (u32 i = 0; i < 4; ++i) if (e0 + 32u * i < E) s[e0 + 32u * i] = v[i];
        }
    }
    u32 key[EPL];  // a lane reads the scores that it wrote itself
    bool bad = false;
#pragma unroll
    for (int j = 0; j < EPL; ++j) {
        const u32 e = lane + 32u * j;
        float c = 0.0f;
        if (e < E) c = p.selection_bias ? __fadd_rn(s[e], bias[e]) : s[e];
        bad |= c != c;
        key[j] = e < E ? ordered_key(c) : 0u;
    }
    if (__any_sync(0xffffffffu, bad)) return false;
    if (p.n_group > 1) {
        u32 b0 = 0, b1 = 0;  // lane g: the two best of group g
        const u32 runs = per >> 5, shift = 31u - __clz(per);
        if (runs) {
            u32 g = 0, i = 0;
#pragma unroll
            for (int j = 0; j < EPL; ++j) {
                const u32 m0 = __reduce_max_sync(0xffffffffu, key[j]);
                const u32 first = __ffs(__ballot_sync(0xffffffffu, key[j] == m0)) - 1u;
                const u32 m1 = __reduce_max_sync(0xffffffffu, lane == first ? 0u : key[j]);
                if (lane == g) { b1 = max(min(b0, m0), max(b1, m1)); b0 = max(b0, m0); }
                if (++i == runs) { i = 0; ++g; }
            }
        } else {
#pragma unroll
            for (int j = 0; j < EPL; ++j) {
                u32 t0 = key[j], t1 = 0;
#pragma unroll 1
                for (u32 d = per >> 1; d; d >>= 1) {
                    const u32 o0 = __shfl_xor_sync(0xffffffffu, t0, d), o1 = __shfl_xor_sync(0xffffffffu, t1, d);
                    t1 = max(min(t0, o0), max(t1, o1));
                    t0 = max(t0, o0);
                }
                const u32 at = lane << shift, g0 = __shfl_sync(0xffffffffu, t0, at & 31u), g1 = __shfl_sync(0xffffffffu, t1, at & 31u);
                if ((at >> 5) == (u32)j) { b0 = g0; b1 = g1; }
            }
        }
        const bool mine = lane < p.n_group;
        const float score = mine ? __fadd_rn(key_value(b0), key_value(b1)) : 0.0f;
        if (__any_sync(0xffffffffu, score != score)) return false;
        u32 gkey = mine ? ordered_key(score) : 0u, gmask = 0;
#pragma unroll 1
        for (u32 k = 0; k < p.topk_group; ++k) {
            const u32 best = __reduce_max_sync(0xffffffffu, gkey), at = __ffs(__ballot_sync(0xffffffffu, gkey == best)) - 1u;
            gmask |= 1u << at;
            if (lane == at) gkey = 0u;
        }
        u32 g = 0, i = 0;
#pragma unroll
        for (int j = 0; j < EPL; ++j) {
            const u32 group = runs ? g : (lane + 32u * j) >> shift;
            if (!((gmask >> (group & 31u)) & 1u)) key[j] = 0u;
            if (++i == runs) { i = 0; ++g; }
        }
    }
    if (scores_out) for (u32 e = lane; e < E; e += 32) scores_out[u64(row) * E + e] = s[e];
    __syncwarp();
    u32 my_id = kNone;
#pragma unroll 1
    for (u32 k = 0; k < p.top_k; ++k) {
        u32 top = 0;
#pragma unroll
        for (int j = 0; j < EPL; ++j) top = max(top, key[j]);
        const u32 best = __reduce_max_sync(0xffffffffu, top);
        u32 id = kNone;
#pragma unroll
        for (int j = EPL - 1; j >= 0; --j) if (key[j] == best) id = lane + 32u * j;
        id = best ? __reduce_min_sync(0xffffffffu, id) : kNone;
#pragma unroll
        for (int j = 0; j < EPL; ++j) if (lane + 32u * j == id) key[j] = 0u;
        if (lane == k) my_id = id;
    }
    *picked = my_id;
    return true;
}

// Output order, weights and the stores of one row; lane k holds pick k in `my_id`, s[] the scores. Returns the lane's id in output order.
__device__ __forceinline__ u32 finish_row(const b200moe_route_policy& p, u32 row, u32 lane, const float* s, u32 my_id,
                                        u32* ids, float* weights) {
    if (p.order == B200MOE_ORDER_ASCENDING_ID) {  // rank sort of the (distinct) ids held one per lane
        u32 rank = 0;
        for (u32 k = 0; k < p.top_k; ++k) { const u32 o = __shfl_sync(0xffffffffu, my_id, k); rank += (o < my_id) ? 1u : 0u; }
        u32 sorted = kNone;
        for (u32 k = 0; k < p.top_k; ++k) {
            const u32 o = __shfl_sync(0xffffffffu, my_id, k), orank = __shfl_sync(0xffffffffu, rank, k);
            if (orank == lane) sorted = o;
        }
        my_id = sorted;
    }
    const float my_s = (lane < p.top_k && my_id != kNone) ? s[my_id] : 0.0f;
    float sum = 0.0f;  // ((0 + s0) + s1) + ... in output order (route_policy.hpp:121-123)
#pragma unroll 1
    for (u32 k0 = 0; k0 < p.top_k; k0 += 8) {  // eight values asked for at once
        float v[8];
#pragma unroll
        for (u32 i = 0; i < 8; ++i) v[i] = __shfl_sync(0xffffffffu, my_s, k0 + i);
#pragma unroll
        for (u32 i = 0; i < 8; ++i) sum = k0 + i < p.top_k ? __fadd_rn(sum, v[i]) : sum;
    }
    const bool renorm = p.renormalize && (p.top_k > 1 || p.renorm_single);
    const float den = __fadd_rn(sum, p.renorm_eps);
    if (lane < p.top_k) {
        ids[u64(row) * p.top_k + lane] = my_id;
        weights[u64(row) * p.top_k + lane] = __fmul_rn(renorm ? __fdiv_rn(my_s, den) : my_s, p.scale);
    }
    return my_id;
}

// One warp selects one row; select_row returns lane k's id in output order (lanes from top_k on: nothing of meaning). `s` points to this warp's scratch of 2 * experts + 32 floats on
// a 16-byte boundary (shared memory).
__host__ __device__ constexpr u32 scratch_floats(u32 experts) { return (2u * experts + 32u + 3u) & ~3u; }
// The general path of a row: any groups, any values (the serial rules where a NaN is among the choices). Returns lane k's pick k.
__device__ __forceinline__ u32 select_row_general(const float* logits, float* scores_out, const float* bias, const b200moe_route_policy& p, u32 row, u32 lane, float* s) {
    const u32 E = p.experts;
    float* c = s + E;
    float* gs = c + E;
    const float* z = logits + u64(row) * E;

    if (p.score == B200MOE_SCORE_SOFTMAX) {  // route_policy.hpp:135-144
        float m = -__uint_as_float(0x7f800000u);
        for (u32 e = lane; e < E; e += 32) { const float v = z[e]; m = v > m ? v : m; }
#pragma unroll
        for (int d = 16; d; d >>= 1) { const float o = __shfl_xor_sync(0xffffffffu, m, d); m = o > m ? o : m; }
        for (u32 e = lane; e < E; e += 32) s[e] = declared_exp(__fsub_rn(z[e], m));
        __syncwarp();
        float sum = 0.0f;
#pragma unroll 8
        for (u32 e = 0; e < E; ++e) sum = __fadd_rn(sum, s[e]);  // ascending serial sum (the declared order), every lane alike
        for (u32 e = lane; e < E; e += 32) s[e] = __fdiv_rn(s[e], sum);
    } else if (p.score == B200MOE_SCORE_SIGMOID) {
        for (u32 e = lane; e < E; e += 32) s[e] = sigmoid_score(z[e]);
    } else {
        for (u32 e = lane; e < E; e += 32) s[e] = sqrt_softplus_score(z[e]);
    }
    for (u32 e = lane; e < E; e += 32) c[e] = p.selection_bias ? __fadd_rn(s[e], bias[e]) : s[e];
    __syncwarp();
    if (scores_out) for (u32 e = lane; e < E; e += 32) scores_out[u64(row) * E + e] = s[e];

    u32 allowed = 0xffffffffu, per = E;
    if (p.n_group > 1) {  // group-limited extension (include/b200moe.h): group score = its two best choices summed
        per = E / p.n_group;
        if (lane < p.n_group) {
            const float* cg = c + lane * per;
            const u32 i0 = serial_pick(p.key, cg, per, kNone);
            const u32 i1 = serial_pick(p.key, cg, per, i0);
            const float b0 = cg[i0], b1 = cg[i1];
            gs[lane] = __fadd_rn(b0, b1);
        }
        __syncwarp();
        u32 gtaken = 0;
        allowed = 0;
        for (u32 k = 0; k < p.topk_group; ++k) {
            const u32 g = k_pass(p.key, gs, p.n_group, lane, gtaken, 0xffffffffu, p.n_group);
            if (g != kNone) allowed |= 1u << g;
        }
    }

    u32 taken = 0, my_id = kNone;
    for (u32 k = 0; k < p.top_k; ++k) {
        const u32 pick = k_pass(p.key, c, E, lane, taken, allowed, per);
        if (lane == k) my_id = pick;
    }
    return my_id;
}

// The same out of line, for a kernel that runs once a call on cold instruction caches, where every jump over code that is not run costs 500 to 1,000 clocks.
static __device__ __noinline__ u32 select_row_apart(const float* logits, float* scores_out, const float* bias, const b200moe_route_policy& p, u32 row, u32 lane, float* s) {
    return select_row_general(logits, scores_out, bias, p, row, lane, s);
}

// Whether a policy's groups let rows take the fast path: all experts one group, runs of 2^i lanes or whole runs of 32.
__host__ __device__ __forceinline__ bool fast_groups(const b200moe_route_policy& p) {
    const u32 run = p.experts / p.n_group;
    return p.n_group == 1 || run % 32 == 0 || (run < 32 && (run & (run - 1u)) == 0);
}

// EPL: a lane's experts on the fast path; 32 EPL is the most that the calling kernel sees. 0: the general path alone, in line.
template <int EPL>
__device__ __forceinline__ u32 select_row(const float* logits, float* scores_out, const float* bias,
                                          const b200moe_route_policy& p, u32 row, u32 lane, float* s,
                                          u32* ids, float* weights) {
    u32 my_id = kNone;
    if constexpr (EPL == 0) {
        my_id = select_row_general(logits, scores_out, bias, p, row, lane, s);
    } else if (!(fast_groups(p) && select_row_fast<EPL>(logits, scores_out, bias, p, row, lane, s, &my_id))) {  // the fast path unless a NaN needs the serial rule
        __syncwarp();
        my_id = select_row_apart(logits, scores_out, bias, p, row, lane, s);
    }
    return finish_row(p, row, lane, s, my_id, ids, weights);
}


}  // namespace select_detail
}  // namespace b200moe
