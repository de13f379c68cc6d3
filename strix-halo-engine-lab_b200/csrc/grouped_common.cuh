// Pieces shared by the grouped forms (grouped_q4k.cu, grouped_q8.cu): packed FP32, asynchronous copies, and the tiles of a window - an
// expert, up to GN of its entries, one of its row tiles - that a persistent grid walks round-robin.
#pragma once
#include "q4k_row.cuh"

namespace b200moe {
namespace grouped {

constexpr u32 kMaxUnion = 1024;

// Two FP32 lanes per instruction (Blackwell packed FP32): each lane is one IEEE round-to-nearest operation, the same result
// as two scalar instructions at half the issue slots. A packed add fed by a packed multiply did not reproduce the scalar
// bits on B200 (it behaves as contracted), so a product is written as a * b + 0: one rounding, of a * b (a product of -0 comes
// out as +0, which no sum of a chain that starts at +0 tells apart).
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
    float2 c;
    asm("{\n\t.reg .b64 z;\n\tmov.b64 z, 0;\n\tfma.rn.f32x2 %0, %1, %2, z;\n\t}" : "=l"(reinterpret_cast<u64&>(c)) : "l"(reinterpret_cast<const u64&>(a)), "l"(reinterpret_cast<const u64&>(b)));
    return c;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    float2 c;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(reinterpret_cast<u64&>(c)) : "l"(reinterpret_cast<const u64&>(a)), "l"(reinterpret_cast<const u64&>(b)));
    return c;
}
__device__ __forceinline__ float2 both(float v) { return make_float2(v, v); }
__device__ __forceinline__ float2 to_float(int2 v) { return make_float2(static_cast<float>(v.x), static_cast<float>(v.y)); }
__device__ __forceinline__ float2 pick(bool c, float2 x, float2 y) { return make_float2(c ? x.x : y.x, c ? x.y : y.y); }

// Shared memory by explicit 32-bit addresses.
__device__ __forceinline__ u32 lds32(u32 a) { u32 v; asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a)); return v; }
__device__ __forceinline__ uint2 lds64(u32 a) { uint2 v; asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a)); return v; }

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(q4k::saddr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async4(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(q4k::saddr(dst)), "l"(src) : "memory");
}

// Bounds of a launch's waits: polls (a microsecond's hint each, about four in fact), and the stage before which a CTA's producers stop asking for copies (test hook).
struct Waits { u32 limit, stall_stage; };
inline Waits debug_waits() {
    const u32 limit = debug_value(B200MOE_DEBUG_WAIT_LIMIT), stall = debug_value(B200MOE_DEBUG_STALL_STAGE);
    return Waits{limit ? limit : 1u << 20, stall ? stall - 1u : 0xffffffffu};
}
// Waits (bounded) until the copies of the last `asked` stages have landed: a CTA must not retire before them. One thread calls it.
__device__ __forceinline__ void drain(u64* full, u32 stages, u32 asked, u32 limit) {
    for (u32 n = asked > stages ? asked - stages : 0u; n < asked; ++n)
        for (u32 i = 0; i < (limit >> 4) + 64u; ++i)
            if (q4k::mbar_try_wait(&full[n % stages], (n / stages) & 1u, q4k::kWaitHintNs)) break;
}

struct Tile { u32 expert, eb, nt, c, tt; };

// Token tiles of an expert with n entries, GN entries each. SHORT_LAST: but for a last one of at most GN / 2, which is cheaper (half of the MMAs).
template <u32 GN, bool SHORT_LAST>
__device__ __forceinline__ u32 whole_tiles(u32 n) { return (n + (SHORT_LAST ? GN / 2 : GN) - 1) / GN; }

// cum[j]: whole token tiles of the first j experts of the union; cum[kTileCounts + j]: their short last ones (n_union + 1 words each). Every thread of the
// block calls it. Returns the token tiles of the window.
constexpr u32 kTileCounts = kMaxUnion + 1;
template <u32 GN, bool SHORT_LAST>
__device__ __forceinline__ u32 count_tiles(const b200moe_routes& routes, u32 n_union, u32* cum) {
    const u32 tid = threadIdx.x, lane = tid & 31u;
    for (u32 j = tid; j < n_union; j += blockDim.x) {
        const u32 n = routes.begins[j + 1] - routes.begins[j], whole = whole_tiles<GN, SHORT_LAST>(n);
        cum[j + 1] = whole;
        cum[kTileCounts + j + 1] = n > GN * whole ? 1u : 0u;
    }
    if (tid < 2) cum[kTileCounts * tid] = 0;
    __syncthreads();
    if (tid < 64) {  // inclusive scans, 32 at a time
        u32* c = cum + kTileCounts * (tid >> 5);
        u32 carry = 0;
        for (u32 j0 = 0; j0 < n_union; j0 += 32) {
            u32 v = j0 + lane < n_union ? c[j0 + lane + 1] : 0u;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) { const u32 o = __shfl_up_sync(0xffffffffu, v, d); if (lane >= (u32)d) v += o; }
            if (j0 + lane < n_union) c[j0 + lane + 1] = carry + v;
            carry += __shfl_sync(0xffffffffu, v, 31);
        }
    }
    __syncthreads();
    return cum[n_union] + cum[kTileCounts + n_union];
}

// Tile id -> (union expert, token tile, row tile): row tiles fastest, then the expert's token tiles, experts ascending. SHORT_LAST: the whole token tiles of all
// experts first, then the short ones. The CTAs walk the ids round-robin, so each then gets as many of either sort as any other, or one more; in one row of
// experts their shares of the short ones are a matter of chance. Q8_0, 64 experts of 2048 -> 1024, 512 and 2048 rows of top 4: 327 -> 320 and 939 -> 932 us a
// call. Not for Q4_K, whose short tiles cost nearly what whole ones do and find the weights in L2 behind these: 128 experts of 2048 -> 768, 512 and 4096
// rows of top 8: 332 -> 337 and 1807 -> 1817.
template <u32 GN, bool SHORT_LAST>
__device__ __forceinline__ Tile find_tile(const b200moe_routes& routes, u32 n_row_tiles, const u32* cum, u32 n_union, u32 id) {
    u32 q = id / n_row_tiles;
    Tile t;
    t.c = id - q * n_row_tiles;
    const u32 n_whole = cum[n_union];
    const bool whole = !SHORT_LAST || q < n_whole;
    if (!whole) { q -= n_whole; cum += kTileCounts; }
    u32 lo = 0, hi = n_union;  // largest j with cum[j] <= q
    while (hi - lo > 1) {
        const u32 mid = (lo + hi) >> 1;
        if (cum[mid] <= q) lo = mid; else hi = mid;
    }
    t.expert = routes.experts[lo];
    const u32 b0 = routes.begins[lo], b1 = routes.begins[lo + 1];
    t.tt = whole ? q - cum[lo] : whole_tiles<GN, SHORT_LAST>(b1 - b0);
    t.eb = b0 + GN * t.tt;
    t.nt = min(GN, b1 - t.eb);
    return t;
}

}  // namespace grouped
}  // namespace b200moe
