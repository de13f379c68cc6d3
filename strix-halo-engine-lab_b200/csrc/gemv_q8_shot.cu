// Routed experts and dense blocks, Q8_0 in the 32-lane-class contract (src/ds41_formats.cpp:45-50), for windows of fewer rows than the tensor-core forms
// take, and for sparse ones of more: a CTA is ONE item and asks for all of its weights at once.
//
// Item = (expert, 64 weight rows): 32 gate and 32 up rows of one output group, or 64 down rows. A stage = a run of 32 blocks (1088 bytes) of the 64 rows, two
// tiled TMA copies of 32 rows each; as many stages as the rows have runs, up to kStages (the places are used again beyond that). Consumer warps (16) take
// four rows each, a lane one of the 32 classes, as in gemv_q8.cu, whose bits these are; the entries' codes are read once for a warp's four rows.
// What bounds it: latencies. One row over 4 of 64 experts of 2048 -> 1024, top 4 (128 + 128 items): the form with a row a warp had one run a warp on its
// way (35 KB a multiprocessor) and each warp's four runs one behind the other: gate/up 11.5 us behind its routes, down 9.7 behind gate/up, where these
// take 8 and 5 (a whole call 33.1 -> 24.9). Where it pays: csrc/api.cu.
// An early launch of down (ChainHints) has its first weights before it waits where it fits on the multiprocessors beside gate/up's CTAs: with one entry a pass (62 and
// 57 registers, 512 threads each) and rows of up to 2048 and 1024 weights (139 and 70 KB); else as those CTAs end.
#include <algorithm>

#include "declared_math.cuh"
#include "grouped_common.cuh"
#include "wide_common.cuh"

namespace b200moe {
namespace {
using namespace q4k;  // the mbarrier / copy wrappers

constexpr u32 kRunBlocks = 32, kRunBytes = kRunBlocks * kQ8Block, kHalf = 32;  // 1088 bytes, rows of a copy
constexpr u32 kStageBytes = 2 * kHalf * kRunBytes, kStages = 3;
constexpr u32 kWarps = 16, kRowsWarp = 64 / kWarps, kThreads = kWarps * 32;
constexpr u32 kMaxEntries = 8;
constexpr u32 kWaitPolls = 1u << 18;  // about a second

struct ShotArgs {
    b200moe_routes routes;
    b200moe_a8_rows in, act;
    float* gate_out;
    float* up_out;
    float* raw;
    u32* summary;
    float limit;
    u32 K, runs, stages, cap;   // weights and runs of a row; stages in shared memory; entries that a pass holds
    u32 rows_per_expert, out_width;
    u32 early;                  // routes and weights are complete before the launch in front was admitted (ChainHints)
    u32 bounded;                // the routes' arrays hold an expert for every CTA
    u32 wait_limit, stall_stage;  // test hook: run `stall_stage` of a CTA's runs and those behind it are not asked for
};

template <bool DOWN, int NR>
__device__ __forceinline__ void shot_run(const unsigned char* st, u32 nb, u32 g0, u32 warp, u32 lane, const i8* codes, const float* deltas, u32 K, u32 nr, float (&cls)[kRowsWarp][NR]) {
    if (lane >= nb) return;
    const u32 g = g0 + lane;
    u32 q[kRowsWarp][8];
    float scale[kRowsWarp];
#pragma unroll
    for (u32 i = 0; i < kRowsWarp; ++i) {
        // block at byte 34 * lane of its run: even lanes start on a word, odd lanes on a halfword
        const u32* w = reinterpret_cast<const u32*>(st + (kRowsWarp * warp + i) * kRunBytes) + ((kQ8Block * lane) >> 2);
        u32 v[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) v[k] = w[k];
        const bool odd = lane & 1u;
        scale[i] = half_bits_to_float(odd ? v[0] >> 16 : v[0] & 0xffffu);
#pragma unroll
        for (int k = 0; k < 8; ++k) q[i][k] = odd ? v[k + 1] : __funnelshift_r(v[k], v[k + 1], 16);
    }
#pragma unroll
    for (int r = 0; r < NR; ++r) {
        if (r < (int)nr) {
            const uint4* c = reinterpret_cast<const uint4*>(codes + u32(r) * K + 32u * g);
            const uint4 c0 = c[0], c1 = c[1];
            const float d = deltas[u32(r) * (K / 32) + g];
#pragma unroll
            for (u32 i = 0; i < kRowsWarp; ++i) {
                int a = __dp4a((int)q[i][0], (int)c0.x, 0), b = __dp4a((int)q[i][4], (int)c1.x, 0);
                a = __dp4a((int)q[i][1], (int)c0.y, a); b = __dp4a((int)q[i][5], (int)c1.y, b);
                a = __dp4a((int)q[i][2], (int)c0.z, a); b = __dp4a((int)q[i][6], (int)c1.z, b);
                a = __dp4a((int)q[i][3], (int)c0.w, a); b = __dp4a((int)q[i][7], (int)c1.w, b);
                cls[i][r] = __fadd_rn(cls[i][r], __fmul_rn(static_cast<float>(a + b), __fmul_rn(scale[i], d)));
            }
        }
    }
}

// grid (items of an expert, union); NR: entries of a pass at most (1, 2, 4 or 8).
template <bool DOWN, int NR>
__global__ void __launch_bounds__(kThreads) q8_shot_kernel(const __grid_constant__ CUtensorMap tm0, const __grid_constant__ CUtensorMap tm1, ShotArgs a) {
    extern __shared__ __align__(128) unsigned char smem[];
    unsigned char* s_a8 = smem + a.stages * kStageBytes;
    i8* s_codes = reinterpret_cast<i8*>(s_a8);                                 // [cap][K]
    float* s_deltas = reinterpret_cast<float*>(s_a8 + a.cap * a.K);            // [cap][K / 32]
    __shared__ u64 full[kStages];
    __shared__ float s_gu[2][kMaxEntries][32];
    __shared__ u32 s_abort;
    const u32 tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u, j = blockIdx.y, chunk = blockIdx.x;
    if (tid == 0) {
        for (u32 i = 0; i < kStages; ++i) mbar_init(&full[i], 1);
        s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (!a.early) chain_begin();
    const u32 n_union = load_l2(a.routes.counts);
    u32 expert = 0, eb = 0, ee = 0;
    if (a.bounded || j < n_union) { expert = load_l2(a.routes.experts + j); eb = load_l2(a.routes.begins + j); ee = load_l2(a.routes.begins + j + 1); }
    if (j >= n_union) {
        if (a.early) chain_begin();
        return;
    }
    const u32 y = expert * a.rows_per_expert + (DOWN ? 2 * kHalf : kHalf) * chunk;
    auto ask = [&](u32 n) {  // one thread: run n % runs into place n % stages
        const u32 x = (n % a.runs) * (kRunBytes / 8);  // 64-bit elements: whole multiples of 1088 bytes
        u64* bar = &full[n % a.stages];
        unsigned char* st = smem + (n % a.stages) * kStageBytes;
        mbar_expect_tx(bar, kStageBytes);  // whole boxes: what lies past the row is filled
        tma_2d(st, &tm0, x, y, bar);
        tma_2d(st + kHalf * kRunBytes, DOWN ? &tm0 : &tm1, x, DOWN ? y + kHalf : y, bar);
    };
    const u32 passes = (ee - eb + a.cap - 1) / a.cap, total = passes * a.runs;  // an expert of more entries than a pass holds has its rows brought in again
    u32 asked = min(min(total, a.stages), a.stall_stage);
    if (tid == 0) for (u32 n = 0; n < asked; ++n) ask(n);
    if (a.early) chain_begin();
    auto drain = [&](u32 from) {  // one thread: the copies asked for land (the wait is bounded) before the CTA retires
        for (u32 n = from; n < asked; ++n)
            for (u32 i = 0; i < (a.wait_limit >> 4) + 64u; ++i)
                if (mbar_try_wait(&full[n % a.stages], (n / a.stages) & 1u, kWaitHintNs)) break;
    };
    // An aborted projection skips the stage: one answer for the block, at the barrier that its first entries' rows are waited for at. A barrier for it alone took 0.2 us of a one-row call.
    const u32 skips = DOWN && a.summary ? *a.summary : 0u;
    const u32 in_stride = a.in.stride ? a.in.stride : a.in.width, groups = a.K / 32;
    bool ok = true;
    u32 n = 0, landed = 0;  // the run in hand; the runs that have been seen to land
    for (u32 p0 = eb; p0 < ee; p0 += a.cap) {
        const u32 nr = min(a.cap, ee - p0);
        const u32 my_slot = lane < nr ? load(a.routes.slots + p0 + lane) : 0u;
        const u32 my_row = DOWN || lane >= nr ? my_slot : load(a.routes.rows + p0 + lane);
        if (p0 != eb) __syncthreads();  // the previous pass has read the entries' rows and the outputs
        for (u32 r = 0; r < nr; ++r) {
            const u32 row = __shfl_sync(0xffffffffu, my_row, r);
            const i8* c = a.in.codes + u64(row) * in_stride;
            for (u32 i = tid; i < a.K / 16; i += kThreads) grouped::cp_async16(s_codes + r * a.K + 16u * i, c + 16u * i);
            const float* d = a.in.deltas + u64(row) * (in_stride / 32);
            for (u32 i = tid; i < groups; i += kThreads) grouped::cp_async4(s_deltas + r * groups + i, d + i);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        if (__syncthreads_or(p0 == eb && skips != 0u)) {
            if (tid == 0) drain(0);
            return;
        }
        float cls[kRowsWarp][NR];
#pragma unroll
        for (u32 i = 0; i < kRowsWarp; ++i)
#pragma unroll
            for (int r = 0; r < NR; ++r) cls[i][r] = 0.0f;
        for (u32 run = 0; run < a.runs; ++run, ++n) {
            // A warp whose wait ran out does no more work, but meets the barriers of the others: the block leaves as one.
            if (ok) ok = __all_sync(0xffffffffu, mbar_wait(&full[n % a.stages], (n / a.stages) & 1u, a.wait_limit, &s_abort));
            if (ok) {
                shot_run<DOWN, NR>(smem + (n % a.stages) * kStageBytes, min(kRunBlocks, groups - run * kRunBlocks), run * kRunBlocks, warp, lane, s_codes, s_deltas, a.K, nr, cls);
                landed = n + 1u;
            }
            if (n + a.stages < total) {  // uniform over the block
                if (__syncthreads_or(!ok)) { ok = false; break; }  // the place has been read
                if (n + a.stages < a.stall_stage) {
                    if (tid == 0) {
                        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                        ask(n + a.stages);
                    }
                    ++asked;
                }
            }
        }
        if (__syncthreads_or(!ok)) { ok = false; break; }
#pragma unroll
        for (int r = 0; r < NR; ++r) {
            if (r < (int)nr) {
                const u32 slot = __shfl_sync(0xffffffffu, my_slot, r);
#pragma unroll
                for (u32 i = 0; i < kRowsWarp; ++i) {
                    const float v = butterfly32(cls[i][r]);
                    const u32 row = kRowsWarp * warp + i;
                    if (lane == 0) {
                        if (DOWN) a.raw[u64(slot) * a.out_width + 2 * kHalf * chunk + row] = v;
                        else s_gu[row >> 5][r][row & 31u] = v;
                    }
                }
            }
        }
        if (!DOWN) {
            __syncthreads();
            if (warp < nr) {  // swiglu_clamped + the A8 rule over the 32 outputs of an entry (src/ds41_moe.cpp:134-146)
                const float gv = s_gu[0][warp][lane], uv = s_gu[1][warp][lane];
                const u32 slot = __shfl_sync(0xffffffffu, my_slot, warp), o = 32u * chunk + lane;
                if (a.gate_out) { a.gate_out[u64(slot) * a.out_width + o] = gv; a.up_out[u64(slot) * a.out_width + o] = uv; }
                const float h = swiglu_ds41(gv, uv, a.limit);  // NaN propagates: this family has no status rule
                float delta;
                int sum;
                const int code = a8_quantize_lane(h, &delta, &sum);
                const u32 act_stride = a.act.stride ? a.act.stride : a.act.width;
                a.act.codes[u64(slot) * act_stride + o] = static_cast<i8>(code);
                if (lane == 0) {
                    a.act.deltas[u64(slot) * (act_stride / 32) + chunk] = delta;
                    if (a.act.sums) a.act.sums[u64(slot) * (act_stride / 32) + chunk] = sum;
                }
            }
        }
    }
    if (!ok) {
        if (tid == 0) {
            drain(landed);
            if (a.summary) atomicOr(a.summary, kAbortBit);
        }
    }
}

struct ShotPlan { u32 runs, stages, cap, smem; };
// K: the row length; rows: the window's (an expert has no more entries).
bool shot_plan(u32 K, u32 rows, ShotPlan* p) {
    if (K == 0 || K % 256 || rows == 0) return false;
    p->runs = (K / 32 + kRunBlocks - 1) / kRunBlocks;
    for (p->cap = std::min(kMaxEntries, rows);; p->cap = (p->cap + 1) / 2) {
        for (p->stages = std::min(p->runs, kStages); p->stages >= 1; --p->stages) {
            p->smem = p->stages * kStageBytes + p->cap * (K + K / 8);
            if (p->smem <= 224u * 1024u && (p->stages >= 2 || p->runs == 1)) return true;
        }
        if (p->cap == 1) return false;
    }
}

void set_waits(ShotArgs* a) {
    const u32 limit = debug_value(B200MOE_DEBUG_WAIT_LIMIT), stall = debug_value(B200MOE_DEBUG_STALL_STAGE);
    a->wait_limit = limit ? limit : kWaitPolls;
    a->stall_stage = stall ? stall - 1u : 0xffffffffu;
}

template <bool DOWN>
int launch_shot(const ShotPlan& p, dim3 grid, const CUtensorMap& tm0, const CUtensorMap& tm1, const ShotArgs& a, cudaStream_t stream) {
    const auto kernel = p.cap == 1 ? q8_shot_kernel<DOWN, 1> : p.cap == 2 ? q8_shot_kernel<DOWN, 2> : p.cap <= 4 ? q8_shot_kernel<DOWN, 4> : q8_shot_kernel<DOWN, 8>;
    if (int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), p.smem)) return rc;
    chain_launch(kernel, grid, kThreads, p.smem, stream, tm0, tm1, a);
    return after_launch(DOWN ? "down_q8_shot" : "gate_up_q8_shot");
}

}  // namespace

bool q8_shot_gate_up_fits(const b200moe_gate_up_view& v, u32 rows) {
    ShotPlan p{};
    return v.shape.gate_type == B200MOE_TYPE_Q8_0 && v.shape.inter % 32 == 0 && aligned(v.weights.gate, 16) && aligned(v.weights.up, 16) && aligned(v.x.codes, 16) &&
           (v.x.stride ? v.x.stride : v.x.width) % 16 == 0 && v.max_union <= 65535u && shot_plan(v.shape.hidden, rows, &p);
}
bool q8_shot_down_fits(const b200moe_down_view& v, u32 rows) {
    ShotPlan p{};
    return v.shape.down_type == B200MOE_TYPE_Q8_0 && v.shape.hidden % 64 == 0 && aligned(v.weights.down, 16) && aligned(v.act.codes, 16) &&
           (v.act.stride ? v.act.stride : v.act.width) % 16 == 0 && v.max_union <= 65535u && shot_plan(v.shape.inter, rows, &p);
}

int launch_gate_up_q8_shot(const b200moe_gate_up_view& v, u32 rows, const ChainHints& hints, cudaStream_t stream) {
    if (v.max_union == 0) return B200MOE_OK;
    ShotPlan p{};
    if (!shot_plan(v.shape.hidden, rows, &p)) return fail(B200MOE_ERR_UNSUPPORTED, "gate_up: the one-item form does not apply to this shape");
    ShotArgs a{};
    a.routes = v.routes; a.in = v.x; a.act = v.act; a.gate_out = v.gate_out; a.up_out = v.up_out; a.summary = v.summary; a.limit = v.shape.limit;
    a.K = v.shape.hidden; a.runs = p.runs; a.stages = p.stages; a.cap = p.cap; a.rows_per_expert = v.shape.inter; a.out_width = v.shape.inter;
    a.bounded = hints.slots >= v.max_union;
    set_waits(&a);
    CUtensorMap tm0, tm1;
    const u64 rb = u64(a.K / 32) * kQ8Block, total = u64(v.shape.experts) * v.shape.inter;
    if (int rc = wide::rows_map(v.weights.gate, rb, total, kRunBytes, kHalf, &tm0)) return rc;
    if (int rc = wide::rows_map(v.weights.up, rb, total, kRunBytes, kHalf, &tm1)) return rc;
    return launch_shot<false>(p, dim3(v.shape.inter / 32, v.max_union), tm0, tm1, a, stream);
}

int launch_down_q8_shot(const b200moe_down_view& v, u32 rows, const ChainHints& hints, cudaStream_t stream) {
    if (v.max_union == 0) return B200MOE_OK;
    ShotPlan p{};
    if (!shot_plan(v.shape.inter, rows, &p)) return fail(B200MOE_ERR_UNSUPPORTED, "down: the one-item form does not apply to this shape");
    ShotArgs a{};
    a.routes = v.routes; a.in = v.act; a.raw = v.raw; a.summary = const_cast<u32*>(v.summary);
    a.K = v.shape.inter; a.runs = p.runs; a.stages = p.stages; a.cap = p.cap; a.rows_per_expert = v.shape.hidden; a.out_width = v.shape.hidden;
    a.early = hints.routes_done; a.bounded = hints.slots >= v.max_union;
    set_waits(&a);
    CUtensorMap tm0;
    if (int rc = wide::rows_map(v.weights.down, u64(a.K / 32) * kQ8Block, u64(v.shape.experts) * v.shape.hidden, kRunBytes, kHalf, &tm0)) return rc;
    return launch_shot<true>(p, dim3(v.shape.hidden / 64, v.max_union), tm0, tm0, a, stream);
}

}  // namespace b200moe
