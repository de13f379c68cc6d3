// Internal launch interface between the C ABI layer (api.cu) and the kernel translation units. Every function
// validates nothing (api.cu has done it), enqueues on `stream` and returns after_launch()'s status.
#pragma once
#include "common.cuh"

namespace b200moe {

// What a caller that composes the launches of a layer knows about those in front of one. routes_done: the routes were complete before the launch in
// front was admitted (chain_begin), so they and the weights may be read before the wait. dense_rows: the launch belongs to a dense block of so many
// rows (entry i is row i and slot i of the only expert), whose weights were complete before the launch in front was admitted. slots: the routes'
// arrays hold so many entries, whatever the union is (0: not known).
struct ChainHints { bool routes_done; u32 dense_rows; u64 slots; };

// a8.cu
// wide (optional, only with bfloat16 x and quantize_a8_vec_ok): the values as FP32 rows of wide_stride, 16-byte aligned
bool quantize_a8_vec_ok(const b200moe_quantize_a8_view& v);
int launch_quantize_a8(const b200moe_quantize_a8_view& v, cudaStream_t stream, float* wide = nullptr, u32 wide_stride = 0);
int launch_rmsnorm_a8(const b200moe_rmsnorm_view& v, cudaStream_t stream);
// out[i] = float(bfloat16 bits in[i]) (exact widening)
int launch_widen_bf16(const u16* in, float* out, u64 count, cudaStream_t stream);

// router.cu
// fused_quantize (optional): the A8 quantiser of the same activations is enqueued first
int launch_router_logits(const b200moe_router_view& v, cudaStream_t stream, const b200moe_quantize_a8_view* fused_quantize = nullptr);
int launch_router_select(const b200moe_router_view& v, cudaStream_t stream);

// routes.cu
u64 routes_scratch_words(u32 rows, u32 top_k, u32 experts);
// what the first launch of a call that owns its status words clears on the way (each may be null): rows, 4 and 1 words
struct RoutesClear { u32* row_status; u32* summary4; u32* summary; };
int launch_routes(const b200moe_routes_view& v, const RoutesClear& clear, cudaStream_t stream);
// zero (optional): count floats cleared on the way
int launch_dense_routes(const b200moe_routes& out, u32 rows, u32* row_status, u32* summary4, float* zero, u64 count, cudaStream_t stream);
// grouped (token-block) form of the Q4_K experts on the tensor cores (grouped_q4k.cu)
bool grouped_gate_up_fits(const b200moe_gate_up_view& v);
bool grouped_down_fits(const b200moe_down_view& v);
u32 grouped_row_tiles(u32 outputs, bool down);  // of an expert
int launch_gate_up_q4k_grouped(const b200moe_gate_up_view& v, cudaStream_t stream);
int launch_down_q4k_grouped(const b200moe_down_view& v, cudaStream_t stream);
// decode windows: selection of r (logits already present) and the routes of the selected ids in one launch
bool select_routes_fusable(const b200moe_router_view& r, u32 top_k);
int launch_select_routes(const b200moe_router_view& r, const b200moe_routes_view& v, const RoutesClear& clear, cudaStream_t stream);

// gemv_q8.cu: Q8_0 x A8 products in the 32-lane-class contract (dense rows and the routed DS41-family experts)
int launch_q8_0_a8(const b200moe_q8a8_view& v, cudaStream_t stream);
int launch_gate_up_q8(const b200moe_gate_up_view& v, cudaStream_t stream);
int launch_down_q8(const b200moe_down_view& v, const ChainHints& hints, cudaStream_t stream);

// gemv_q4k.cu: Q4_K x A8 rows in the four-chain contract (routed Qwen-family experts; Q8_0 four-chain down)
int launch_gate_up_q4k(const b200moe_gate_up_view& v, cudaStream_t stream);
int launch_down_q4k(const b200moe_down_view& v, cudaStream_t stream);
// gemv_ds41_any.cu: the DS41 family over any of its block types (Q8_0, Q2_K), one weight row per warp, weights read in place.
int launch_gate_up_ds41_any(const b200moe_gate_up_view& v, cudaStream_t stream);
int launch_down_ds41_any(const b200moe_down_view& v, cudaStream_t stream);
int launch_down_q8_chain4(const b200moe_down_view& v, u32 rows, const ChainHints& hints, cudaStream_t stream);
u32 chain4_mma_chunks(const b200moe_down_view& v);  // items an expert makes in the form, 0 where it does not apply
int launch_down_chain4_mma(const b200moe_down_view& v, const ChainHints& hints, cudaStream_t stream);

// gemv_q4k_stream.cu: the same Q4_K contracts as persistent kernels fed by bulk copies (decode windows up to 64 rows)
bool stream_gate_up_fits(const b200moe_gate_up_view& v, u32 rows);
bool stream_down_fits(const b200moe_down_view& v, u32 rows);
int launch_gate_up_q4k_stream(const b200moe_gate_up_view& v, u32 rows, cudaStream_t stream);
int launch_down_q4k_stream(const b200moe_down_view& v, u32 rows, cudaStream_t stream);

// gemv_q4k_wide.cu: the same contracts with SEGMENTS of the rows (and of the entries' A8 rows) streamed by TMA: any row
// length, windows of any size whose routes fit shared memory
bool wide_gate_up_fits(const b200moe_gate_up_view& v, u32 rows);
bool wide_down_fits(const b200moe_down_view& v, u32 rows);
int launch_gate_up_q4k_wide(const b200moe_gate_up_view& v, u32 rows, const ChainHints& hints, cudaStream_t stream);
int launch_down_q4k_wide(const b200moe_down_view& v, u32 rows, const ChainHints& hints, cudaStream_t stream);
// gemv_q8_shot.cu: the same contract, a CTA one item with all of its weights asked for at once (windows of a few rows)
bool q8_shot_gate_up_fits(const b200moe_gate_up_view& v, u32 rows);
bool q8_shot_down_fits(const b200moe_down_view& v, u32 rows);
int launch_gate_up_q8_shot(const b200moe_gate_up_view& v, u32 rows, const ChainHints& hints, cudaStream_t stream);
int launch_down_q8_shot(const b200moe_down_view& v, u32 rows, const ChainHints& hints, cudaStream_t stream);
// gemv_q8_wide.cu: the Q8_0 x A8 lane-class contract in the same streaming skeleton, for windows of many rows.
bool q8_wide_gate_up_fits(const b200moe_gate_up_view& v, u32 rows);
bool q8_wide_down_fits(const b200moe_down_view& v, u32 rows);
int launch_gate_up_q8_wide(const b200moe_gate_up_view& v, u32 rows, cudaStream_t stream);
int launch_down_q8_wide(const b200moe_down_view& v, u32 rows, cudaStream_t stream);
// gemv_q8_mma.cu: the same contract with the integer dots on the tensor cores (mma.sync s8 x s8), lane classes shared out over the warps.
bool q8_mma_gate_up_fits(const b200moe_gate_up_view& v, u32 rows);
bool q8_mma_down_fits(const b200moe_down_view& v, u32 rows);
int launch_gate_up_q8_mma(const b200moe_gate_up_view& v, u32 rows, cudaStream_t stream);
int launch_down_q8_mma(const b200moe_down_view& v, u32 rows, cudaStream_t stream);
// grouped_q8.cu: the same contract for experts with many entries, class sums in registers.
bool grouped_q8_gate_up_fits(const b200moe_gate_up_view& v);
bool grouped_q8_down_fits(const b200moe_down_view& v);
int launch_gate_up_q8_grouped(const b200moe_gate_up_view& v, cudaStream_t stream);
int launch_down_q8_grouped(const b200moe_down_view& v, cudaStream_t stream);
// value of a B200MOE_DEBUG_* hook (api.cu)
u32 debug_value(u32 key);
u32 experts_met(const b200moe_shape& s, u64 slots, u32 max_union);  // that have an entry, of the max_union that may, where the choice is spread evenly (api.cu)

// prologue.cu: A8 + router logits of a decode window (rows <= 8) in one launch; q.x / q.x_is_bf16 say where the activations are (r.x is not read)
bool prologue_fusable(const b200moe_router_view& r);
int launch_prologue(const b200moe_router_view& r, const b200moe_quantize_a8_view& q, cudaStream_t stream);

// combine.cu
int launch_merge_first_error(b200moe_first_error* record, const u32* summary, u32 domain, cudaStream_t stream);
// skip_bits: bits of the job summary with which no row is combined. zero_skipped: rows of y and y_bf16 that are left out become zeros
int launch_combine(const b200moe_combine_view& v, cudaStream_t stream, u32 skip_bits = B200MOE_JOB_WAIT_ABORTED, bool zero_skipped = false, const ChainHints& hints = {});
int launch_canonical_sum(const float* a, const float* b, const float* c, u64 count, float* y, cudaStream_t stream);
int launch_fill_u32(u32* p, u32 value, u64 count, cudaStream_t stream);
// order[row][k] (slots in ascending expert id) for the PARTS combine when no routes were built
int launch_row_order(const u32* ids, u32 rows, u32 top_k, u32* order, cudaStream_t stream);

}  // namespace b200moe
