// Shared host/device helpers of the B200 MoE FFN library.
//
// Every translation unit of the library is compiled with --fmad=false -prec-div=true -prec-sqrt=true -ftz=false: the
// arithmetic contracts are written as single IEEE-754 binary32 operations (the reference builds its exact kernels
// the same way, cmake/QwenCuda.cmake:49), so FP32 code written in the declared order gives the host reference's bits.
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <atomic>
#include <cstdarg>
#include <cstdint>
#include <cstdio>
#include <string>
#include <utility>

#include "../../include/b200moe.h"

namespace b200moe {

using u8 = std::uint8_t;
using u16 = std::uint16_t;
using u32 = std::uint32_t;
using u64 = std::uint64_t;
using i8 = std::int8_t;
using i32 = std::int32_t;

// ---- host: error text, launch accounting --------------------------------------------------------------------------
std::string& last_error_slot();
int fail(int code, const char* fmt, ...);
std::atomic<u64>& launch_counter();
// Checks the launch that was just enqueued; counts it. Returns B200MOE_OK or B200MOE_ERR_CUDA.
int after_launch(const char* what);
// True once a device with the sm_100a image is usable; otherwise records why and returns false.
bool device_ready();
// Raises a kernel's dynamic shared memory limit when `bytes` needs more than it has been given so far (per device).
int ensure_dynamic_smem(const void* kernel, u32 bytes);
// Asks for the largest shared-memory carve-out for a kernel that itself needs little (see api.cu).
int prefer_max_shared(const void* kernel);
// Multiprocessors of the current device (148 on a B200; queried, not assumed).
int device_sm_count();

inline cudaStream_t as_stream(void* s) { return static_cast<cudaStream_t>(s); }
inline bool aligned(const void* p, std::size_t a) { return (reinterpret_cast<std::uintptr_t>(p) % a) == 0; }

#define B200_REQUIRE(cond, ...)                                                  \
    do {                                                                         \
        if (!(cond)) return ::b200moe::fail(B200MOE_ERR_INVALID_ARGUMENT, __VA_ARGS__); \
    } while (0)

constexpr u32 kQ8Block = 34, kQ4KBlock = 144, kQ5KBlock = 176, kQ51Block = 24, kQ2KBlock = 84;
inline u64 row_bytes_of(u32 type, u32 width) {
    switch (type) {
        case B200MOE_TYPE_Q8_0: return u64(width / 32) * kQ8Block;
        case B200MOE_TYPE_Q5_1: return u64(width / 32) * kQ51Block;
        case B200MOE_TYPE_Q5_K: return u64(width / 256) * kQ5KBlock;
        case B200MOE_TYPE_Q2_K: return u64(width / 256) * kQ2KBlock;
        default: return u64(width / 256) * kQ4KBlock;
    }
}
// gate / up of the Qwen A8 family (K-quant super-blocks, four-chain pair rule); down types whose term reads the code sums
inline bool is_kquant(u32 type) { return type == B200MOE_TYPE_Q4_K || type == B200MOE_TYPE_Q5_K; }
// tensors of the DS41 family (32 lane classes + butterfly, declared_exp SwiGLU with the clamp)
inline bool is_ds41_type(u32 type) { return type == B200MOE_TYPE_Q8_0 || type == B200MOE_TYPE_Q2_K; }
inline bool down_reads_sums(u32 type) { return type == B200MOE_TYPE_Q4_K || type == B200MOE_TYPE_Q5_1; }

// ---- device helpers ------------------------------------------------------------------------------------------------
#if defined(__CUDACC__)
// ---- the chain of a call's launches ----------------------------------------------------------------------------------
// A call is a chain of dependent launches, most of them a few microseconds long. Each is enqueued with programmatic stream
// serialisation: it is brought onto the SMs while the launch before it still runs and waits there, in chain_begin, until
// that one has completed and its writes are visible. What every kernel launched so keeps to:
//  * Every CTA waits, on every path, and writes nothing to global memory before. A launch that has passed its wait knows that everything enqueued before it is
//    complete.
//  * It admits its successor only behind its own wait (chain_begin does both). So a launch that runs at all knows that what lies in front of the launch in
//    front is complete; one that admitted first would take that from every early reader behind it.
//  * Before its wait it reads only what it is told to be older than the launch in front (ChainHints: routes, order, weights, ids, expert tensors), past L1.
//  * Everything else it reads behind the wait, by plain loads (load below), never through the read-only path: the kernel runs already while its predecessor
//    writes, and such a load may be moved in front of the wait.
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_admit() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void chain_begin() {
    chain_wait();
    chain_admit();
}
template <class T>
__device__ __forceinline__ T load(const T* p) { return *p; }
// The same past the L1 cache, for what is known to be complete before the wait (ChainHints): the multiprocessor's L1 may hold lines of an earlier call.
__device__ __forceinline__ u32 load_l2(const u32* p) { return __ldcg(p); }
// Whether the block leaves a stage out because the job's summary says so: one answer for all of its threads (every one calls it; no barrier where there is no summary). Another block of the same
// launch may raise the word meanwhile, and threads that read it one by one could part: those that stay would wait at a barrier of counted warps for good.
__device__ __forceinline__ bool block_skips(const u32* summary) { return summary && __syncthreads_or(*summary != 0u) != 0; }
// Enqueues a kernel of the chain; its status is read by after_launch.
template <class... P, class... A>
inline void chain_launch_attrs(u32 extra, void (*kernel)(P...), dim3 grid, dim3 block, u32 smem, cudaStream_t stream, A&&... args) {
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributePreferredSharedMemoryCarveout;
    attr[1].val.sharedMemCarveout = cudaSharedmemCarveoutMaxL1;
    cudaLaunchConfig_t c{};
    c.gridDim = grid; c.blockDim = block; c.dynamicSmemBytes = smem; c.stream = stream; c.attrs = attr; c.numAttrs = 1 + extra;
    (void)cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);
}
template <class... P, class... A>
inline void chain_launch(void (*kernel)(P...), dim3 grid, dim3 block, u32 smem, cudaStream_t stream, A&&... args) {
    chain_launch_attrs(0, kernel, grid, block, smem, stream, std::forward<A>(args)...);
}
// The same for a kernel that reads its weights several times out of L1, of no more CTAs than multiprocessors: behind a launch that takes all shared memory it would run with the
// L1 that is left beside that. With several CTAs a multiprocessor the preference would cost their places.
template <class... P, class... A>
inline void chain_launch_l1(void (*kernel)(P...), dim3 grid, dim3 block, u32 smem, cudaStream_t stream, A&&... args) {
    chain_launch_attrs(u64(grid.x) * grid.y * grid.z <= static_cast<u64>(device_sm_count()) ? 1u : 0u, kernel, grid, block, smem, stream, std::forward<A>(args)...);
}
// Whether a launch of so many CTAs, several of which share a multiprocessor, is better a programmatic one. Such CTAs come onto the multiprocessors as the launch in
// front leaves them, so that what leaves first gets as many as it can hold and the others none: up to two a multiprocessor that does not matter, and the start
// that is saved does; above, the most loaded multiprocessor decides, and the chain's instructions cost every CTA (RMSNorm of 409 rows of 7168 22.9 us as a
// programmatic launch behind another, 18.5 as a plain one; of 741 rows of 4096 20.0 and 17.2).
inline bool chain_pays(u64 ctas) { return ctas <= 2u * static_cast<u64>(device_sm_count()); }
template <bool CHAIN>  // a kernel's instance for plain launches: all in front of it is complete, and it admits nothing early
__device__ __forceinline__ void chain_begin_if() { if (CHAIN) chain_begin(); }
// A plain launch of an instance without the chain's instructions; its status is read by after_launch.
template <class... P, class... A>
inline void plain_launch(void (*kernel)(P...), dim3 grid, dim3 block, u32 smem, cudaStream_t stream, A&&... args) {
    kernel<<<grid, block, smem, stream>>>(static_cast<P>(args)...);
}
// A launch that needs little shared memory: see prefer_max_shared (a preference that cannot be set is no error).
template <class... P, class... A>
inline void small_launch(void (*kernel)(P...), dim3 grid, dim3 block, u32 smem, cudaStream_t stream, A&&... args) {
    (void)prefer_max_shared(reinterpret_cast<const void*>(kernel));
    chain_launch(kernel, grid, block, smem, stream, std::forward<A>(args)...);
}
__device__ __forceinline__ float half_bits_to_float(u32 h) {  // exact for every fp16 value, subnormals included
    return __half2float(__ushort_as_half(static_cast<unsigned short>(h)));
}
__device__ __forceinline__ bool finite_f(float x) { return (__float_as_uint(x) & 0x7f800000u) != 0x7f800000u; }
// The largest of a warp's magnitudes; a NaN is left out, as std::max(amax, |x|) leaves it out, unless there is nothing else. The bits of
// magnitudes order as they do, so one reduction instruction does it.
__device__ __forceinline__ float warp_max_abs(float x) {
    const bool nan = x != x;
    const u32 m = __reduce_max_sync(0xffffffffu, nan ? 0u : __float_as_uint(x) & 0x7fffffffu);
    return __all_sync(0xffffffffu, nan) ? __uint_as_float(0x7fffffffu) : __uint_as_float(m);
}
__device__ __forceinline__ int warp_sum_i(int v) {
    return __reduce_add_sync(0xffffffffu, v);
}
// The declared butterfly: v[l] = v[l] + v[l ^ d], d = 16 .. 1 (src/core/integer_math.hpp:43-47). Addition is
// commutative bit for bit, so every lane ends with the tree's value.
__device__ __forceinline__ float butterfly32(float v) {
#pragma unroll
    for (int d = 16; d; d >>= 1) v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, d));
    return v;
}
// amax / 127 rounded once, by a product in double: that is 2^-52 from the quotient, which lies no closer than 2^-32 to a rounding boundary
// (magnitudes from 2^-119 on, whose quotients are normal).
__device__ __forceinline__ float over_127(float amax) { return static_cast<float>(static_cast<double>(amax) * (1.0 / 127.0)); }
// One A8 group of 32 values held one per lane (src/cpu/core/reference.cpp:35-55). Returns the code; delta and sum
// are the same in every lane. A group of NaNs alone gets a NaN for its delta, where the host rule gives 1 (codes of -127 in both).
__device__ __forceinline__ int a8_quantize_lane(float x, float* delta_out, int* sum_out) {
    const float amax = warp_max_abs(x);
    const bool tiny = amax > 0.0f && amax < 0x1p-119f;
    const float delta = (amax == 0.0f || tiny) ? 1.0f : __fdiv_rn(amax, 127.0f);
    const float r = tiny ? 0.0f : rintf(__fdiv_rn(x, delta));
    const float lo = (-127.0f < r) ? r : -127.0f;  // std::max(-127, r): a NaN quotient gives -127
    const float cl = (lo < 127.0f) ? lo : 127.0f;
    const int code = static_cast<int>(cl);
    *delta_out = delta;
    *sum_out = warp_sum_i(code);
    return code;
}
__device__ __forceinline__ u16 bf16_rne_bits(float v) {  // src/cuda/models/qwen/qwen_moe.cu:333-334
    const u32 b = __float_as_uint(v);
    return static_cast<u16>((b + 0x7fffu + ((b >> 16) & 1u)) >> 16);
}
#endif

}  // namespace b200moe
