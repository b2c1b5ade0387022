// Shared helpers for the sm_100a decode-path kernels: status/error plumbing, storage-dtype
// conversions and small warp utilities.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <cstdarg>
#include <cstdio>

#include "../../include/mynn_b200.h"
#include "smem_limit.h"

namespace mynn {

// ---- host-side status ----------------------------------------------------------------------
void set_error(const char *fmt, ...);
extern std::atomic<long long> g_launches;

inline int fail(int code, const char *fmt, ...) __attribute__((format(printf, 2, 3)));
inline int fail(int code, const char *fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    set_error("%s", buf);
    return code;
}

#define MYNN_CUDA_OK(expr)                                                                                 \
    do {                                                                                                   \
        cudaError_t e__ = (expr);                                                                          \
        if (e__ != cudaSuccess)                                                                            \
            return mynn::fail(MYNN_E_CUDA, "%s failed: %s (%s:%d)", #expr, cudaGetErrorString(e__), __FILE__, \
                              __LINE__);                                                                   \
    } while (0)

// Call after every kernel launch: counts it and turns a launch error into a status code.
#define MYNN_LAUNCH_OK(name)                                                                          \
    do {                                                                                              \
        mynn::g_launches.fetch_add(1, std::memory_order_relaxed);                                     \
        cudaError_t e__ = cudaGetLastError();                                                         \
        if (e__ != cudaSuccess)                                                                       \
            return mynn::fail(MYNN_E_CUDA, "launch of %s failed: %s", name, cudaGetErrorString(e__)); \
    } while (0)

inline size_t dtype_size(int dt) { return dt == MYNN_F32 ? 4 : 2; }
inline bool dtype_ok(int dt) { return dt == MYNN_F32 || dt == MYNN_BF16 || dt == MYNN_F16; }

// ---- device-side storage conversions ---------------------------------------------------------
template <typename T>
__device__ __forceinline__ float to_f32(T v);
template <>
__device__ __forceinline__ float to_f32<float>(float v) { return v; }
template <>
__device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <>
__device__ __forceinline__ float to_f32<__half>(__half v) { return __half2float(v); }

template <typename T>
__device__ __forceinline__ T from_f32(float v);
template <>
__device__ __forceinline__ float from_f32<float>(float v) { return v; }
template <>
__device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }
template <>
__device__ __forceinline__ __half from_f32<__half>(float v) { return __float2half_rn(v); }

// One RoPE pair (xl, xh = the elements half a head apart) with the roundings of the engine's CPU kernel: two products and
// one sum, each rounded to f32, never contracted into a fused multiply-add.  Every kernel that rotates what it stores uses these, so the
// stand-alone RoPE kernel and the rotation inside the decode attention kernel give the same bits.
__device__ __forceinline__ float rope_low(float xl, float xh, float c, float s) { return __fsub_rn(__fmul_rn(xl, c), __fmul_rn(xh, s)); }
__device__ __forceinline__ float rope_high(float xl, float xh, float c, float s) { return __fadd_rn(__fmul_rn(xh, c), __fmul_rn(xl, s)); }
// The exception: the 16-bit keys of a streaming cache, which are rotated anew at each step, by a kernel of their own or on their way into the product, with
// the first product not rounded.  An element against its partner half a head away.
__device__ __forceinline__ float rope_cached(float x, float partner, float c, float s, bool low) { return __fmaf_rn(x, c, low ? -__fmul_rn(partner, s) : __fmul_rn(partner, s)); }

// One store point: round to storage dtype and come back to f32.
template <typename T>
__device__ __forceinline__ float round_store(float v) { return to_f32<T>(from_f32<T>(v)); }

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// ---- programmatic dependent launch -----------------------------------------------------------------------------
// Most kernels of a step are launched with the programmatic-stream-serialization attribute (launch_dependent): they may become resident
// while the kernel in front still runs.  A dependent writes nothing before pdl_wait(), and before it reads only what no kernel since the last
// full barrier on its stream (a copy, a synchronisation) writes.  A model's step begins with the copy of its inputs, so its weights,
// positions and the state that earlier steps left may be read early; an operator's caller may have made any operand with the kernel right in
// front, so the operators read nothing early: each early read stands behind a flag that only a model's step sets (settled,
// fixed_weights).  A prefetch into L2 is no read.  What the kernel in front triggers, and when, makes no difference to this.
// pdl_wait() returns when the grid in front has completed and is visible; since the kernels of a chain wait, that covers all before it.  The
// one that does not, tp_reduce_norm_limbs_kernel, polls for each word it takes from the grid in front.
// pdl_trigger() says when the next kernel may become resident: at the start where this kernel leaves room beside it (lean products leave eight SMs, where whole tiles of rows ask for it four, to the row kernels), when the
// accumulators are complete in the tcgen05 products (step of batch 32: 3.98 -> 3.85 ms; a trigger at their start made the kernels two and three
// places ahead take registers and shared memory from the running one, 4.63 -> 5.31 ms), when its own loads are here in the norms of few rows.
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void prefetch_l2(const void *p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Library options (mynn_b200_set_option).
extern int g_ksplit_override;            // forced cluster K split of the DequantMatMul kernels, 0 = automatic
extern int g_prefill_attention_mode;     // see MYNN_OPT_PREFILL_ATTENTION
extern int g_fuse_rope;                  // see MYNN_OPT_FUSE_ROPE
extern int g_decode_ring;                // see MYNN_OPT_DECODE_RING
extern std::atomic<int> g_inject_stall;  // see MYNN_OPT_INJECT_STALL; consumed by the next launch it applies to

// A launch in clusters of `cluster` CTAs along x (1: none).  dependent: it may begin while the kernel in front of it drains; what the kernel may
// do before its pdl_wait stands above.  Else everything in front has completed when it starts.
template <typename... KArgs, typename... Args>
inline cudaError_t launch_ex(bool dependent, unsigned cluster, void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args... args) {
    cudaLaunchAttribute attr[2];
    unsigned n = 0;
    if (dependent) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (cluster > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = cluster;
        attr[n].val.clusterDim.y = 1;
        attr[n++].val.clusterDim.z = 1;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = n;
    return cudaLaunchKernelEx(&cfg, kern, static_cast<KArgs>(args)...);
}
template <typename... KArgs, typename... Args>
inline cudaError_t launch_plain(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args... args) {
    return launch_ex(false, 1, kern, grid, block, smem, st, args...);
}
template <typename... KArgs, typename... Args>
inline cudaError_t launch_dependent(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args... args) {
    return launch_ex(true, 1, kern, grid, block, smem, st, args...);
}

// Dispatch a launcher template over the three storage dtypes.
#define MYNN_DISPATCH_DTYPE(dt, T, ...)                       \
    switch (dt) {                                             \
        case MYNN_F32: { using T = float; __VA_ARGS__; } break;          \
        case MYNN_BF16: { using T = __nv_bfloat16; __VA_ARGS__; } break; \
        case MYNN_F16: { using T = __half; __VA_ARGS__; } break;         \
        default: return mynn::fail(MYNN_E_ARG, "bad dtype %d", dt);      \
    }

}  // namespace mynn
