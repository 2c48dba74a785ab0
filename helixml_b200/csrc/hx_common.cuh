// Shared helpers of the helix_b200 CUDA library: error reporting, dtype access, fast math.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <cstdarg>
#include <cstdio>

#include "../../include/helix_b200.h"

namespace hx {

// Records a printf-style message for the calling thread and returns `st`.
hx_status fail(hx_status st, const char *fmt, ...);

inline hx_status cuda_fail(cudaError_t e, const char *what) {
    return fail(HX_ERR_BACKEND, "%s: %s", what, cudaGetErrorString(e));
}

#define HX_CUDA(call)                                              \
    do {                                                           \
        cudaError_t e__ = (call);                                  \
        if (e__ != cudaSuccess) return hx::cuda_fail(e__, #call);  \
    } while (0)

#define HX_REQUIRE(cond, st, ...)                       \
    do {                                                \
        if (!(cond)) return hx::fail(st, __VA_ARGS__);  \
    } while (0)

// Checks the launch that was just made.
inline hx_status check_launch(const char *kernel) {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fail(HX_ERR_BACKEND, "launch of %s failed: %s", kernel, cudaGetErrorString(e));
    return HX_OK;
}

inline size_t dtype_size(int dt) { return dt == HX_F32 ? 4 : dt == HX_BF16 ? 2 : 1; }

// Number of SMs of the current device, cached per device.
int sm_count();

// Device memory for the tensors the module layer makes and drops on every call (results, workspaces, uploaded inputs).
// cudaMalloc and cudaFree cost 0.1 to several ms each and cudaFree waits for the whole device; a freed block is kept
// here instead and handed to the next request of about its size.  Both calls may come from any thread.  A block may
// only be returned when everything that touches it was queued on the legacy default stream (stream order is what
// keeps the next owner's work behind it).  At most kPoolCachedBytes per device stay cached; what goes beyond that and
// everything on an allocation failure is given back with cudaFree.
constexpr size_t kPoolCachedBytes = (size_t)512 << 20;
hx_status pool_alloc(void **dptr, size_t bytes);
void pool_release(void *dptr, int device);   // back to the cache; `device` is where it was allocated
void pool_discard(void *dptr, int device);   // a real cudaFree (waits for the device)
void pool_trim(int device);                  // gives every cached block of the device back

// resid[i] += x[i] (x fp32 or bf16): the residual update where no GEMM epilogue can do it.
hx_status residual_add(float *resid, const void *x, int x_dtype, int64_t n, cudaStream_t st);

// The kernel HX_SCAN_AUTO picks for a d_state == 16 problem on the current device (selective_scan.cu); the Mamba
// block plans its launches and its workspace with the same rule.
namespace scan {
enum class ScanKind { Tiled, Direct, LookBack };
ScanKind auto_kind(const hx_scan_args *a);
int auto_channels_per_lane(const hx_scan_args *a);  // 1 or 2: what the one-lane-per-channel kernel would run with
hx_status launch_wide(const hx_scan_args *a, cudaStream_t st);  // any d_state and alignment (scan_wide.cu); a validated
}  // namespace scan

// Translation units with bounded device-side waits keep a status word each; these read (and
// optionally clear) them.  hx_device_status() ORs them together.
hx_status read_status_scan(int *v, bool clear);
hx_status read_status_gemm(int *v, bool clear);
hx_status read_status_convx(int *v, bool clear);

// ---------------------------------------------------------------- chained launches
// A decode step is about a hundred dependent kernels of a few microseconds.  Launched with `chain` set, a kernel starts
// while its predecessor in the stream still runs, as soon as every CTA of that one has called chain_trigger(); before
// chain_wait() returns it may touch nothing but constants (weights), and chain_wait() returns when the predecessor has
// completed.  Every kernel of a chain therefore triggers first, fetches its weights, waits (in every thread) and goes on:
// set-up and weight fetch of a kernel run under the one before it.  Launched without `chain`, both calls do nothing.
__device__ __forceinline__ void chain_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <typename... P, typename... V>
inline cudaError_t launch_chained(bool chain, void (*kernel)(P...), dim3 grid, dim3 block, cudaStream_t st, V... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.stream = st;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = chain ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// hx_mamba_block_step; `chained`: the kernel queued before this call on `stream` is part of the same decode step, so
// nothing that writes a weight can still be running when the first kernel starts early (decode.cu).
hx_status mamba_block_step(const hx_mamba_step_args *a, bool chained, void *stream);

// ---------------------------------------------------------------- device-side helpers
template <typename T> __device__ __forceinline__ float ld_f32(const T *p);
template <> __device__ __forceinline__ float ld_f32<float>(const float *p) { return *p; }
template <> __device__ __forceinline__ float ld_f32<__nv_bfloat16>(const __nv_bfloat16 *p) { return __bfloat162float(*p); }

template <typename T> __device__ __forceinline__ void st_f32(T *p, float v);
template <> __device__ __forceinline__ void st_f32<float>(float *p, float v) { *p = v; }
template <> __device__ __forceinline__ void st_f32<__nv_bfloat16>(__nv_bfloat16 *p, float v) { *p = __float2bfloat16_rn(v); }

constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;

__device__ __forceinline__ float ex2_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float lg2_approx(float x) {
    float y;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float rcp_approx(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// x / (1 + exp(-x)) with one ex2 and one rcp on the special-function unit.
__device__ __forceinline__ float silu_fast(float x) {
    return x * rcp_approx(1.0f + ex2_approx(-kLog2e * x));
}
// The same through tanh: x sigmoid(x) = h + h tanh(h), h = x / 2.  One special-function result instead of two;
// tanh.approx is good to about 2^-11 relative, which is below the rounding of a bf16 result.
__device__ __forceinline__ float silu_tanh(float x) {
    const float h = 0.5f * x;
    float t;
    asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(h));
    return fmaf(h, t, h);
}
// Accurate forms used by the parity-baseline kernels.
__device__ __forceinline__ float silu_acc(float x) { return x / (1.0f + expf(-x)); }
__device__ __forceinline__ float softplus_acc(float v) { return v > 20.0f ? v : logf(1.0f + expf(v)); }

}  // namespace hx
