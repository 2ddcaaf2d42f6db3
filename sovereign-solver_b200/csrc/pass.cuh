// pass.cuh -- how the passes of an iteration follow one another
// (kernels_fast.cu, kernels_exact.cu).
#pragma once

#include <cuda_runtime.h>

#include "engine.cuh"

namespace pdhg {
namespace {

// The passes of an iteration are launched as programmatic dependents
// (launch_pass): pass_begin lets the next pass's CTAs start as soon as this
// pass's have all started, pass_wait waits until the pass before is complete
// and its writes are visible. Between the two a kernel touches only what no
// pass writes: the matrix, the bounds, and the control state, which the check
// and restart kernels write (launched in full order). That part of a pass, its
// launch and two or three dependent loads, is most of a small pass's 4 us.
__device__ __forceinline__ void pass_begin() { cudaTriggerProgrammaticLaunchCompletion(); }
__device__ __forceinline__ void pass_wait() { cudaGridDependencySynchronize(); }

// Loads of what the pass before wrote. EARLY kernels (launched as programmatic
// dependents): ordinary, coherent loads, which the wait covers -- a
// non-coherent one may hit a line that a pass still running beside this
// kernel's start brought into L1 -- and volatile, so that none moves above the
// wait. The others gather through the non-coherent path, whose loads the
// compiler may move across stores: on a pass bound by HBM that is worth more
// than the early start (the 10M-column transportation LP's primal: 55.7 us
// non-coherent, 60.2 us coherent).
__device__ __forceinline__ float coherent_ld(const float* p) {
    float v;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ double coherent_ld(const double* p) {
    double v;
    asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ float4 coherent_ld(const float4* p) {
    float4 v;
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ double2 coherent_ld(const double2* p) {
    double2 v;
    asm volatile("ld.global.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
    return v;
}
template <bool EARLY, class V>
__device__ __forceinline__ V gather_ld(const V* p) {
    if constexpr (EARLY) return coherent_ld(p);
    else return __ldg(p);
}

// Launches one pass (smem: dynamic shared memory). early: the launch may begin
// while the kernel before it in the stream still runs (programmatic dependent
// launch); only after a kernel that begins with pass_begin, and with no other
// predecessor.
template <class... P, class... Q>
cudaError_t launch_pass_smem(void (*kernel)(P...), int grid, bool early, cudaStream_t s, size_t smem,
                             const Q&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(grid));
    cfg.blockDim = dim3(kBlock);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = early ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}
template <class... P, class... Q>
cudaError_t launch_pass(void (*kernel)(P...), int grid, bool early, cudaStream_t s, const Q&... args) {
    return launch_pass_smem(kernel, grid, early, s, 0, args...);
}

}  // namespace
}  // namespace pdhg
