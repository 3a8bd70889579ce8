// Shared helpers for the xg_sm100 kernel library: error reporting, dtype traits, 16-byte vectors.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <cstdarg>
#include <cstdio>

#include "../../include/xg_sm100.h"

namespace xg {

// Thread-local message buffer behind xg_last_error().
char* last_error_buf();
int fail(int code, const char* fmt, ...);

inline int check_launch(const char* what) {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fail(XG_ERR_LAUNCH, "%s: %s", what, cudaGetErrorString(e));
    return XG_OK;
}

// ---- launches ---------------------------------------------------------------------------------
// Kernels are launched with programmatic stream serialisation: the next kernel's CTAs may be placed, and set up their
// barriers and tensor memory, while this one drains. A kernel therefore calls pdl_wait() before its first access to global
// memory (it returns once the previous kernel has completed and its writes are visible) and pdl_trigger() once its own CTA
// holds all the resources it will ask for (tensor memory above all: a successor that took columns a CTA of this grid still
// needs would wait for a kernel that waits for it). Every kernel has to reach pdl_wait(), or its own successor would not be
// ordered behind its predecessor. What it saves on B200 is the set-up and launch latency between two kernels of a stream.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// for kernels without a set-up worth overlapping
__device__ __forceinline__ void pdl_sync() {
    pdl_trigger();
    pdl_wait();
}

struct LaunchOptions {
    unsigned cluster = 0;  // CTAs per thread-block cluster where the kernel does not fix it itself (one that does: early = false)
    // false: plain stream order. For grids below a full set of resident CTAs of which several fit one SM: placed early,
    // they pack onto the few SMs that the previous kernel leaves free and share them for good (a 128-CTA fp32 dense layer
    // at two CTAs per SM took 1.7 x as long behind a tensor-core kernel).
    bool early = true;
};
// Thread-block clusters keep plain stream order whatever the caller asks for. One that was placed early - eight CTAs that read
// each other's shared memory (gemm_fma_kernel), behind another launch of the same kernel - raised a misaligned-address error on
// B200. Reading has not shown a cause (what is excluded: see launch_fma), so the form is not used by any kernel.
constexpr bool placed_early(const LaunchOptions& o) { return o.early && o.cluster <= 1; }
static_assert(placed_early({}) && placed_early({.cluster = 1}) && !placed_early({.cluster = 2}) && !placed_early({.cluster = 8}), "clusters: stream order");
template <typename... P, typename... A>
void launch_with(const LaunchOptions& o, void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, const A&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    unsigned n = 0;
    if (placed_early(o)) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (o.cluster) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = o.cluster;
        attr[n].val.clusterDim.y = 1;
        attr[n++].val.clusterDim.z = 1;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    (void)cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);  // the caller's check_launch() picks up a failure
}
template <typename... P, typename... A>
void launch(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, const A&... args) {
    launch_with(LaunchOptions{}, kern, grid, block, smem, st, args...);
}

// Opt a kernel in to `bytes` of dynamic shared memory, once per device (`done`: one bit per device).
template <typename K>
bool reserve_smem(K kern, int bytes, std::atomic<uint64_t>& done) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return false;
    const uint64_t bit = 1ull << (dev & 63);
    if (done.load(std::memory_order_acquire) & bit) return true;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    done.fetch_or(bit, std::memory_order_release);
    return true;
}

inline int num_sms() {
    static thread_local int cached_dev = -1;
    static thread_local int cached = 148;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 148;
    if (dev != cached_dev) {
        int n = 0;
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && n > 0) cached = n;
        cached_dev = dev;
    }
    return cached;
}

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

inline int dtype_size(int dtype) { return dtype == XG_F32 ? 4 : ((dtype == XG_BF16 || dtype == XG_F16) ? 2 : 0); }

template <typename T>
struct Cvt;
template <>
struct Cvt<float> {
    static __device__ __forceinline__ float to_f(float v) { return v; }
    static __device__ __forceinline__ float from_f(float v) { return v; }
};
template <>
struct Cvt<__nv_bfloat16> {
    static __device__ __forceinline__ float to_f(__nv_bfloat16 v) { return __bfloat162float(v); }
    static __device__ __forceinline__ __nv_bfloat16 from_f(float v) { return __float2bfloat16_rn(v); }
};
template <>
struct Cvt<__half> {
    static __device__ __forceinline__ float to_f(__half v) { return __half2float(v); }
    static __device__ __forceinline__ __half from_f(float v) { return __float2half_rn(v); }
};

// GELU (erf form) for epilogues whose result is rounded to a 16-bit type: erfc from Abramowitz & Stegun 7.1.26
// (absolute error <= 1.5e-7, against a 16-bit rounding step of 2^-9 or 2^-11 relative), one reciprocal, one exp2 and
// five FMAs instead of erff's branches; for v < 0 the factor 1 + erf is the formula's erfc term itself, so the tail
// does not cancel. fp32 outputs keep erff.
__device__ __forceinline__ float gelu_erf_16bit(float v) {
    const float x = fabsf(v) * 0.70710678118654752f;
    const float t = __fdividef(1.0f, fmaf(0.3275911f, x, 1.0f));
    float poly = fmaf(1.061405429f, t, -1.453152027f);
    poly = fmaf(poly, t, 1.421413741f);
    poly = fmaf(poly, t, -0.284496736f);
    poly = fmaf(poly, t, 0.254829592f);
    const float e = poly * t * __expf(-x * x);  // erfc(|v| / sqrt(2))
    return 0.5f * v * (v >= 0.f ? 2.0f - e : e);
}

// 16-byte vector of T (4 floats or 8 half-precision values).
template <typename T>
struct alignas(16) Vec16 {
    static constexpr int N = 16 / sizeof(T);
    T v[N];
};

template <typename T>
__device__ __forceinline__ Vec16<T> ld16(const T* p) {
    Vec16<T> r;
    *reinterpret_cast<uint4*>(&r) = *reinterpret_cast<const uint4*>(p);
    return r;
}
// Streaming 16-byte load that does not allocate in L1 (data read exactly once).
template <typename T>
__device__ __forceinline__ Vec16<T> ld16_stream(const T* p) {
    Vec16<T> r;
    uint4 u;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(u.x), "=r"(u.y), "=r"(u.z), "=r"(u.w)
                 : "l"(p));
    *reinterpret_cast<uint4*>(&r) = u;
    return r;
}
template <typename T>
__device__ __forceinline__ void st16(T* p, const Vec16<T>& r) {
    *reinterpret_cast<uint4*>(p) = *reinterpret_cast<const uint4*>(&r);
}

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

}  // namespace xg
