// Element access of the K/V cache for the attention kernels.  The cache holds fp32 (the reference's precision) or,
// as an option, fp16: keys are rotated in fp32 and rounded to nearest-even when they are appended, values are rounded
// when they are appended, and every kernel widens what it reads back to fp32 — scores, softmax and the weighted
// sum are accumulated in fp32 either way.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>

namespace dj {

template <typename T> struct KvIo;

template <> struct KvIo<float> {
    // the value a later step will read back for x (fp32 cache: x itself)
    static __device__ __forceinline__ float stored(float x) { return x; }
    static __device__ __forceinline__ float4 ld4(const float* p) { return __ldg(reinterpret_cast<const float4*>(p)); }
    static __device__ __forceinline__ float4 ld4_shared(const float* p) { return *reinterpret_cast<const float4*>(p); }
    static __device__ __forceinline__ void st4(float* p, const float4& v) { *reinterpret_cast<float4*>(p) = v; }
    static __device__ __forceinline__ void st2(float* p, float a, float b) { *reinterpret_cast<float2*>(p) = make_float2(a, b); }
};

template <> struct KvIo<__half> {
    static __device__ __forceinline__ float stored(float x) { return __half2float(__float2half_rn(x)); }
    static __device__ __forceinline__ float4 ld4(const __half* p) {
        const uint2 u = __ldg(reinterpret_cast<const uint2*>(p));
        const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&u.x)), b = __half22float2(*reinterpret_cast<const __half2*>(&u.y));
        return make_float4(a.x, a.y, b.x, b.y);
    }
    static __device__ __forceinline__ float4 ld4_shared(const __half* p) {
        const uint2 u = *reinterpret_cast<const uint2*>(p);
        const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&u.x)), b = __half22float2(*reinterpret_cast<const __half2*>(&u.y));
        return make_float4(a.x, a.y, b.x, b.y);
    }
    static __device__ __forceinline__ void st4(__half* p, const float4& v) {
        st2(p, v.x, v.y);
        st2(p + 2, v.z, v.w);
    }
    static __device__ __forceinline__ void st2(__half* p, float a, float b) { *reinterpret_cast<__half2*>(p) = __floats2half2_rn(a, b); }
};

}  // namespace dj
