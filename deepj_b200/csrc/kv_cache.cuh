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
    static __device__ __forceinline__ void st4(float* p, const float4& v) { *reinterpret_cast<float4*>(p) = v; }
    // 16 bytes of a row
    static __device__ __forceinline__ void ld_piece(const float* p, float* v) {
        const float4 a = *reinterpret_cast<const float4*>(p);
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    }
    static __device__ __forceinline__ void st_piece(float* p, const float* v) { *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]); }
    static __device__ __forceinline__ void st2(float* p, float a, float b) { *reinterpret_cast<float2*>(p) = make_float2(a, b); }
};

template <> struct KvIo<__half> {
    static __device__ __forceinline__ float stored(float x) { return __half2float(__float2half_rn(x)); }
    static __device__ __forceinline__ float4 ld4(const __half* p) {
        const uint2 u = __ldg(reinterpret_cast<const uint2*>(p));
        const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&u.x)), b = __half22float2(*reinterpret_cast<const __half2*>(&u.y));
        return make_float4(a.x, a.y, b.x, b.y);
    }
    static __device__ __forceinline__ void ld_piece(const __half* p, float* v) {
        const uint4 u = *reinterpret_cast<const uint4*>(p);
        const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&w[j]));
            v[2 * j] = a.x; v[2 * j + 1] = a.y;
        }
    }
    static __device__ __forceinline__ void st_piece(__half* p, const float* v) {
        uint32_t w[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const __half2 h = __floats2half2_rn(v[2 * j], v[2 * j + 1]);
            w[j] = *reinterpret_cast<const uint32_t*>(&h);
        }
        *reinterpret_cast<uint4*>(p) = make_uint4(w[0], w[1], w[2], w[3]);
    }
    static __device__ __forceinline__ void st4(__half* p, const float4& v) {
        st2(p, v.x, v.y);
        st2(p + 2, v.z, v.w);
    }
    static __device__ __forceinline__ void st2(__half* p, float a, float b) { *reinterpret_cast<__half2*>(p) = __floats2half2_rn(a, b); }
};

}  // namespace dj
