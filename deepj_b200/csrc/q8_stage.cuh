// Activation staging of the Q8 GEMV: fp32 values → three int8 digit columns + one power-of-two scale per 32-k block.
#pragma once
#include "q8_common.cuh"

namespace dj {

constexpr int kGemvWarps = 8;
constexpr int kGemvThreads = kGemvWarps * 32;
constexpr int kGemvXsPad = 32;              // bytes of padding per activation digit column
constexpr int kGemvColsPerRow = 3;          // digit columns per activation row in shared memory: d2, d1, d0

// Four consecutive values of a 32-k block (eight lanes share one) → digit columns and block scale, in the order of the int8 MMA's B
// fragment, so that lane t fetches both of its registers (k = 4t … 4t+3 and k = 16+4t … 16+4t+3) with one 8-byte load at
// offset 8t: value k of a block sits at 8·((k mod 16)/4) + 4·(k/16) + k mod 4.  `to` is the place of the lane's values in the first column.
// With a gain the digits are those of x·γ, and the caller multiplies the finished sums by 1/rms
// (Σ_k w_k·(x_k·γ_k)/rms = Σ_k w_k·(x_k/rms·γ_k)); ss collects Σx².
__device__ __forceinline__ void gemv_digits4(const float4& x, const float4& gain, bool gained, float& ss, int8_t* to, int ldxs, bool first, float* xsc) {
    float v[4] = {x.x, x.y, x.z, x.w};
    ss = fmaf(v[0], v[0], ss); ss = fmaf(v[1], v[1], ss); ss = fmaf(v[2], v[2], ss); ss = fmaf(v[3], v[3], ss);
    if (gained) { v[0] *= gain.x; v[1] *= gain.y; v[2] *= gain.z; v[3] *= gain.w; }
    float amax = fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3])));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 4));
    // as digits16: s = 2^(exponent(amax)+2), q = rne(v·2^23/s); at least the s whose 2^23/s is the largest power of two (with a gain x·γ is taken
    // before the norm, and a block below 2^-106 would meet an infinite factor)
    int sbits = 0x3f800000;
    if (amax > 0.0f && amax < 1e36f) sbits = max(__float_as_int(amax) & 0x7f800000, 21 << 23) + 0x01000000;
    const float mul = __int_as_float(0x7f000000 - sbits) * 8388608.0f;
    uint32_t u[4];
#pragma unroll
    for (int e = 0; e < 4; e++) u[e] = (uint32_t)(__float2int_rn(v[e] * mul) + 0x808080);
    const uint32_t t0 = __byte_perm(u[0], u[1], 0x5140), t1 = __byte_perm(u[2], u[3], 0x5140);
    const uint32_t t2 = __byte_perm(u[0], u[1], 0x7362), t3 = __byte_perm(u[2], u[3], 0x7362);
    *reinterpret_cast<uint32_t*>(to) = __byte_perm(t2, t3, 0x5410) ^ 0x80808080u;
    *reinterpret_cast<uint32_t*>(to + ldxs) = __byte_perm(t0, t1, 0x7632) ^ 0x80808080u;
    *reinterpret_cast<uint32_t*>(to + 2 * ldxs) = __byte_perm(t0, t1, 0x5410) ^ 0x80808080u;
    if (first) *xsc = __int_as_float(sbits) * (1.0f / 8388608.0f);
}

}  // namespace dj
