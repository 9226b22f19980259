// Projections with bf16 weights: out = stage(x) · Wᵀ, W [N][Kp] bf16 row-major (Kp = K rounded up to 8, zero padded).
//
// The reference has no such weights (its Q8 format is this library's own as well); checkpoints that ship in bf16 keep
// their exact values this way.  Activations and accumulation are fp32 everywhere except in the many-row tensor-core
// form (bf16_gemm_tc.cu), which rounds the staged operand to bf16.
//
//   k_bf16_gemv       1-16 rows (bf16_gemv.cu)
//   k_bf16_gemm_f32   many rows, fp32 FMA arithmetic (models run in 32-bit)
//   k_bf16_block      block-diagonal: head h's outputs read head h's slice of the row
//   k_stage_rows      the staged operand of the many-row kernels, as fp32 or bf16 rows in the workspace
#include "row_operand.cuh"

#include <algorithm>
#include <set>

namespace dj {
namespace {

constexpr int kRowSmemMax = 200 * 1024;          // of a staged row

__device__ __forceinline__ float bf_lo(uint32_t u) { return __uint_as_float(u << 16); }
__device__ __forceinline__ float bf_hi(uint32_t u) { return __uint_as_float(u & 0xffff0000u); }

// Four values to a row of fp32 or bf16.
__device__ __forceinline__ void put4(float* o, const float4& v) { *reinterpret_cast<float4*>(o) = v; }
__device__ __forceinline__ void put4(__nv_bfloat16* o, const float4& v) {
    const __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
    *reinterpret_cast<uint2*>(o) = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
}

// One row per block: the staged operand as fp32 or bf16, for rows in 16-byte pieces.  A normed first segment of up to
// 1024 · CH columns stays in registers: one load round trip with its gain, gate and base beside it, the pieces' sums of squares
// meet in shared memory, one store per piece.  The rest is copied, four pieces of a thread in flight.  With a row map, row i of the output
// holds source row map[i] / div (zeros where map[i] < 0).  2048 rows: of 4096 (norm, sum) 27 µs on average through
// shared memory, 26 this way, of 11008 27 and 19 (512 threads instead of four pieces a thread: 29).
template <typename OutT, int CH>
__global__ void __launch_bounds__(256) k_stage_rows(const RowOperand a, const RowOperand b, int K1p, int Kp, const int* __restrict__ map, int div,
                                                    OutT* __restrict__ out) {
    __shared__ float s_ss[256 * CH], s_scale[kMaxNormGroups];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    auto ld4 = [](const float* p, int q) { return reinterpret_cast<const float4*>(p)[q]; };
    auto gated = [](const float4& v, const float4& g) {
        return make_float4(v.x * sigmoid_f(g.x), v.y * sigmoid_f(g.y), v.z * sigmoid_f(g.z), v.w * sigmoid_f(g.w));
    };
    pdl_wait();
    pdl_launch_dependents();
    int m = blockIdx.x;
    OutT* const o = out + (size_t)blockIdx.x * Kp;
    if (map != nullptr) {
        m = map[m];
        if (m < 0) {
            for (int k = tid; k < Kp; k += 256) o[k] = (OutT)0.0f;
            return;
        }
        m /= div;
    }
    auto copy = [&](const RowOperand& seg, OutT* to) {
        const float* x = seg.x + (size_t)m * seg.ldx;
        const float* g = seg.gate ? seg.gate + (size_t)m * seg.ldg : nullptr;
#pragma unroll 4
        for (int q = tid; q < seg.k / 4; q += 256) {
            float4 v = ld4(x, q);
            if (g) v = gated(v, ld4(g, q));
            put4(to + 4 * q, v);
        }
    };
    if (a.groups > 0) {
        const float* x = a.x + (size_t)m * a.ldx;
        const float* more = a.gate ? a.gate + (size_t)m * a.ldg : a.base ? a.base + (size_t)m * a.ldbase : nullptr;
        const int n4 = a.k / 4, len4 = n4 / a.groups;
        float4 v[CH], w[CH], e[CH];
#pragma unroll
        for (int i = 0; i < CH; i++) {
            const int q = tid + i * 256;
            v[i] = w[i] = e[i] = make_float4(0, 0, 0, 0);
            if (q < n4) { v[i] = ld4(x, q); w[i] = ld4(a.gamma, q); if (more) e[i] = ld4(more, q); }
        }
        if (b.k > 0) copy(b, o + K1p);           // its loads go out while the sums meet
#pragma unroll
        for (int i = 0; i < CH; i++) s_ss[tid + i * 256] = fmaf(v[i].w, v[i].w, fmaf(v[i].z, v[i].z, fmaf(v[i].y, v[i].y, v[i].x * v[i].x)));
        __syncthreads();
        if (a.groups == 1) {                     // every warp for itself
            float ss = 0.0f;
            for (int q = lane; q < n4; q += 32) ss += s_ss[q];
            for (int f = 16; f > 0; f >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, f);
            if (lane == 0) s_scale[warp] = 1.0f / sqrtf(ss / (float)a.k + a.eps);
            __syncwarp();
        } else {
            for (int g = warp; g < a.groups; g += 8) {
                float ss = 0.0f;
                for (int q = lane; q < len4; q += 32) ss += s_ss[g * len4 + q];
                for (int f = 16; f > 0; f >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, f);
                if (lane == 0) s_scale[g] = 1.0f / sqrtf(ss / (float)(4 * len4) + a.eps);
            }
            __syncthreads();
        }
#pragma unroll
        for (int i = 0; i < CH; i++) {
            const int q = tid + i * 256;
            if (q >= n4) break;
            const float s = s_scale[a.groups == 1 ? warp : q / len4];
            float4 y = make_float4((v[i].x * s) * w[i].x, (v[i].y * s) * w[i].y, (v[i].z * s) * w[i].z, (v[i].w * s) * w[i].w);
            if (a.base) {
                y = make_float4(fmaf(a.mult, y.x, e[i].x), fmaf(a.mult, y.y, e[i].y), fmaf(a.mult, y.z, e[i].z), fmaf(a.mult, y.w, e[i].w));
                if (a.sum) reinterpret_cast<float4*>(a.sum + (size_t)m * a.ldsum)[q] = y;
            }
            if (a.gate) y = gated(y, e[i]);
            put4(o + 4 * q, y);
        }
    } else {
        copy(a, o);
        if (b.k > 0) copy(b, o + K1p);
    }
    for (int k = a.k + tid; k < (b.k > 0 ? K1p : Kp); k += 256) o[k] = (OutT)0.0f;
    if (b.k > 0)
        for (int k = K1p + b.k + tid; k < Kp; k += 256) o[k] = (OutT)0.0f;
}

// The same for any alignment and length: through shared memory.  With a row map, row i of the output holds source row map[i] / div
// (zeros where map[i] < 0).
template <typename OutT>
__global__ void __launch_bounds__(256) k_stage_rows_any(const RowOperand a, const RowOperand b, int K1p, int Kp, const int* __restrict__ map, int div,
                                                    OutT* __restrict__ out) {
    extern __shared__ __align__(16) float xs[];
    __shared__ float scratch[kRowScratchMax];
    const RowScratch sc(scratch, kMaxNormGroups);
    pdl_wait();
    pdl_launch_dependents();
    int m = blockIdx.x;
    OutT* o = out + (size_t)blockIdx.x * Kp;
    if (map != nullptr) {
        m = map[m];
        if (m < 0) {
            for (int k = threadIdx.x; k < Kp; k += 256) o[k] = (OutT)0.0f;
            return;
        }
        m /= div;
    }
    stage_segment(a, m, sc, [&](int k) -> float& { return xs[k]; }, true);
    if (b.k > 0) {
        __syncthreads();
        stage_segment(b, m, sc, [&](int k) -> float& { return xs[K1p + k]; });
    }
    for (int k = a.k + (int)threadIdx.x; k < (b.k > 0 ? K1p : Kp); k += 256) xs[k] = 0.0f;
    if (b.k > 0)
        for (int k = K1p + b.k + (int)threadIdx.x; k < Kp; k += 256) xs[k] = 0.0f;
    __syncthreads();
    for (int k = (int)threadIdx.x * 2; k < Kp; k += 512) {       // Kp is even
        if constexpr (sizeof(OutT) == 2) *reinterpret_cast<__nv_bfloat162*>(o + k) = __floats2bfloat162_rn(xs[k], xs[k + 1]);
        else *reinterpret_cast<float2*>(o + k) = make_float2(xs[k], xs[k + 1]);
    }
}

// out[m] = base[m] + mult · norm(x[m])·gamma, one row per block; out may be base
__global__ void __launch_bounds__(256) k_norm_add(const RowOperand x, float* out, int ldo) {
    extern __shared__ __align__(16) float xs[];
    __shared__ float scratch[kRowScratchMax];
    const RowScratch sc(scratch, kMaxNormGroups);
    pdl_wait();
    pdl_launch_dependents();
    stage_segment(x, blockIdx.x, sc, [&](int k) -> float& { return xs[k]; });
    __syncthreads();
    for (int k = threadIdx.x; k < x.k; k += 256) out[(size_t)blockIdx.x * ldo + k] = xs[k];
}

// out[M × N] = A[M][Kp] (fp32) · W[N][Kp]ᵀ in fp32 FMAs: 64 × 64 tiles, 4 × 4 outputs per thread.
struct F32GemmParams {
    const float* a; const __nv_bfloat16* w; int M, N, Kp;
    const float* residual; int ldr; float* out; int ldo; int gluRow; float limit; float* glu; int ldglu; float softcap;
    const float* bias; int pair;
};
__global__ void __launch_bounds__(256) k_bf16_gemm_f32(const F32GemmParams p) {
    __shared__ float As[16][68], Ws[16][68];
    pdl_wait();
    pdl_launch_dependents();
    const int tid = threadIdx.x, m0 = blockIdx.y * 64, n0 = blockIdx.x * 64;
    const int tm = (tid >> 4) * 4, tn = (tid & 15) * 4;
    float acc[4][4] = {};
    for (int k0 = 0; k0 < p.Kp; k0 += 16) {
        for (int i = tid; i < 1024; i += 256) {
            const int r = i >> 4, k = i & 15;
            As[k][r] = (m0 + r < p.M && k0 + k < p.Kp) ? p.a[(size_t)(m0 + r) * p.Kp + k0 + k] : 0.0f;
            Ws[k][r] = (n0 + r < p.N && k0 + k < p.Kp) ? __bfloat162float(p.w[(size_t)(n0 + r) * p.Kp + k0 + k]) : 0.0f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 16; k++) {
            const float4 av = *reinterpret_cast<const float4*>(&As[k][tm]), wv = *reinterpret_cast<const float4*>(&Ws[k][tn]);
            const float a[4] = {av.x, av.y, av.z, av.w}, w[4] = {wv.x, wv.y, wv.z, wv.w};
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int m = m0 + tm + i;
        if (m >= p.M) continue;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int n = n0 + tn + j;
            if (n >= p.N) continue;
            if (n >= p.gluRow) {                         // gluRow is even and so is tn: a pair never leaves the thread
                if (((n - p.gluRow) & 1) == 0 && j < 3) p.glu[(size_t)m * p.ldglu + ((n - p.gluRow) >> 1)] = pair_f(acc[i][j], acc[i][j + 1], p.limit, p.pair);
            } else {
                float v = acc[i][j];
                if (p.bias) v += p.bias[n];
                if (p.residual) v += p.residual[(size_t)m * p.ldr + n];
                p.out[(size_t)m * p.ldo + n] = softcap_f(v, p.softcap);
            }
        }
    }
}

// Block-diagonal projection: out[m][h·os + n] = W[h·Nb + n] · x[m][h·xs …].  grid (heads, row tiles, groups of MR rows);
// few rows take one weight row per lane group and block, its first chunk in flight before the dependency wait.
template <int MR>
__global__ void __launch_bounds__(256) k_bf16_block(const float* __restrict__ x, int ldx, int xstr, const __nv_bfloat16* __restrict__ w, int K, int Kp, int Nb,
                                                    float* __restrict__ out, int ldo, int ostr, int M, int tile) {
    extern __shared__ __align__(16) float xs[];          // [MR][Kp]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int h = blockIdx.x, m0 = blockIdx.z * MR;
    const int chunks = Kp / 8;
    int lpr = 1;
    while (lpr < 32 && lpr < chunks) lpr <<= 1;          // lanes per weight row
    const int rpw = 32 / lpr, sub = lane / lpr, l = lane - sub * lpr;
    const int hi = min(Nb, ((int)blockIdx.y + 1) * tile);
    uint4 first = make_uint4(0, 0, 0, 0);
    {
        const int n = blockIdx.y * tile + warp * rpw + sub;
        if (n < hi && l < chunks) first = __ldg(reinterpret_cast<const uint4*>(w + ((size_t)h * Nb + n) * Kp + l * 8));
    }
    pdl_wait();
    pdl_launch_dependents();
#pragma unroll
    for (int m = 0; m < MR; m++)
        for (int k = threadIdx.x; k < Kp; k += 256) xs[m * Kp + k] = (k < K && m0 + m < M) ? x[(size_t)(m0 + m) * ldx + (size_t)h * xstr + k] : 0.0f;
    __syncthreads();
    for (int base = blockIdx.y * tile + warp * rpw; base < hi; base += 8 * rpw) {
        const int n = base + sub;
        float acc[MR];
#pragma unroll
        for (int m = 0; m < MR; m++) acc[m] = 0.0f;
        if (n < hi) {
            const __nv_bfloat16* wr = w + ((size_t)h * Nb + n) * Kp;
            for (int c = l; c < chunks; c += lpr) {
                const uint4 d = c == l && base == (int)blockIdx.y * tile + warp * rpw ? first : __ldg(reinterpret_cast<const uint4*>(wr + c * 8));
#pragma unroll
                for (int m = 0; m < MR; m++) {
                    const float4 x0 = *reinterpret_cast<const float4*>(xs + m * Kp + c * 8), x1 = *reinterpret_cast<const float4*>(xs + m * Kp + c * 8 + 4);
                    float v = acc[m];
                    v = fmaf(bf_lo(d.x), x0.x, v); v = fmaf(bf_hi(d.x), x0.y, v);
                    v = fmaf(bf_lo(d.y), x0.z, v); v = fmaf(bf_hi(d.y), x0.w, v);
                    v = fmaf(bf_lo(d.z), x1.x, v); v = fmaf(bf_hi(d.z), x1.y, v);
                    v = fmaf(bf_lo(d.w), x1.z, v); v = fmaf(bf_hi(d.w), x1.w, v);
                    acc[m] = v;
                }
            }
        }
#pragma unroll
        for (int m = 0; m < MR; m++) {
            for (int o = lpr >> 1; o > 0; o >>= 1) acc[m] += __shfl_xor_sync(0xffffffffu, acc[m], o);
            if (l == 0 && n < hi && m0 + m < M) out[(size_t)(m0 + m) * ldo + (size_t)h * ostr + n] = acc[m];
        }
    }
}

__global__ void __launch_bounds__(256) k_bf16_store(const float* __restrict__ src, int rows, int cols, __nv_bfloat16* __restrict__ dst, long long dst_ld) {
    const long long total = (long long)rows * cols;
    for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < total; i += (long long)gridDim.x * 256)
        dst[(i / cols) * dst_ld + i % cols] = __float2bfloat16_rn(src[i]);
}

void raise_smem(const void* kernel, size_t bytes) {
    static std::set<const void*> done;
    if (bytes > 40 * 1024 && done.insert(kernel).second)
        DJ_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kRowSmemMax));
}

}  // namespace

void launch_bf16_store(const float* src, int rows, int cols, __nv_bfloat16* dst, long long dst_ld, cudaStream_t s) {
    if (rows <= 0 || cols <= 0) return;
    launch_k(k_bf16_store, dim3((unsigned)std::min<long long>(((long long)rows * cols + 255) / 256, 16ll * g_num_sms)), dim3(256), 0, s, false, src, rows, cols, dst,
             dst_ld);
}

// False where the rows do not come in 16-byte pieces or are too long for the registers.
template <typename OutT>
static bool stage_rows_in_registers(const RowOperand& a, const RowOperand& b, int Kp, int rows, const int* map, int div, OutT* out, cudaStream_t s) {
    const int K1p = pad8(a.k);
    auto aligned = [](const RowOperand& r) {
        return (((uintptr_t)r.x | (uintptr_t)r.gate | (uintptr_t)r.base | (uintptr_t)r.sum | (uintptr_t)r.gamma) & 15) == 0 &&
               ((r.k | r.ldx | (r.gate ? r.ldg : 0) | (r.base ? r.ldbase : 0) | (r.sum ? r.ldsum : 0)) & 3) == 0 && (r.groups < 2 || r.k / r.groups % 4 == 0);
    };
    if (((uintptr_t)out & 15) != 0 || !aligned(a) || (b.k > 0 && (!aligned(b) || b.groups > 0)) || (a.groups > 0 && a.k > 4096)) return false;
    auto go = [&](auto kernel) { launch_k(kernel, dim3((unsigned)rows), dim3(256), 0, s, true, a, b, K1p, Kp, map, div, out); };
    if (a.groups == 0 || a.k <= 1024) go(k_stage_rows<OutT, 1>);
    else if (a.k <= 2048) go(k_stage_rows<OutT, 2>);
    else go(k_stage_rows<OutT, 4>);
    return true;
}
template <typename OutT>
static void stage_rows(const RowOperand& a, const RowOperand& b, int Kp, int rows, const int* map, int div, OutT* out, cudaStream_t s) {
    if (stage_rows_in_registers(a, b, Kp, rows, map, div, out, s)) return;
    raise_smem((const void*)k_stage_rows_any<OutT>, (size_t)Kp * 4);
    launch_k(k_stage_rows_any<OutT>, dim3((unsigned)rows), dim3(256), (size_t)Kp * 4, s, true, a, b, pad8(a.k), Kp, map, div, out);
}

void launch_stage_rows(const RowOperand& a, const RowOperand& b, int Kp, int rows, const int* map, int div, void* out, bool bf16, cudaStream_t s) {
    if (bf16) stage_rows(a, b, Kp, rows, map, div, (__nv_bfloat16*)out, s);
    else stage_rows(a, b, Kp, rows, map, div, (float*)out, s);
}

void launch_norm_add(const RowOperand& x, float* out, int ldo, int rows, cudaStream_t s) {
    if (ldo == x.k && x.k % 4 == 0 && stage_rows_in_registers(x, RowOperand(), x.k, rows, nullptr, 1, out, s)) return;
    const size_t smem = (size_t)pad8(x.k) * 4;
    raise_smem((const void*)k_norm_add, smem);
    launch_k(k_norm_add, dim3((unsigned)rows), dim3(256), smem, s, true, x, out, ldo);
}

constexpr int kGvMaxM = 16;      // up to here passes of the GEMV

size_t bf16_linear_ws_floats(const Bf16LinearArgs& a) {
    return a.M <= kGvMaxM ? 0 : (size_t)a.M * a.w.Kp;
}

const char* bf16_linear_check(const Bf16LinearArgs& a) {
    if ((size_t)a.w.Kp * 4 > (size_t)kRowSmemMax - 1024) return "reduction length too large";
    if (a.a.groups > kMaxNormGroups || a.b.groups > kMaxNormGroups) return "too many norm groups";
    if ((a.a.groups > 0 && a.a.k % a.a.groups != 0) || (a.b.groups > 0 && a.b.k % a.b.groups != 0)) return "norm groups must divide the row";
    return nullptr;
}

void launch_bf16_linear(const Bf16LinearArgs& a, cudaStream_t s) {
    if (a.M <= 0 || a.w.N <= 0) return;
    if (a.M <= kGvMaxM) {
        launch_bf16_gemv(a, s);
        return;
    }
    if (!a.exact && launch_bf16_gemm_tc(a, nullptr, s)) return;
    launch_stage_rows(a.a, a.b, a.w.Kp, a.M, nullptr, 1, a.ws, false, s);
    F32GemmParams p = {a.ws, a.w.w, a.M, a.w.N, a.w.Kp, a.residual, a.ldr, a.out, a.ldo, a.gluRow, a.limit, a.glu, a.ldglu, a.softcap,
                       a.bias, a.pair};
    launch_k(k_bf16_gemm_f32, dim3((a.w.N + 63) / 64, (a.M + 63) / 64), dim3(256), 0, s, true, p);
}

void launch_bf16_block_linear(const float* x, int ldx, int xstr, const Bf16View& w, int heads, float* out, int ldo, int ostr, int M, cudaStream_t s) {
    const int Nb = w.N / heads;
    const dim3 block(256);
    int lpr = 1;
    while (lpr < 32 && lpr < w.Kp / 8) lpr <<= 1;
    const int tile = M <= 4 ? 8 * (32 / lpr) : 64;
    const unsigned tiles = (unsigned)((Nb + tile - 1) / tile);
    auto go = [&](auto kernel, int MR) {
        const size_t smem = (size_t)MR * w.Kp * 4;
        raise_smem((const void*)kernel, smem);
        launch_k(kernel, dim3((unsigned)heads, tiles, (unsigned)((M + MR - 1) / MR)), block, smem, s, true, x, ldx, xstr, w.w, w.K, w.Kp, Nb, out, ldo, ostr, M, tile);
    };
    if (M == 1) go(k_bf16_block<1>, 1);
    else go(k_bf16_block<4>, 4);
}

}  // namespace dj
