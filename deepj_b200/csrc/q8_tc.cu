// Q8 linear for many activation rows (prompts, several sequences at once): tcgen05 tensor-core tiles, one accumulation
// per scale block.
//
// A Q8 weight is code · scale with one fp32 scale per 32 k, so a product over one block is scale · Σ x·code, and a code is
// exact in fp16.  The kernel multiplies the raw codes, block by block, and applies the scale afterwards in fp32:
//     D_b  = C_b · X_lo · 2^-11 + C_b · X_hi  tensor cores, K = 32, fp32 accumulator in tensor memory
//     acc += scale_b · D_b                    fp32 fused multiply-adds in registers
// X_hi + X_lo · 2^-11 is the activation as two fp16 values (≈ 22 bits, after a power-of-two row scaling by the pre-pass, which also
// applies the norm).  Weights enter without any rounding, and two MMAs per k-step are enough.  Folding the scale into the
// operand instead (weights as hi + lo fp16 pairs, accumulated over all of K) takes three, and the conversion costs 2.75
// instructions per weight instead of 1.25.
//
// The tile is 128 weight rows × NT activation rows with the weights as the M side: a thread of the promoting warps owns a
// tensor-memory lane = one weight row, so its block scale is one register and its result rows are stored 128 contiguous
// bytes at a time.  The fp16 codes go to tensor memory too and enter the MMAs from there: with them in shared memory the
// converters' stores and the MMAs' operand reads together asked for its whole 128 bytes a cycle (measured: 8 MMAs of
// 128 × 64 × 16 took 780 cycles beside the converters and 392 alone).  28 warps:
//   warps 0-15   read the block's accumulator (tcgen05.ld, 32 lanes × NT/4 columns each) and add it to registers; afterwards
//                the epilogue.  Half the time of such a step is the latency of its barrier and loads, so four warps per
//                scheduler share it (eight warps of NT/2 columns: 832 cycles per pair of blocks at NT = 96)
//   warps 16-23  convert, as two groups of four that take the stages in turn: one weight row per thread, 32 codes → 64 bytes
//                of fp16 per block, stored to its lane
//   warp 24      copies the activation images (one plain bulk copy per stage)
//   warp 25      streams the raw codes: 128-byte × 128-row boxes through the tensor-memory accelerator
//   warps 26-27  issue the MMAs (128 × NT × 16, four per block) into a ring of accumulators and commit, taking the stages in
//                turn: the waits and commits of one stage cost an issuing thread ≈ 400 cycles, in which the other one issues
// SwiGLU takes 64 gate and 64 up rows per tile, so the pair meets in one epilogue.  When the grid leaves SMs idle the
// reduction is split over the CTAs of a cluster, which add their parts through distributed shared memory in split order.
// Every wait is bounded: when a bound expires the CTA records an error code, stops waiting, lets its copies in flight
// land, frees its tensor memory and returns without storing its results.  A bound times this kernel alone: a wait that ends
// only with the activation images, which an earlier kernel writes, comes behind the dependency wait, so an earlier kernel that
// takes its time (an exchange polling a late peer) costs none of it.  The first weights are loaded and converted before that.
#include "kernels.h"
#include "q8_tma.cuh"
#include "tc_common.cuh"
#include <cfloat>
#include <cuda_fp16.h>

namespace dj {
namespace {

constexpr int kRows = 128;                               // weight rows of a tile
constexpr int kBlockK = 32;                              // one scale block
constexpr int kGroup = 4;                                // blocks per raw-code box: 128 bytes of a weight row
constexpr int kRawBytes = kRows * kBlockK * kGroup;      // raw codes of one group: 16 KB
constexpr int kPromoteWarps = 16, kConvertWarps = 8;      // converters: two groups of four
constexpr int kCopyWarp = kPromoteWarps + kConvertWarps, kRawWarp = kCopyWarp + 1, kMmaWarp = kCopyWarp + 2;   // two MMA warps
constexpr int kTcThreads = 896;
constexpr int kLoBits = 11;                              // the low halves are stored 2^11 times too large
constexpr float kLoUp = (float)(1 << kLoBits);
constexpr int kFold = 8;                                 // blocks of a running sum (see the promoting warps)
constexpr int kMaxSplits = 8;                            // portable cluster size
// Registers: 896 threads × 72 at launch; 512 × 88 + 384 × 48 = 63488 afterwards.
constexpr int kPromoteRegs = 88, kOtherRegs = 48;

// Below 128 activation rows a block's products take less time than the barriers around them: a pipeline stage then holds two
// blocks (rows of 128 bytes, 128-byte swizzle) and accumulators are handed over in pairs.
constexpr int blocks_per_stage(int nt) { return nt < 128 ? 2 : 1; }
template <int NT, bool FOLD> struct TileShape {
    static constexpr int kPer = blocks_per_stage(NT);
    static constexpr int kStages = kPer == 2 ? 4 : 6;
    static constexpr int kRawStages = 4;
    static constexpr int kRowBytes = 64 * kPer;
    static constexpr int kXBytes = NT * kRowBytes;                   // one half (hi or lo) of a stage's activations
    static constexpr int kStageBytes = 2 * kXBytes;
    // tensor memory: accumulators, handed over kPer at a time, then per stage the fp16 codes (16 columns of two per block)
    static constexpr int kAccStride = NT < 32 ? 32 : NT;
    static constexpr int kSlots = kPer == 2 && NT <= 32 ? 4 : 2;
    static constexpr int kWCols = 16 * kPer, kWBase = kSlots * kPer * kAccStride;
    static constexpr int kCols = NT / 4;                             // accumulator columns per promoting warp
    static constexpr size_t kPipe = (size_t)kStages * kStageBytes + (size_t)kRawStages * kRawBytes;
    static constexpr size_t kSmem = kPipe + 1024 + (FOLD ? (size_t)NT * kRows * 4 : 0);
    static constexpr uint32_t kIdesc = (1u << 4) | ((uint32_t)(NT >> 3) << 17) | ((uint32_t)(kRows >> 4) << 24);   // fp16 × fp16 → fp32, K-major
    // K-major: 8-row groups 8 · kRowBytes apart, descriptor version 1, layout type 4 (64-byte swizzle) or 2 (128-byte)
    static constexpr uint64_t kDesc = ((uint64_t)1 << 16) | ((uint64_t)(8 * kRowBytes >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)(kPer == 1 ? 4 : 2) << 61);
    static_assert(kWBase + kStages * kWCols <= 512, "tensor memory");
    static_assert((size_t)NT * kRows * 4 <= kPipe, "the partial tile fits the pipeline's memory");
    static_assert(kCols % 4 == 0 && kFold == 2 * kGroup, "totals move four columns at a time, over two groups of blocks");
    static_assert(kSmem + 2048 <= 227 * 1024, "shared memory of one CTA");
};

// byte offset of 16-byte chunk c of row r inside a swizzled K-major tile of 32 or 64 halves per row
__host__ __device__ __forceinline__ int swz_off(int r, int c, int per) {
    return per == 1 ? r * 64 + ((c ^ ((r >> 1) & 3)) << 4) : r * 128 + ((c ^ (r & 7)) << 4);
}

__device__ __forceinline__ uint32_t pack_h2(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));      // first source → upper half
    return r;
}

// NC consecutive columns of the warp's 32 lanes → v, asynchronously
template <int NC> __device__ __forceinline__ void tmem_ld_nowait(uint32_t taddr, uint32_t* v) {
    if constexpr (NC >= 16) {
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                     : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
                       "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                     : "r"(taddr));
        if constexpr (NC > 16) tmem_ld_nowait<NC - 16>(taddr + 16, v + 16);
    } else if constexpr (NC == 8) {
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]) : "r"(taddr));
    } else {
        static_assert(NC == 4, "columns come in fours, eights and sixteens");
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(taddr));
    }
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&v)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                 ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]) : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// D (tensor memory) = or += A (tensor memory) · B (shared memory); the second form scales D by 2^-kLoBits first
__device__ __forceinline__ void umma_f16_ts(uint32_t d, uint32_t a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}"
                 ::"r"(d), "r"(a), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void umma_f16_ts_down(uint32_t d, uint32_t a, uint64_t bdesc, uint32_t idesc) {
    asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, 1, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p, %4;\n}"
                 ::"r"(d), "r"(a), "l"(bdesc), "r"(idesc), "n"(kLoBits) : "memory");
}

// acc (two floats) += v (two floats) · s (the same float twice).  Volatile: v comes from an asynchronous load, and no use of it
// may be scheduled before the wait.
__device__ __forceinline__ void fma2(unsigned long long& acc, uint32_t v0, uint32_t v1, unsigned long long s) {
    asm volatile("{\n .reg .b64 v;\n mov.b64 v, {%1, %2};\n fma.rn.f32x2 %0, v, %3, %0;\n}" : "+l"(acc) : "r"(v0), "r"(v1), "l"(s));
}

// Two running sums move to their totals: returns total + sum, and sum keeps what that rounded off.  An infinite total leaves NaN
// there, which the minimum takes back to a finite value (it is one of the largest that matter: a part cut off a total above
// 2^90 may be lost, as in a plain sum), so the total stays infinite.
__device__ __forceinline__ unsigned long long move_sum(unsigned long long& sum, unsigned long long total) {
    unsigned long long t, d;
    float x, y;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(t) : "l"(total), "l"(sum));
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(t), "l"(total));
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(sum), "l"(d));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(d));
    asm("mov.b64 %0, {%1, %2};" : "=l"(sum) : "f"(fminf(x, 0x1p66f)), "f"(fminf(y, 0x1p66f)));
    return t;
}

// A whole warp waits.  The first try decides nearly always (the instruction itself waits for a while); entering the bounded
// loop costs more than 100 cycles even when the barrier is ready (measured: 170 against 48).  The vote makes the result
// uniform for the compiler, so that what follows (descriptors, stage addresses) can stay in uniform registers.
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int* error, int code) {
    if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
    return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag, error, code));
}
// Whether a phase is over, without waiting for it.
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n .reg .pred P;\n elect.sync _|P, 0xffffffff;\n selp.u32 %0, 1, 0, P;\n}" : "=r"(p));
    return p != 0;
}

__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t peer_addr(uint32_t addr, uint32_t rank) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
    return a;
}
__device__ __forceinline__ float ld_peer(uint32_t addr) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
    return v;
}

// ───────────── pre-pass: fp32 activations → hi/lo fp16 images ─────────────
// x · 2^s = hi + lo / 2^11: the low half is stored 2^11 times too large, so that it keeps its 11 bits as a normal fp16 number
// down to 2^-24 of the row's largest value (unscaled it would lose them from 2^-17 on).
// Image: per tile of nt rows and stage of per blocks, X_hi then X_lo in the swizzled layout that the MMA reads, so that a stage
// is one contiguous copy.  Blocks that fill up the last stage are zeros.  rowscale[m] undoes the power-of-two row scaling in
// the epilogue.  Rows from M on are left alone: they only reach result rows that are never stored.  One block per row; norm:
// RMSNorm (γ) or LayerNorm (γ, β).
constexpr int kXThreads = 256;
struct XImages {
    const float* x; int ldx;
    const float* gamma; const float* beta; float eps;
    int K, nS, nt, per;
    unsigned char* images; float* rowscale;
};

struct RowScale { float down; bool finite; };
__device__ __forceinline__ RowScale row_scale(float amax, float* rowscale) {
    // A power of two brings the row's largest value into [2^14, 2^15).  Both that factor and its inverse stay normal numbers: a
    // largest value below 2^-112 is scaled as if it were that (a subnormal one then still has all its bits in fp16), and a row
    // with an infinity as the largest finite exponent.  Such a row has no low halves: they would turn the infinity, and every
    // result of the row is infinite or NaN with it, into NaN.
    const int ebits = min(max(__float_as_int(amax) & 0x7f800000, 15 << 23), 254 << 23);
    const float down = __uint_as_float((268u << 23) - (unsigned)ebits);
    const bool finite = amax <= FLT_MAX;
    if (threadIdx.x == 0) *rowscale = __int_as_float(ebits - (14 << 23));
    return {down, finite};
}
__device__ __forceinline__ void put_chunk(const XImages& p, int m, int c, const float (&v)[8], const RowScale& s) {
    uint32_t hi[4], lo[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const float a = v[2 * j] * s.down, b = v[2 * j + 1] * s.down;
        hi[j] = pack_h2(a, b);
        const float2 back = __half22float2(*reinterpret_cast<const __half2*>(&hi[j]));
        lo[j] = s.finite ? pack_h2((a - back.x) * kLoUp, (b - back.y) * kLoUp) : 0u;
    }
    const int rowBytes = 64 * p.per, mt = m / p.nt, r = m - mt * p.nt, st = c / (4 * p.per), cc = c - st * 4 * p.per;
    unsigned char* t = p.images + ((size_t)mt * p.nS + st) * 2 * p.nt * rowBytes + swz_off(r, cc, p.per);
    *reinterpret_cast<uint4*>(t) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    *reinterpret_cast<uint4*>(t + p.nt * rowBytes) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
}
template <typename F>
__device__ __forceinline__ float block_all(float v, float* r, F join) {      // joined over the block; r: one float per warp
    for (int o = 16; o > 0; o >>= 1) v = join(v, __shfl_xor_sync(0xffffffffu, v, o));
    if ((threadIdx.x & 31) == 0) r[threadIdx.x >> 5] = v;
    __syncthreads();
    v = r[0];
#pragma unroll
    for (int q = 1; q < kXThreads / 32; q++) v = join(v, r[q]);
    return v;
}

// The row in registers, up to CH chunks of eight values per thread: one load round trip, the gain's ahead of the dependency wait.
// 123 rows of 2048: 4.7 µs with passes over memory for each sum, 3.1 this way; 2048 rows of 4096 22 and 13.  Six chunks are one block per SM:
// many rows of 6400 with LayerNorm took 1.4 times as long with their product as passes did, in four chunks as long.
template <int CH>
__global__ void __launch_bounds__(kXThreads) k_x_images(const XImages p) {
    __shared__ float red[3][kXThreads / 32];
    pdl_launch_dependents();
    const int tid = threadIdx.x, m = blockIdx.x;
    constexpr bool EARLY = CH <= 4;                  // the shift too (with six chunks it would leave no registers)
    float v[CH][8], g[CH][8], b[CH][8];
    auto load = [&](const float* from, float (&to)[CH][8], float fill) {
#pragma unroll
        for (int i = 0; i < CH; i++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int k = (tid + i * kXThreads) * 8 + 4 * h;
                float4 a = make_float4(fill, fill, fill, fill);
                if (k < p.K && from != nullptr) a = *reinterpret_cast<const float4*>(from + k);
                to[i][4 * h] = a.x; to[i][4 * h + 1] = a.y; to[i][4 * h + 2] = a.z; to[i][4 * h + 3] = a.w;
            }
    };
    if (p.gamma != nullptr) load(p.gamma, g, 0.0f);
    if (EARLY && p.beta != nullptr) load(p.beta, b, 0.0f);
    pdl_wait();
    load(p.x + (size_t)m * p.ldx, v, 0.0f);
    auto add = [](float a, float b) { return a + b; };
    if (p.beta != nullptr) {
        float sm = 0.0f;
#pragma unroll
        for (int i = 0; i < CH; i++)
#pragma unroll
            for (int e = 0; e < 8; e++) sm += v[i][e];
        const float mean = block_all(sm, red[0], add) * (1.0f / (float)p.K);
#pragma unroll
        for (int i = 0; i < CH; i++)
#pragma unroll
            for (int e = 0; e < 8; e++)
                if ((tid + i * kXThreads) * 8 + (e & 4) < p.K) v[i][e] -= mean;
    }
    float amax = 0.0f;
    if (p.gamma != nullptr) {
        float ss = 0.0f;
#pragma unroll
        for (int i = 0; i < CH; i++)
#pragma unroll
            for (int e = 0; e < 8; e++) ss = fmaf(v[i][e], v[i][e], ss);
        const float root = sqrtf(block_all(ss, red[1], add) * (1.0f / (float)p.K) + p.eps);
        if (p.beta != nullptr) {                     // LayerNorm divides by it, RMSNorm multiplies
            if (!EARLY) load(p.beta, b, 0.0f);
#pragma unroll
            for (int i = 0; i < CH; i++)
                if ((tid + i * kXThreads) * 8 < p.K) {       // (dividing zeros is slow: 64 rows of 512, with the product, 9.9 µs, 7.6 without)
#pragma unroll
                    for (int e = 0; e < 8; e++) v[i][e] = __fdiv_rn(v[i][e], root) * g[i][e] + b[i][e];
                }
        } else {
            const float inv = __frcp_rn(root);
#pragma unroll
            for (int i = 0; i < CH; i++)
#pragma unroll
                for (int e = 0; e < 8; e++) v[i][e] = (v[i][e] * inv) * g[i][e];
        }
    }
#pragma unroll
    for (int i = 0; i < CH; i++)
#pragma unroll
        for (int e = 0; e < 8; e++) amax = fmaxf(amax, fabsf(v[i][e]));
    const RowScale s = row_scale(block_all(amax, red[2], [](float a, float b) { return fmaxf(a, b); }), p.rowscale + m);
#pragma unroll
    for (int i = 0; i < CH; i++)
        if (tid + i * kXThreads < p.nS * p.per * 4) put_chunk(p, m, tid + i * kXThreads, v[i], s);
}

// Rows of any length: a pass for each sum, four neighbouring values a thread and step (eight, as the chunks are: 64 rows of 14336, with the product, 42 µs in place of 34).
__global__ void __launch_bounds__(kXThreads) k_x_images_long(const XImages p) {
    __shared__ float red[3][kXThreads / 32];
    pdl_launch_dependents();
    pdl_wait();
    const int tid = threadIdx.x, m = blockIdx.x;
    const float* xr = p.x + (size_t)m * p.ldx;
    auto add = [](float a, float b) { return a + b; };
    float mean = 0.0f, inv = 1.0f;
    if (p.beta != nullptr) {
        float sm = 0.0f;
        for (int k = tid * 4; k < p.K; k += 4 * kXThreads) {
            const float4 v = *reinterpret_cast<const float4*>(xr + k);
            sm += (v.x + v.y) + (v.z + v.w);
        }
        mean = block_all(sm, red[0], add) * (1.0f / (float)p.K);
    }
    if (p.gamma != nullptr) {
        float ss = 0.0f;
        for (int k = tid * 4; k < p.K; k += 4 * kXThreads) {
            float4 v = *reinterpret_cast<const float4*>(xr + k);
            v.x -= mean; v.y -= mean; v.z -= mean; v.w -= mean;
            ss = fmaf(v.x, v.x, ss); ss = fmaf(v.y, v.y, ss); ss = fmaf(v.z, v.z, ss); ss = fmaf(v.w, v.w, ss);
        }
        const float root = sqrtf(block_all(ss, red[1], add) * (1.0f / (float)p.K) + p.eps);
        inv = p.beta != nullptr ? root : __frcp_rn(root);      // LayerNorm divides by it, RMSNorm multiplies
    }
    auto value = [&](float v, float g, float b) {
        if (p.beta != nullptr) return __fdiv_rn(v - mean, inv) * g + b;
        return p.gamma != nullptr ? (v * inv) * g : v;
    };
    auto load4 = [&](int k, float* v) {
        const float4 a = *reinterpret_cast<const float4*>(xr + k);
        float4 g = make_float4(1.f, 1.f, 1.f, 1.f), b = make_float4(0.f, 0.f, 0.f, 0.f);
        if (p.gamma) g = *reinterpret_cast<const float4*>(p.gamma + k);
        if (p.beta) b = *reinterpret_cast<const float4*>(p.beta + k);
        v[0] = value(a.x, g.x, b.x); v[1] = value(a.y, g.y, b.y); v[2] = value(a.z, g.z, b.z); v[3] = value(a.w, g.w, b.w);
    };
    float amax = 0.0f;
    for (int k = tid * 4; k < p.K; k += 4 * kXThreads) {
        float v[4];
        load4(k, v);
        amax = fmaxf(amax, fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3]))));
    }
    const RowScale s = row_scale(block_all(amax, red[2], [](float a, float b) { return fmaxf(a, b); }), p.rowscale + m);
    for (int c = tid; c < p.nS * p.per * 4; c += kXThreads) {
        float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int h = 0; h < 2; h++)
            if (c * 8 + 4 * h < p.K) load4(c * 8 + 4 * h, v + 4 * h);
        put_chunk(p, m, c, v, s);
    }
}

struct TcParams {
    CUtensorMap codes, codes2;          // boxes of 128 bytes × 128 rows (64 rows of each for SwiGLU)
    const unsigned char* images; const float* rowscale;
    const float* scales; const float* scales2;
    const float* bias; const float* bias2;
    const float* residual; int ldr;
    float* out; int ldo;
    int M, N, nb, nK, nS;               // nK blocks, nS stages of the whole reduction
    int swiglu, gelu;
    int splits, ktPer;                  // CTAs of a cluster share the reduction, ktPer blocks (a multiple of 4) each
    int lo;                             // 1: the X_lo product is added
    int coarse;                         // 1: block scales rounded to 11 bits
    int* error;
};

// Four block scales from block k on; past the row's end zeros, which only meet blocks that do not exist.  Rows are laid out in multiples
// of four blocks, so the scalar half is not taken, but the kernel is compiled better with it: with the vector load alone a prompt of 123 rows through 11
// layers of width 2048 takes 1445 µs instead of 1375; with the rounding moved to the use, 512 rows of 4096 → 4096 take 63.3 instead of 54.2
// and 123 of 11008 → 4096 47.6 instead of 41.8; with the load as volatile assembly 256 of 11008 → 4096 81 instead of 73.
__device__ __forceinline__ float4 load_scales(const float* row, int k, int nb, bool vec, bool coarse) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (vec) {
        if (k < nb) v = *reinterpret_cast<const float4*>(row + k);
    } else {
        if (k < nb) v.x = row[k];
        if (k + 1 < nb) v.y = row[k + 1];
        if (k + 2 < nb) v.z = row[k + 2];
        if (k + 3 < nb) v.w = row[k + 3];
    }
    if (coarse) {
        auto cut = [](float f) { return __uint_as_float((__float_as_uint(f) + 0x1000u) & 0xffffe000u); };      // 11 bits, at any size
        v = make_float4(cut(v.x), cut(v.y), cut(v.z), cut(v.w));
    }
    return v;
}

template <int NT, bool FOLD>
__global__ void __launch_bounds__(kTcThreads, 1) k_q8_gemm_tc(const __grid_constant__ TcParams p) {
    using S = TileShape<NT, FOLD>;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    __shared__ __align__(8) unsigned long long s_bar[2 * S::kStages + 2 * S::kRawStages + 2 * S::kSlots];
    __shared__ uint32_t s_tmem;
    __shared__ volatile int s_abort;
    __shared__ float s_rowscale[NT], s_bias[kRows];

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int split = (int)blockIdx.x, m0 = (int)blockIdx.y * NT;
    const int rowsOut = p.swiglu ? kRows / 2 : kRows;             // output columns of a tile
    const int n0 = (int)blockIdx.z * rowsOut;
    const int kt0 = split * p.ktPer;
    const int nK = min(p.ktPer, p.nK - kt0);                      // blocks of this CTA; at least one
    const uint32_t raw_s = smem_u32(smem_raw), base = (raw_s + 1023u) & ~1023u;      // the swizzled tiles want 1024-byte alignment
    unsigned char* const smem = smem_raw + (base - raw_s);
    // layout: [stage: X_hi | X_lo] × kStages, then [raw codes 16 KB] × kRawStages
    const uint32_t rawBase = base + S::kStages * S::kStageBytes;
    auto full = [&](int s) { return smem_u32(&s_bar[s]); };
    auto empty = [&](int s) { return smem_u32(&s_bar[S::kStages + s]); };
    auto rawFull = [&](int s) { return smem_u32(&s_bar[2 * S::kStages + s]); };
    auto rawEmpty = [&](int s) { return smem_u32(&s_bar[2 * S::kStages + S::kRawStages + s]); };
    auto accFull = [&](int a) { return smem_u32(&s_bar[2 * S::kStages + 2 * S::kRawStages + a]); };
    auto accEmpty = [&](int a) { return smem_u32(&s_bar[2 * S::kStages + 2 * S::kRawStages + S::kSlots + a]); };

    if (tid == 0) {
        for (int s = 0; s < S::kStages; s++) { mbar_init(full(s), 1 + kConvertWarps / 2); mbar_init(empty(s), 1); }
        for (int s = 0; s < S::kRawStages; s++) { mbar_init(rawFull(s), 1); mbar_init(rawEmpty(s), kConvertWarps); }
        for (int a = 0; a < S::kSlots; a++) { mbar_init(accFull(a), 1); mbar_init(accEmpty(a), kPromoteWarps); }
        s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kMmaWarp) tmem_alloc(smem_u32(&s_tmem), 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    pdl_launch_dependents();

    if (warp < kPromoteWarps) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kPromoteRegs));
        const int quarter = warp & 3, part = warp >> 2;
        const int r = quarter * 32 + lane;                        // tile row = tensor-memory lane
        const bool second = p.swiglu && r >= kRows / 2;
        const int n = min(n0 + (second ? r - kRows / 2 : r), p.N - 1);
        const float* const srow = (second ? p.scales2 : p.scales) + (size_t)n * p.nb;
        const bool vec = (p.nb & 3) == 0;
        const uint32_t lane_base = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(part * S::kCols);
        unsigned long long acc[S::kCols / 2];
#pragma unroll
        for (int j = 0; j < S::kCols / 2; j++) acc[j] = 0ull;
        // The blocks' sums are added one after another, which over the 50 to 350 blocks of a row rounds more than the products
        // do.  FOLD: every kFold blocks a running sum moves to a total in shared memory, and what the total's rounding cuts off stays
        // in the running sum, so the error no longer grows with the length (against 64 bits 1.78e-7 at K = 1600 and 2.1e-7 at 5648
        // without, 0.93e-7 and 1.02e-7 with it).  Four columns of a thread lie side by side; they take turns, so that the warps
        // never stop for all of them at once: a block costs 3, 5, 15, 25 and 40 % more from 16 to 128 rows (all columns at once: 0, 3, 19, 47, 41).
        ulonglong2* const total = reinterpret_cast<ulonglong2*>(smem + S::kPipe) + tid;
        if (FOLD)
#pragma unroll
            for (int q = 0; q < S::kCols / 4; q++) total[q * kPromoteWarps * 32] = make_ulonglong2(0ull, 0ull);
        auto fold = [&](int odd, int i) {                         // after block i of an even or odd group
            constexpr int turns = kGroup / S::kPer;               // per group
#pragma unroll
            for (int q = 0; q < S::kCols / 4; q++)
                if (q % (kFold / S::kPer) == i / S::kPer + odd * turns) {
                    ulonglong2* const at = total + q * kPromoteWarps * 32;
                    const ulonglong2 o = *at;
                    *at = make_ulonglong2(move_sum(acc[2 * q], o.x), move_sum(acc[2 * q + 1], o.y));
                }
        };
        float4 next = load_scales(srow, kt0, p.nb, vec, p.coarse);
        // accumulator and phase parity of the i-th block of group g
        auto slot_of = [](int g, int i) { return S::kSlots == 4 ? (g & 1) * 2 + i / 2 : i / S::kPer % 2; };
        auto parity_of = [](int g, int i) { return (uint32_t)(S::kSlots == 4 ? g >> 1 : S::kPer == 2 ? g : i >> 1) & 1u; };
        auto add = [&](const uint32_t* v, float sc) {
            unsigned long long ss;
            asm("mov.b64 %0, {%1, %1};" : "=l"(ss) : "f"(sc));
#pragma unroll
            for (int j = 0; j < S::kCols / 2; j++) fma2(acc[j], v[2 * j], v[2 * j + 1], ss);
        };
        pdl_wait();                                               // ahead of the first bounded wait
        // what the epilogue needs of memory besides the residual: loaded there, it would wait for it
        if (tid < NT) s_rowscale[tid] = m0 + tid < p.M ? p.rowscale[m0 + tid] : 0.0f;
        else if (tid >= 128 && tid < 128 + kRows) {
            const int i = tid - 128;
            const bool up = p.swiglu && i >= kRows / 2;
            const float* const bias = up ? p.bias2 : p.bias;
            const int at = n0 + (up ? i - kRows / 2 : i);
            s_bias[i] = bias != nullptr && at < p.N ? bias[at] : 0.0f;
        }
        bool ok = true, ready = false;                            // ready: the next accumulator was seen complete already
        // Two groups per turn of the loop, so that whose turn it is among the totals (FOLD) and most parities are constants.
        constexpr int kUnroll = 2;
        for (int g0 = 0, b0 = 0; b0 < nK && ok; g0 += kUnroll) {
#pragma unroll
            for (int h = 0; h < kUnroll; h++, b0 += kGroup) {
                if (b0 >= nK || !ok) break;
                const int g = g0 + h;
                const float4 cur = next;
                if (b0 + kGroup < nK) next = load_scales(srow, kt0 + b0 + kGroup, p.nb, vec, p.coarse);
#pragma unroll
                for (int i = 0; i < kGroup; i += S::kPer) {
                    if (b0 + i >= nK) break;
                    const int slot = slot_of(g, i);
                    if (!__all_sync(0xffffffffu, ready)) ok = warp_wait(accFull(slot), parity_of(g, i), &s_abort, p.error, 202);
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t from = lane_base + (uint32_t)(slot * S::kPer * S::kAccStride);
                    const bool both = S::kPer == 2 && b0 + i + 1 < nK;                    // not an odd last block
                    uint32_t v[S::kPer][S::kCols];
                    tmem_ld_nowait<S::kCols>(from, v[0]);
                    tmem_wait_ld();
                    if (both) {
                        tmem_ld_nowait<S::kCols>(from + S::kAccStride, v[S::kPer - 1]);
                        add(v[0], i == 0 ? cur.x : i == 1 ? cur.y : i == 2 ? cur.z : cur.w);
                        tmem_wait_ld();
                    }
                    tc_fence_before();                                // everything is read: the MMAs may write here again
                    __syncwarp();
                    if (lane == 0) mbar_arrive(accEmpty(slot));
                    const int gn = i + S::kPer == kGroup ? g + 1 : g, in = (i + S::kPer) % kGroup;
                    ready = mbar_test(accFull(slot_of(gn, in)), parity_of(gn, in));
                    if (both) add(v[S::kPer - 1], i == 0 ? cur.y : cur.w);
                    else add(v[0], i == 0 ? cur.x : i == 1 ? cur.y : i == 2 ? cur.z : cur.w);
                    if (FOLD) fold(h, i);
                }
            }
        }
        // Every MMA of this CTA has completed (its last commits have been waited for) and every copy has landed: the pipeline's
        // memory takes the tile as [activation row][weight row].
        float* const mine = reinterpret_cast<float*>(smem) + (size_t)part * S::kCols * kRows + r;
#pragma unroll
        for (int j = 0; j < S::kCols / 2; j++) {
            float lo, hi;
            asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(acc[j]));
            if (FOLD) {
                const float2 t = reinterpret_cast<const float2*>(total + j / 2 * kPromoteWarps * 32)[j & 1];
                lo += t.x; hi += t.y;
            }
            mine[(2 * j) * kRows] = lo;
            mine[(2 * j + 1) * kRows] = hi;
        }
        // ── epilogue: CTA `split` of the cluster finishes every splits-th activation row; a warp stores 128 contiguous bytes ──
        // A warp's rows go in batches whose loads (the peers' parts, the residual) are in flight together.
        // Row by row each one waited for a load that could not pass the store before it: a CTA of 64 blocks took 14.4, 15.5, 20.7, 25.0
        // and 35.9 µs from 16 to 128 rows, and takes 13.6, 14.3, 18.0, 20.5 and 30.6.
        // Batches of eight are no faster, and slower where a CTA has few rows: their code has to be fetched first.
        constexpr int kBatch = 4;
        const int chunks = rowsOut / 32, phases = kPromoteWarps / chunks;      // 4 × 4, or 2 × 8 for SwiGLU
        const int rc = (warp % chunks) * 32 + lane, no = n0 + rc;
        const int first = split + p.splits * (warp / chunks), stride = p.splits * phases;
        tc_fence_before();
        __syncwarp();
        if (p.splits > 1) cluster_sync_all(); else asm volatile("bar.sync 1, %0;" ::"n"(kPromoteWarps * 32) : "memory");
        const int mEnd = s_abort ? 0 : min(NT, p.M - m0);
        const float bv = s_bias[rc], bv2 = p.swiglu ? s_bias[rc + kRows / 2] : 0.0f;
        float* const tile = reinterpret_cast<float*>(smem) + rc;
        if (p.splits > 1) {
            // the sum of all parts, in split order, replaces this CTA's own part of its rows (nobody else reads those)
            for (int half = 0; half <= p.swiglu; half++) {
                const uint32_t col = base + (uint32_t)(rc + half * (kRows / 2)) * 4;
                for (int i0 = 0; first + i0 * stride < mEnd; i0 += kBatch) {
                    float sum[kBatch] = {};
                    for (int z = 0; z < p.splits; z += 2) {                     // splits are a power of two
                        const uint32_t from0 = peer_addr(col, (uint32_t)z), from1 = peer_addr(col, (uint32_t)z + 1);
                        float x[kBatch], y[kBatch];
#pragma unroll
                        for (int e = 0; e < kBatch; e++) {
                            const int row = first + (i0 + e) * stride;
                            x[e] = row < mEnd ? ld_peer(from0 + (uint32_t)(row * kRows) * 4) : 0.0f;
                            y[e] = row < mEnd ? ld_peer(from1 + (uint32_t)(row * kRows) * 4) : 0.0f;
                        }
#pragma unroll
                        for (int e = 0; e < kBatch; e++) sum[e] = (sum[e] + x[e]) + y[e];
                    }
#pragma unroll
                    for (int e = 0; e < kBatch; e++)
                        if (first + (i0 + e) * stride < mEnd) tile[(first + (i0 + e) * stride) * kRows + half * (kRows / 2)] = sum[e];
                }
            }
        }
        for (int i0 = 0; first + i0 * stride < mEnd; i0 += kBatch) {
            float rv[kBatch];
#pragma unroll
            for (int e = 0; e < kBatch; e++) {
                const int row = first + (i0 + e) * stride;
                rv[e] = p.residual != nullptr && no < p.N && row < mEnd ? p.residual[(size_t)(m0 + row) * p.ldr + no] : 0.0f;
            }
#pragma unroll
            for (int e = 0; e < kBatch; e++) {
                const int row = first + (i0 + e) * stride;
                if (row >= mEnd) break;
                const float rs = s_rowscale[row];
                float v = tile[row * kRows] * rs + bv;
                if (p.swiglu) {
                    const float sig = 1.0f / (1.0f + expf(-v));
                    v = (v * sig) * (tile[row * kRows + kRows / 2] * rs + bv2);
                } else if (p.gelu) v = gelu_ref(v);
                if (p.residual != nullptr) v += rv[e];
                if (no < p.N) p.out[(size_t)(m0 + row) * p.ldo + no] = v;
            }
        }
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kOtherRegs));
        if (warp < kPromoteWarps + kConvertWarps) {
            // ── codes → fp16: thread r of a group owns tile row r; group g takes stages g, g + 2, … ──
            const int r = tid & 127, grp = (warp - kPromoteWarps) >> 2;
            const uint32_t wLane = tmem + ((uint32_t)((warp & 3) * 32) << 16) + S::kWBase;
            int rawAt = -1;                                       // raw group whose arrival has been waited for
            for (int i = grp; i * S::kPer < nK; i += 2) {
                const int b = i * S::kPer, g = b / kGroup, j = b % kGroup, rs = g % S::kRawStages, s = i % S::kStages;
                if (i >= S::kStages && i < S::kStages + 2) pdl_wait();    // from here on stages come back from the MMAs
                if (g != rawAt) { warp_wait(rawFull(rs), (g / S::kRawStages) & 1, &s_abort, p.error, 206); rawAt = g; }
                const unsigned char* src = smem + (size_t)S::kStages * S::kStageBytes + (size_t)rs * kRawBytes + r * 128;
                uint4 w[2 * S::kPer];
#pragma unroll
                for (int q = 0; q < 2 * S::kPer; q++) w[q] = *reinterpret_cast<const uint4*>(src + (((2 * j + q) ^ (r & 7)) << 4));
                if (i >= S::kStages) warp_wait(empty(s), (i / S::kStages - 1) & 1, &s_abort, p.error, 201);
                tc_fence_after();
#pragma unroll
                for (int q = 0; q < 2 * S::kPer; q++) {           // 16 codes → 8 columns
                    const uint32_t u4[4] = {w[q].x, w[q].y, w[q].z, w[q].w};
                    uint32_t h[8];
#pragma unroll
                    for (int e = 0; e < 4; e++) {                 // sign flip, byte under exponent 0x64 = 1024 + 128 + code, subtract 1152: exact
                        const uint32_t u = u4[e] ^ 0x80808080u;
                        const uint32_t a01 = __byte_perm(u, 0x64646464u, 0x4140), a23 = __byte_perm(u, 0x64646464u, 0x4342);
                        asm("sub.f16x2 %0, %1, %2;" : "=r"(h[2 * e]) : "r"(a01), "r"(0x64806480u));
                        asm("sub.f16x2 %0, %1, %2;" : "=r"(h[2 * e + 1]) : "r"(a23), "r"(0x64806480u));
                    }
                    tmem_st8(wLane + (uint32_t)(s * S::kWCols + 8 * q), h);
                }
                tmem_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(full(s));
                    // only now, after this group's last stage of the box: the stores above waited for the raw codes to reach
                    // registers; released right behind the load instructions, the buffer was refilled under them
                    if (S::kPer == 2 || j >= 2) mbar_arrive(rawEmpty(rs));
                }
            }
        } else if (warp == kCopyWarp) {
            pdl_wait();                                           // the images come from the pre-pass
            const unsigned char* src = p.images + ((size_t)blockIdx.y * p.nS + kt0 / S::kPer) * S::kStageBytes;
            const int n = (nK + S::kPer - 1) / S::kPer;
            int i = 0, s = 0;
            for (uint32_t round = 0; i < n; i++, src += S::kStageBytes) {
                if (round > 0 && !warp_wait(empty(s), (round - 1) & 1, &s_abort, p.error, 203)) break;
                if (elect_one()) {
                    mbar_arrive_expect_tx(full(s), S::kStageBytes);
                    bulk_g2s(base + s * S::kStageBytes, src, S::kStageBytes, full(s));
                }
                __syncwarp();
                if (++s == S::kStages) { s = 0; round++; }
            }
            if (i < n && lane == 0)                               // gave up: let the copies in flight land before the block goes
                for (int back = i - 1; back >= 0 && back >= i - S::kStages; back--)
                    for (unsigned w = 0; w < (1u << 16) && !mbar_try_wait(full(back % S::kStages), (back / S::kStages) & 1); w++) {}
        } else if (warp >= kMmaWarp) {
            const bool lo = p.lo != 0;
            // One thread's instructions are this loop's length, so stage and accumulator numbers are compile-time constants: the
            // descriptors become immediates on top of two uniform registers.
            const int which = warp - kMmaWarp;
            const uint32_t d0 = __shfl_sync(0xffffffffu, tmem, 0);
            const uint64_t x0 = S::kDesc | (base >> 4);
            pdl_wait();
            bool ok = true;
            for (uint32_t it = 0; it * (S::kStages * S::kPer) < (uint32_t)nK && ok; it++) {
#pragma unroll
                for (int u2 = 0; u2 < S::kStages; u2 += 2) {
                    const int u = u2 + which;
                    const int b = (int)it * S::kStages * S::kPer + u * S::kPer;
                    if (b >= nK) break;
                    static_assert(S::kSlots == 2 || (S::kSlots == 4 && S::kStages == 4), "a slot belongs to one issuing warp");
                    const int a = u % S::kSlots;
                    const uint32_t aRound = it * (S::kStages / S::kSlots) + u2 / S::kSlots;         // earlier uses of this accumulator
                    ok = (aRound == 0 || warp_wait(accEmpty(a), (aRound - 1) & 1, &s_abort, p.error, 204)) &&
                         warp_wait(full(u), it & 1, &s_abort, p.error, 205);
                    if (!ok) break;
                    tc_fence_after();
                    if (elect_one()) {
#pragma unroll
                        for (int j = 0; j < S::kPer; j++) {
                            if (j > 0 && b + j >= nK) break;
                            // a block is 16 columns of the codes and 64 bytes of an activation row, a k-step of 16 half of that
                            const uint32_t w = d0 + (uint32_t)(S::kWBase + u * S::kWCols + 16 * j);
                            const uint64_t xh = x0 + (uint32_t)(u * S::kStageBytes / 16 + 4 * j), xl = xh + S::kXBytes / 16;
                            const uint32_t d = d0 + (uint32_t)((a * S::kPer + j) * S::kAccStride);
                            // the small products first: an accumulation cuts the sum to 24 bits, so only the two at the
                            // full sum's size cost anything (four of them the other way round: 1.45e-7 of error against 64 bits
                            // at K = 688, 1.14e-7 this way)
                            if (lo) {
                                umma_f16_ts(d, w, xl, S::kIdesc, 0);
                                umma_f16_ts(d, w + 8, xl + 2, S::kIdesc, 1);
                                umma_f16_ts_down(d, w, xh, S::kIdesc);
                            } else umma_f16_ts(d, w, xh, S::kIdesc, 0);
                            umma_f16_ts(d, w + 8, xh + 2, S::kIdesc, 1);
                        }
                        umma_commit(accFull(a));
                        umma_commit(empty(u));
                    }
                    __syncwarp();
                }
            }
        } else if (warp == kRawWarp) {
            const int nG = (nK + kGroup - 1) / kGroup;            // weights depend on no earlier kernel: no wait before them
            int g = 0, s = 0;
            for (uint32_t round = 0; g < nG; g++) {
                if (g == S::kRawStages) pdl_wait();               // the first refill: the converters may be waiting for stages
                if (round > 0 && !warp_wait(rawEmpty(s), (round - 1) & 1, &s_abort, p.error, 207)) break;
                if (elect_one()) {
                    const uint32_t dst = rawBase + s * kRawBytes;
                    const int kx = (kt0 + g * kGroup) * kBlockK;
                    mbar_arrive_expect_tx(rawFull(s), kRawBytes);
                    tma_box(dst, &p.codes, kx, n0, rawFull(s));
                    if (p.swiglu) tma_box(dst + kRawBytes / 2, &p.codes2, kx, n0, rawFull(s));
                }
                __syncwarp();
                if (++s == S::kRawStages) { s = 0; round++; }
            }
            if (g < nG && lane == 0)
                for (int back = g - 1; back >= 0 && back >= g - S::kRawStages; back--)
                    for (unsigned w = 0; w < (1u << 16) && !mbar_try_wait(rawFull(back % S::kRawStages), (back / S::kRawStages) & 1); w++) {}
        }
        __syncwarp();
        pdl_wait();
        if (p.splits > 1) cluster_sync_all();
    }
    __syncwarp();
    if (p.splits > 1) cluster_sync_all(); else __syncthreads();   // peers have read this CTA's part
    if (warp == kMmaWarp) { tc_fence_after(); tmem_dealloc(tmem, 512); }
}

// ───────────── layout of a launch ─────────────
struct TcPlan { int nt, mTiles, nTiles, splits, ktPer; double us; };

// CTAs of this kernel that run at once in clusters of `sp`: one per SM, but a cluster stays inside a GPC, whose SMs are no
// multiple of it (148 SMs take 74 clusters of two, 33 of four and 15 of eight).
int cluster_slots(int sp) {
    if (sp == 1) return g_num_sms;
    auto ask = [](int size) {
        constexpr size_t smem = TileShape<128, false>::kSmem;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)size); cfg.blockDim = dim3(kTcThreads); cfg.dynamicSmemBytes = smem;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = (unsigned)size; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
        cfg.attrs = at; cfg.numAttrs = 1;
        int n = 0;
        if (cudaFuncSetAttribute(k_q8_gemm_tc<128, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
            cudaOccupancyMaxActiveClusters(&n, k_q8_gemm_tc<128, false>, &cfg) != cudaSuccess || n < 1) {
            cudaGetLastError();
            n = g_num_sms * 13 / 16 / size;
        }
        return n * size;
    };
    static const int slots[3] = {ask(2), ask(4), ask(8)};
    return slots[sp == 2 ? 0 : sp == 4 ? 1 : 2];
}

bool folds(int K, int ktPer) { return K % 128 != 0 && ktPer > kFold; }

// Tile width and reduction split with the least estimated time: rounds of CTAs over the SMs, each round a fixed part and one per
// block, the exchange of a cluster, and the pre-pass.  The costs of a width are from grids of whole rounds (148 r CTAs, two and six
// rounds at K = 1024 and 4096); with totals a block costs what one round of K = 8208 takes.  One round of 8 or 32 blocks per CTA
// takes 0.5-1.5, 0-1.4 and 1.0-3.7 µs more in clusters of 2, 4 and 8 than alone.  The pre-pass is from 64 to 512 rows of 2048 and 8192.
// Over 34 shapes of 20 to 2048 rows the estimates are within 8 % of the times measured, and the choice is the fastest but for
// 2048 x 2048 x 8192 (128 rows 222 µs, 96 rows 211).
TcPlan tc_plan(int M, int K, int N, bool swiglu) {
    static const struct { int nt; double cta, block, blockFold; } widths[] = {
        {16, 3.4, 0.158, 0.167}, {32, 3.9, 0.161, 0.171}, {64, 5.1, 0.200, 0.235}, {96, 7.4, 0.210, 0.27}, {128, 7.7, 0.333, 0.52}};
    const int nK = (K + kBlockK - 1) / kBlockK, rowsOut = swiglu ? kRows / 2 : kRows;
    const int nTiles = (N + rowsOut - 1) / rowsOut;
    const double pre = 0.8 + 0.3e-3 * K + 2e-6 * (double)M * K;
    TcPlan best = {}; best.us = 1e30;
    for (const auto& w : widths) {
        const int nt = w.nt;
        const int mTiles = (M + nt - 1) / nt;
        for (int sp = 1; sp <= kMaxSplits; sp *= 2) {
            const int ktPer = ((nK + sp - 1) / sp + kGroup - 1) / kGroup * kGroup;
            if (sp > 1 && (sp - 1) * ktPer >= nK) continue;                       // a CTA without blocks
            const int slots = cluster_slots(sp);
            const long ctas = (long)mTiles * nTiles * sp;
            const long rounds = (ctas + slots - 1) / slots;
            const double block = folds(K, ktPer) ? w.blockFold : w.block;
            const double us = pre + (double)rounds * (block * (ktPer < nK ? ktPer : nK) + w.cta) + (sp > 1 ? 0.4 + 0.15 * sp : 0.0);
            if (us < best.us) best = {nt, mTiles, nTiles, sp, ktPer, us};
        }
    }
    return best;
}

bool encode_codes(const Q8View& w, int rows, CUtensorMap* map) {
    EncodeTiledFn enc = encode_tiled_fn();
    if (!enc || ((uintptr_t)w.codes & 15) != 0 || w.Kp % 16 != 0) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)w.Kp, (cuuint64_t)w.N};
    const cuuint64_t strides[1] = {(cuuint64_t)w.Kp};
    const cuuint32_t box[2] = {(cuuint32_t)(kBlockK * kGroup), (cuuint32_t)rows};
    const cuuint32_t estr[2] = {1u, 1u};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<int8_t*>(w.codes), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int NT, bool FOLD> void run_as(const TcParams& p, const TcPlan& pl, cudaStream_t s) {
    using S = TileShape<NT, FOLD>;
    static bool attr = false;
    if (!attr) {
        DJ_CUDA_CHECK(cudaFuncSetAttribute(k_q8_gemm_tc<NT, FOLD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::kSmem));
        attr = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)pl.splits, (unsigned)pl.mTiles, (unsigned)pl.nTiles);
    cfg.blockDim = dim3(kTcThreads);
    cfg.dynamicSmemBytes = S::kSmem;
    cfg.stream = s;
    cudaLaunchAttribute at[2];
    int n = 0;
    if (pl.splits > 1) {
        at[n].id = cudaLaunchAttributeClusterDimension;
        at[n].val.clusterDim.x = (unsigned)pl.splits; at[n].val.clusterDim.y = 1; at[n].val.clusterDim.z = 1;
        n++;
    }
    if (g_use_pdl) { at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization; at[n].val.programmaticStreamSerializationAllowed = 1; n++; }
    cfg.attrs = at;
    cfg.numAttrs = (unsigned)n;
    g_launches++;
    DJ_CUDA_CHECK(cudaLaunchKernelEx(&cfg, k_q8_gemm_tc<NT, FOLD>, p));
}
template <int NT> void run(const TcParams& p, const TcPlan& pl, bool fold, cudaStream_t s) {
    if (fold) run_as<NT, true>(p, pl, s); else run_as<NT, false>(p, pl, s);
}

}  // namespace

int g_tc_terms = 3;

void q8_tc_plan(int M, int K, int N, bool swiglu, int* tileRows, int* splits) {
    const TcPlan pl = tc_plan(M, K, N, swiglu);
    *tileRows = pl.nt; *splits = pl.splits;
}
double q8_tc_estimate_us(int M, int K, int N, bool swiglu) { return tc_plan(M, K, N, swiglu).us; }

size_t q8_tc_ws_floats(int M, int K, int N, bool swiglu) {
    const TcPlan pl = tc_plan(M, K, N, swiglu);
    const size_t mPad = (size_t)pl.nt * pl.mTiles, nK = ((size_t)(K + kBlockK - 1) / kBlockK + 1) / 2 * 2;
    return nK * mPad * kBlockK + mPad;          // hi + lo halves = 4 bytes per value, then the row scales
}

// out = x · W (+ fused norm / bias / residual / GELU / SiLU-gate) for M ≥ 1 rows on the tensor cores.
// Returns false when the shape is outside the kernel's domain.
bool launch_q8_linear_tc(const Q8LinearArgs& a, float* ws, cudaStream_t s) {
    const int K = a.w.K, N = a.w.N, M = a.M;
    const bool swiglu = a.w2.codes != nullptr;
    if (ws == nullptr || ((uintptr_t)ws & 127) != 0 || M < 1 || K % 4 != 0 || g_dev_error == nullptr) return false;
    if (((uintptr_t)a.x & 15) != 0 || a.ldx % 4 != 0 || ((uintptr_t)a.gamma & 15) != 0 || ((uintptr_t)a.beta & 15) != 0) return false;
    if (((uintptr_t)a.w.scales & 15) != 0 || (swiglu && ((uintptr_t)a.w2.scales & 15) != 0)) return false;
    if (swiglu && a.act != 0) return false;
    TcParams p = {};
    if (!encode_codes(a.w, swiglu ? kRows / 2 : kRows, &p.codes) || (swiglu && !encode_codes(a.w2, kRows / 2, &p.codes2))) return false;
    const TcPlan pl = tc_plan(M, K, N, swiglu);
    if (pl.nTiles > 65535 || pl.mTiles > 65535) return false;
    const int per = blocks_per_stage(pl.nt);
    p.nK = (K + kBlockK - 1) / kBlockK; p.nS = (p.nK + per - 1) / per; p.nb = a.w.nb;
    unsigned char* const images = reinterpret_cast<unsigned char*>(ws);
    float* const rowscale = ws + (size_t)p.nS * per * kBlockK * pl.nt * pl.mTiles;
    const XImages xi = {a.x, a.ldx, a.gamma, a.beta, a.eps, K, p.nS, pl.nt, per, images, rowscale};
    const int chunks = (p.nS * per * 4 + kXThreads - 1) / kXThreads;     // of eight values per thread
    launch_k(chunks == 1 ? k_x_images<1> : chunks == 2 ? k_x_images<2> : chunks == 3 ? k_x_images<3> : chunks == 4 ? k_x_images<4> : chunks <= 6 ? k_x_images<6> : k_x_images_long, dim3((unsigned)M),
             dim3(kXThreads), 0, s, true, xi);
    p.images = images; p.rowscale = rowscale;
    p.scales = a.w.scales; p.scales2 = a.w2.scales; p.bias = a.bias; p.bias2 = a.bias2;
    p.residual = a.residual; p.ldr = a.ldr; p.out = a.out; p.ldo = a.ldo;
    p.M = M; p.N = N; p.swiglu = swiglu; p.gelu = a.act == 1;
    // K a multiple of 128: what runs these shapes with fewer rows keeps 16 bits of the activations, and a plain running sum is
    // far below that.  The kernels of the other lengths are 32-bit sums in short chains, and their error is the line here.
    const bool fold = folds(K, pl.ktPer);
    p.splits = pl.splits; p.ktPer = pl.ktPer; p.lo = g_tc_terms & 1; p.coarse = (g_tc_terms & 2) == 0; p.error = g_dev_error;
    switch (pl.nt) {
        case 16: run<16>(p, pl, fold, s); break;
        case 32: run<32>(p, pl, fold, s); break;
        case 64: run<64>(p, pl, fold, s); break;
        case 96: run<96>(p, pl, fold, s); break;
        default: run<128>(p, pl, fold, s); break;
    }
    return true;
}

}  // namespace dj

// Precision of the many-row path: bit 0 adds the X_lo product (activations at ≈ 22 bits, else 11 and half the products), bit 1
// keeps the block scales in fp32 (else they are rounded to 11 bits, which saves nothing: the weights' part of the setting is
// kept for callers that compare precisions).  Drops the cached CUDA graphs, which hold the old value.
extern "C" int deepj_cuda_tc_configure(int32_t correction_terms) {
    if (correction_terms < 0 || correction_terms > 3) { dj::set_last_error("tc_configure: correction_terms must be 0..3"); return 1; }
    if (dj::g_tc_terms != correction_terms) { dj::g_tc_terms = correction_terms; dj::invalidate_graphs(); }
    return 0;
}
