// Q8 GEMV on the integer tensor pipe with warp-private TMA rings — the decode kernel for up to four activation rows per pass, for
// reduction lengths that are multiples of 32.
//
// One int8 MMA m16n8k32 per 32-k block of 16 weight rows; the codes are the A operand as they are, the activations three
// base-256 digit columns with a power-of-two block scale; the integer block sums are exact, converted to fp32 exactly (an
// integer add and a subtraction on the main pipes) and (weight scale × activation scale) × sum is accumulated in fp32.  One
// lane of a warp issues four tiled bulk copies per item (two 8-row × 128-byte boxes of codes, two 8-row × 4 boxes of scales,
// straight from the [N][K] / [N][K/32] layout of the format, 128-byte swizzle; boxes of 16 rows took 25 % longer in long
// streams) that complete on a warp-private mbarrier, and the warp reads its MMA operands with one ldmatrix.x4 per block.
//
// Two blocks of 8 warps per SM; warp w owns the 128-k groups w, w+8, … of every tile of its block and stages exactly those groups of the
// activations itself; its sums of a tile, the digits recombined, go to shared memory, and one barrier per 16 tiles (or at the
// end) stands between them and the outputs.  (One block per SM with rings twice as deep: 5.9 against 4.7 ms for eight 7B steps, 8 warps
// do not keep up with the stream.)  A launch of a few microseconds runs most of its code once, and fetching 1 KB of code
// that another kernel has displaced takes 0.15 µs: the conversion is a loop over four groups in registers, and rows that do not come in
// 16-byte pieces have a form of their own (PLAIN), whose lanes also fill the rings themselves, with cp.async, so that it serves
// without tensor maps too.  Measured from the dependency wait to the last block's end, against the kernel with everything
// unrolled and a barrier per tile: 2048 → 2048 1.9-2.6 µs (1.9-2.9), gate and up of 5632 5.9 (7.6), 5632 → 2048 5.7 (6.0), head of
// 32000 × 2048 13.2 (15.6), gate and up of 11008 × 4096 18.0 (19.2), 4096 → 4096 4.0 (5.2).  GPT blocks (LayerNorm, GELU, reduction lengths of 1600)
// came from a cp.async kernel of 8.0 µs per launch: gpt2xl_request 9.5 → 8.5 ms.
#include <cuda.h>

#include <algorithm>

#include "kernels.h"
#include "q8_common.cuh"
#include "q8_stage.cuh"
#include "q8_tma.cuh"

namespace dj {

namespace {

constexpr int kWarps = kGemvWarps;
constexpr int kThreads = kGemvThreads;
constexpr int kItemK = kTmaItemK;
constexpr int kCodeBytes = 16 * kItemK;             // 16 rows × 128 code bytes, two 1024-byte swizzle atoms
constexpr int kScaleBytes = 16 * 16;                // 16 rows × 4 block scales
constexpr int kItemBytes = kCodeBytes + kScaleBytes;
constexpr int kMaxDepth = 4;
constexpr int kChunk = 16;                          // tiles × activation rows between two barriers
constexpr int kSpinLimit = 1 << 22;                 // polls of one item's barrier before the kernel gives up on it
constexpr int kErrTmaWait = 330;                    // device error code: an item never arrived

struct GemvTmaParams {
    CUtensorMap codes, scales, codes2, scales2;     // boxes of 8 rows; the second pair is the SwiGLU up projection
    Q8View w, w2;                   // the same weights, for the PLAIN form
    const float* x; int ldx;
    const float* gamma; const float* beta; float eps;      // beta: LayerNorm instead of RMSNorm
    const float* bias; const float* bias2;
    const float* residual; int ldr;
    float* out; int ldo;
    int K, N, M, act;               // act 1: GELU behind the bias
    int share, extra;               // granules of 8 rows per block; the first `extra` blocks have one more
    int depth, chunk;               // ring items per warp; tiles between two barriers
    int* error;
    unsigned long long* trace;
};

__device__ __noinline__ float gelu_call(float v) { return gelu_ref(v); }

// NM = 2 takes three or four activation rows in one pass over the weights (a second MMA per block).
// PLAIN: rows, gain and shift by single values; a warp copies its items itself, 16 bytes a lane and copy, laid out as the boxes are.
template <bool SWIGLU, int NM, bool GPT, bool PLAIN>
__global__ void __launch_bounds__(kThreads, 2) k_q8_gemv_tma(const __grid_constant__ GemvTmaParams p) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) unsigned long long s_bar[kWarps * kMaxDepth];
    __shared__ __align__(16) float s_mean[GPT ? 4 * kWarps : 4];
    __shared__ __align__(16) float s_ss[4 * kWarps]; // the warps' parts of Σx² per activation row (RMSNorm at the output)
    // layout (from a 1024-byte boundary, which the swizzle pattern wants): code rings [warps][depth][2048], scale rings
    // [warps][depth][256], digits int8 [3M][K+pad], block scales fp32 [M][K/32], sums [tiles of a chunk][M][16 rows][warps]
    const uint32_t raw_s = smem_u32(smem_raw);
    unsigned char* const smem = smem_raw + (((raw_s + 1023u) & ~1023u) - raw_s);
    const int nGroups = (p.K + kItemK - 1) / kItemK, nBlocks = nGroups * 4, ldxs = nGroups * kItemK + kGemvXsPad;
    unsigned char* const ringS = smem + (size_t)kWarps * p.depth * kCodeBytes;
    int8_t* const xd = reinterpret_cast<int8_t*>(ringS + (size_t)kWarps * p.depth * kScaleBytes);
    float* const xsc = reinterpret_cast<float*>(reinterpret_cast<unsigned char*>(xd) + (size_t)kGemvColsPerRow * p.M * ldxs);
    float* const s_part = xsc + (size_t)p.M * nBlocks;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    const bool tracing = p.trace != nullptr && blockIdx.x == 0 && tid == 0;
    if (tracing) { p.trace[0] = gtime(); p.trace[6] = 0ull; }
    // this block's granules; a tile is two of them (SwiGLU: one of the gate and the same of the up projection)
    const int bx = blockIdx.x, granules = p.share + (bx < p.extra), row0 = (bx * p.share + min(bx, p.extra)) * 8;
    const int tiles = SWIGLU ? granules : (granules + 1) / 2;

    const uint32_t myC = smem_u32(smem) + (uint32_t)(warp * p.depth) * kCodeBytes;
    const uint32_t myS = smem_u32(ringS) + (uint32_t)(warp * p.depth) * kScaleBytes;
    const uint32_t myBar = smem_u32(&s_bar[warp * kMaxDepth]);
    if (lane < p.depth) mbar_init(myBar + 8 * lane, PLAIN ? 32 : 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    __syncwarp();

    // flat (tile, group) sequence of this warp; rows past N are filled with zeros by the copy engine and never stored, the second
    // half of a tile that is not this block's holds anything and is not stored either
    int itile = 0, igrp = warp, islot = 0;
    auto issue_next = [&]() {
        if (igrp >= nGroups || itile >= tiles) return;
        if (PLAIN) {                                 // rows past N and columns past the row are zeros here too
            const uint32_t bar = myBar + 8 * islot, dc = myC + (uint32_t)islot * kCodeBytes, ds = myS + (uint32_t)islot * kScaleBytes;
            const int row = row0 + itile * (SWIGLU ? 8 : 16);
            auto source = [&](int r, int& n) -> const Q8View& { n = row + (SWIGLU ? r & 7 : r); return SWIGLU && r >= 8 ? p.w2 : p.w; };
#pragma unroll
            for (int i = 0; i < 4; i++) {            // piece c of row r sits at r · 128 + ((c ^ (r & 7)) · 16)
                const int r = i * 4 + (lane >> 3), c = lane & 7, k = igrp * kItemK + c * 16;
                int n;
                const Q8View& w = source(r, n);
                const bool on = n < p.N && k < p.K;
                cp_async16_zfill(dc + r * kItemK + ((c ^ (r & 7)) << 4), w.codes + (on ? (size_t)n * w.Kp + k : 0), on);
            }
            if (lane < 16) {
                int n;
                const Q8View& w = source(lane, n);
                cp_async16_zfill(ds + lane * 16, w.scales + (n < p.N ? (size_t)n * w.nb + igrp * 4 : 0), n < p.N);
            }
            cp_async_arrive(bar);
        } else if (lane == 0) {
            const uint32_t bar = myBar + 8 * islot, dc = myC + (uint32_t)islot * kCodeBytes, ds = myS + (uint32_t)islot * kScaleBytes;
            const int row = row0 + itile * (SWIGLU ? 8 : 16);
            if (SWIGLU) {
                mbar_arrive_expect_tx(bar, kItemBytes);
                tma_box(dc, &p.codes, igrp * kItemK, row, bar);
                tma_box(dc + kCodeBytes / 2, &p.codes2, igrp * kItemK, row, bar);
                tma_box(ds, &p.scales, igrp * 4, row, bar);
                tma_box(ds + kScaleBytes / 2, &p.scales2, igrp * 4, row, bar);
            } else {
                const bool half = 2 * itile + 1 == granules;
                mbar_arrive_expect_tx(bar, half ? kItemBytes / 2 : kItemBytes);
                tma_box(dc, &p.codes, igrp * kItemK, row, bar);
                if (!half) tma_box(dc + kCodeBytes / 2, &p.codes, igrp * kItemK, row + 8, bar);
                tma_box(ds, &p.scales, igrp * 4, row, bar);
                if (!half) tma_box(ds + kScaleBytes / 2, &p.scales, igrp * 4, row + 8, bar);
            }
        }
        igrp += kWarps;
        if (igrp >= nGroups) { igrp = warp; itile++; }
        islot = islot + 1 == p.depth ? 0 : islot + 1;
    };
    // Weights never depend on the previous kernel, so streaming starts before the wait.
#pragma unroll 1
    for (int d = 0; d < p.depth; d++) issue_next();
    pdl_launch_dependents();
    if (tracing) p.trace[1] = gtime();
    // the norm's gain is a weight as well
    constexpr int kAhead = 4;                        // groups of a warp in registers
    float4 xv[kAhead], gv[kAhead];
    auto ld4 = [&](const float* q, int grp) {        // zeros behind the row's end
        const int k = grp * kItemK + lane * 4;
        if (k >= p.K) return make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        return PLAIN ? make_float4(q[k], q[k + 1], q[k + 2], q[k + 3]) : *reinterpret_cast<const float4*>(q + k);
    };
    auto load_gain = [&]() {
#pragma unroll
        for (int u = 0; u < kAhead; u++)
            if (p.gamma && warp + kWarps * u < nGroups) gv[u] = ld4(p.gamma, warp + kWarps * u);
    };
    load_gain();
    pdl_wait();
    if (tracing) p.trace[2] = gtime();

    auto sum8 = [](const float* q) {                 // in warp order
        const float4 a = *reinterpret_cast<const float4*>(q), b = *reinterpret_cast<const float4*>(q + 4);
        return ((((((a.x + a.y) + a.z) + a.w) + b.x) + b.y) + b.z) + b.w;
    };
    // activations → digit columns in the MMA fragment's order; every warp converts the groups it consumes and goes on by itself, the
    // next row's first groups on their way while it converts a row's last
    auto load_row = [&](const float* xrow) {
#pragma unroll
        for (int u = 0; u < kAhead; u++)
            if (warp + kWarps * u < nGroups) xv[u] = ld4(xrow, warp + kWarps * u);
    };
    load_row(p.x);
    const int j8 = lane & 7, pos = j8 < 4 ? 8 * j8 : 8 * (j8 - 4) + 4;
#pragma unroll 1
    for (int m = 0; m < p.M; m++) {
        const float* xrow = p.x + (size_t)m * p.ldx;
        int8_t* const dcol = xd + (size_t)(kGemvColsPerRow * m) * ldxs;
        float* const xscRow = xsc + (size_t)m * nBlocks;
        float ss = 0.0f, mean = 0.0f, inv = 1.0f;
        if (GPT && p.beta) {                         // LayerNorm1D (norm/LayerNorm1D.java:34-71): the row's mean, then its biased variance, over the block
#pragma unroll 1
            for (int pass = 0; pass < 2; pass++) {
                float part = 0.0f;
                auto add = [&](const float4& v, int grp) {
                    if (grp * kItemK + lane * 4 >= p.K) return;
                    const float d[4] = {v.x - mean, v.y - mean, v.z - mean, v.w - mean};
#pragma unroll
                    for (int e = 0; e < 4; e++) part = pass ? fmaf(d[e], d[e], part) : part + d[e];
                };
#pragma unroll
                for (int u = 0; u < kAhead; u++)
                    if (warp + kWarps * u < nGroups) add(xv[u], warp + kWarps * u);
#pragma unroll 1
                for (int grp = warp + kWarps * kAhead; grp < nGroups; grp += kWarps) add(ld4(xrow, grp), grp);
                for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
                float* const to = (pass ? s_ss : s_mean) + m * kWarps;
                if (lane == 0) to[warp] = part;
                __syncthreads();
                const float all = sum8(to) * (1.0f / (float)p.K);
                if (pass) inv = __frcp_rn(sqrtf(all + p.eps)); else mean = all;
            }
        }
#pragma unroll 1
        for (int g0 = warp; g0 < nGroups; g0 += kWarps * kAhead) {
#pragma unroll
            for (int u = 0; u < kAhead; u++) {
                const int grp = g0 + kWarps * u;
                if (grp >= nGroups) break;                           // warp-uniform
                float4 v = xv[u];
                if (GPT && p.beta) {                 // (the gain is zero behind the row's end)
                    const float4 b = ld4(p.beta, grp);
                    v = make_float4(((v.x - mean) * inv) * gv[u].x + b.x, ((v.y - mean) * inv) * gv[u].y + b.y, ((v.z - mean) * inv) * gv[u].z + b.z,
                                    ((v.w - mean) * inv) * gv[u].w + b.w);
                }
                gemv_digits4(v, gv[u], p.gamma != nullptr && !(GPT && p.beta), ss, dcol + grp * kItemK + (lane >> 3) * 32 + pos, ldxs, j8 == 0,
                             xscRow + grp * 4 + (lane >> 3));
                const bool more = grp + kWarps * kAhead < nGroups;
                if (more || m + 1 < p.M) {
                    const int to = more ? grp + kWarps * kAhead : warp + kWarps * u;
                    xv[u] = ld4(more ? xrow : xrow + p.ldx, to);
                    if (p.gamma && nGroups > kWarps * kAhead) gv[u] = ld4(p.gamma, to);
                }
            }
        }
        if (p.gamma && !(GPT && p.beta)) {
            for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
            if (lane == 0) s_ss[m * kWarps + warp] = ss;
        }
    }
    __syncwarp();
    if (tracing) p.trace[3] = gtime();

    // lane (g,t) feeds column g of MMA q: activation row 2q + g/4, digit g%4 (digit 3 does not exist)
    bool hasCol[NM]; const unsigned char* xcol[NM]; const float* myxsc[NM];
    float acc[NM][4];
#pragma unroll
    for (int q = 0; q < NM; q++) {
        const int mrow = 2 * q + (g >> 2);
        hasCol[q] = mrow < p.M && (g & 3) != 3;
        xcol[q] = reinterpret_cast<const unsigned char*>(xd) + (size_t)(hasCol[q] ? kGemvColsPerRow * mrow + (g & 3) : 0) * ldxs + t * 8;
        // the lane's two result columns 2t, 2t+1 belong to activation row 2q + t/2
        const int rrow = 2 * q + (t >> 1);
        myxsc[q] = xsc + (size_t)(rrow < p.M ? rrow : 0) * nBlocks;
    }
    // ldmatrix.x4 addresses: lanes 0-7 rows 0-7 of the block's first 16-byte chunk, 8-15 rows 8-15 of it, 16-23 and
    // 24-31 the same rows of the second chunk; chunk c of row r sits at r·128 + ((c ^ (r & 7)) · 16)
    const int lrow = (lane & 7) + ((lane >> 3) & 1) * 8;
    const uint32_t lmBase = (uint32_t)lrow * 128u;
    const uint32_t lmChunk = (uint32_t)((lane >> 4) ^ (lrow & 7));
    int cslot = 0, limit = kSpinLimit;
    uint32_t phases = 0;
    const int chunk = p.chunk;
#pragma unroll 1
    for (int tile0 = 0; tile0 < tiles; tile0 += chunk) {
        const int many = min(chunk, tiles - tile0);
        // output o of the chunk: tile o / (M·rows), activation row, row; its operands are fetched ahead of the tiles
        constexpr int kRows = SWIGLU ? 8 : 16;
        const int perTile = p.M * kRows, ot = tid / perTile, om = (tid - ot * perTile) / kRows, orow = tid % kRows;
        const int n = row0 + (tile0 + ot) * kRows + orow;
        const bool mine = ot < many && n < p.N && n < row0 + granules * 8;
        float bias = 0.0f, other = 0.0f;
        if (mine) {
            if (p.bias) bias = p.bias[n];
            if (SWIGLU) { if (p.bias2) other = p.bias2[n]; }
            else if (p.residual) other = p.residual[(size_t)om * p.ldr + n];
        }
#pragma unroll 1
        for (int i = 0; i < many; i++) {
#pragma unroll
            for (int q = 0; q < NM; q++) acc[q][0] = acc[q][1] = acc[q][2] = acc[q][3] = 0.0f;
#pragma unroll 1
            for (int grp = warp; grp < nGroups; grp += kWarps) {
                const uint32_t bar = myBar + 8 * cslot;
                const uint32_t parity = (phases >> cslot) & 1u;
                bool ready = mbar_try_wait(bar, parity);
#pragma unroll 1
                for (int spin = 0; !ready && spin < limit; spin++) ready = mbar_try_wait(bar, parity);
                if (!ready) {                               // never on a healthy device: flag it, stop waiting long, keep the control flow
                    if (lane == 0) atomicCAS(p.error, 0, kErrTmaWait);
                    limit = 64;
                }
                phases ^= 1u << cslot;
                const uint32_t sc = myC + (uint32_t)cslot * kCodeBytes;
                const unsigned char* ss = ringS + ((size_t)warp * p.depth + cslot) * kScaleBytes;
                const float4 s0 = *reinterpret_cast<const float4*>(ss + g * 16);            // row g: its four block scales
                const float4 s1 = *reinterpret_cast<const float4*>(ss + (g + 8) * 16);      // row g+8
                const float s0v[4] = {s0.x, s0.y, s0.z, s0.w}, s1v[4] = {s1.x, s1.y, s1.z, s1.w};
                float xsv[NM][4];
#pragma unroll
                for (int q = 0; q < NM; q++) {
                    const float4 v = *reinterpret_cast<const float4*>(myxsc[q] + grp * 4);
                    xsv[q][0] = v.x; xsv[q][1] = v.y; xsv[q][2] = v.z; xsv[q][3] = v.w;
                }
#pragma unroll
                for (int b = 0; b < 4; b++) {
                    uint32_t a[4];
                    ldmatrix_x4(a, sc + lmBase + ((lmChunk ^ (uint32_t)(2 * b)) << 4));
                    const int blk = grp * 4 + b;
#pragma unroll
                    for (int q = 0; q < NM; q++) {
                        uint2 xb = make_uint2(0u, 0u);
                        if (hasCol[q]) xb = *reinterpret_cast<const uint2*>(xcol[q] + blk * 32);
                        int cc[4] = {0, 0, 0, 0};
                        mma_s8_16832(cc, a[0], a[1], a[2], a[3], xb.x, xb.y);
                        const float f0 = s0v[b] * xsv[q][b], f1 = s1v[b] * xsv[q][b];
                        acc[q][0] = fmaf(f0, int_to_float_exact(cc[0]), acc[q][0]);
                        acc[q][1] = fmaf(f0, int_to_float_exact(cc[1]), acc[q][1]);
                        acc[q][2] = fmaf(f1, int_to_float_exact(cc[2]), acc[q][2]);
                        acc[q][3] = fmaf(f1, int_to_float_exact(cc[3]), acc[q][3]);
                    }
                }
                __syncwarp();           // every lane has read the slot before lane 0 hands it to the copy engine again
                issue_next();
                cslot = cslot + 1 == p.depth ? 0 : cslot + 1;
            }
            // the warp's sums, digits recombined: lanes of even t hold the upper two digits of activation row 2q + t/2, their neighbours the last
#pragma unroll
            for (int q = 0; q < NM; q++) {
                const float d0 = __shfl_down_sync(0xffffffffu, acc[q][0], 1), d1 = __shfl_down_sync(0xffffffffu, acc[q][2], 1);
                const int m = 2 * q + (t >> 1);
                if ((t & 1) == 0 && m < p.M) {
                    float* to = s_part + ((i * p.M + m) * 16 + g) * kWarps + warp;
                    to[0] = fmaf(acc[q][0], 65536.0f, fmaf(acc[q][1], 256.0f, d0));
                    to[8 * kWarps] = fmaf(acc[q][2], 65536.0f, fmaf(acc[q][3], 256.0f, d1));
                }
            }
        }
        if (tracing && tile0 == 0) p.trace[4] = gtime();
        __syncthreads();
        if (mine) {
            const float* from = s_part + ((ot * p.M + om) * 16 + orow) * kWarps;
            float v = sum8(from), inv = 1.0f;
            if (p.gamma && !(GPT && p.beta)) {
                inv = __frcp_rn(sqrtf(sum8(s_ss + om * kWarps) * (1.0f / (float)p.K) + p.eps));
                v *= inv;
            }
            if (p.bias) v += bias;
            if (GPT && p.act == 1) v = gelu_call(v);
            if (SWIGLU) {
                float u = sum8(from + 8 * kWarps) * inv;
                if (p.bias2) u += other;
                const float sig = 1.0f / (1.0f + expf(-v));
                v = (v * sig) * u;                   // SiLU(gate) ⊙ up
            } else if (p.residual) v += other;
            p.out[(size_t)om * p.ldo + n] = v;
        }
        if (tile0 + chunk < tiles) __syncthreads();
    }
    if (tracing) p.trace[5] = gtime();
    if (p.trace != nullptr && tid == 0) atomicMax(p.trace + 6, gtime());
}

size_t tma_smem_bytes(int K, int M, int depth, int chunk) {
    const size_t groups = (K + kItemK - 1) / kItemK;
    return 1024 + (size_t)kWarps * depth * kItemBytes + (size_t)kGemvColsPerRow * M * (groups * kItemK + kGemvXsPad) + M * groups * 16 +
           (size_t)chunk * M * 16 * kWarps * 4;
}
constexpr size_t kSmemHalf = 111 * 1024;         // two blocks per SM
constexpr size_t kSmemWhole = 224 * 1024;        // a block with its SM to itself

// Ring items per warp and tiles between two barriers beside the digits of M rows, so that two blocks share an SM; depth 0: they
// do not fit.  Several rows that need a whole SM are taken in passes of fewer rows instead, or with shorter rings: launch to launch,
// against one block per SM, 4 rows of 4096 → 12288 28.2 → 18.3 µs (two barriers in place of one), 2 of 11008 → 4096 25.4 → 15.9 (two ring
// items), 4 of it 41.5 → 31.1 (two passes).  A single row may take an SM for one block.
struct Ring { int depth, chunk; };
Ring ring_for(int K, int M) {
    const int full = kChunk / M;
    for (int d = kMaxDepth; d >= 2; d--)
        for (int c = full; c >= 1; c = d == kMaxDepth ? 0 : c / 2)
            if (tma_smem_bytes(K, M, d, c) <= kSmemHalf) return {d, c};
    return {M == 1 && tma_smem_bytes(K, M, 3, full) <= kSmemWhole ? 3 : 0, full};
}

template <bool SWIGLU, int NM, bool GPT, bool PLAIN>
void launch_tma(GemvTmaParams& p, cudaStream_t s) {
    static bool attrSet = false;
    if (!attrSet) {
        DJ_CUDA_CHECK(cudaFuncSetAttribute(k_q8_gemv_tma<SWIGLU, NM, GPT, PLAIN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemWhole));
        attrSet = true;
    }
    const int granules = (p.N + 7) / 8, gx = std::min(SWIGLU ? granules : (granules + 1) / 2, 2 * g_num_sms);
    p.share = granules / gx; p.extra = granules % gx;
    const Ring r = ring_for(p.K, p.M);
    p.depth = r.depth; p.chunk = r.chunk;
    launch_k(k_q8_gemv_tma<SWIGLU, NM, GPT, PLAIN>, dim3(gx), dim3(kThreads), tma_smem_bytes(p.K, p.M, r.depth, r.chunk), s, true, p);
}

}  // namespace

// Tensor maps over one Q8 weight: codes [N][Kp] bytes in boxes of 8 rows × 128 bytes (128-byte swizzle) and
// scales [N][nb] floats in boxes of 8 rows × 4.
bool q8_encode_weight_maps(const Q8View& w, CUtensorMap* codes, CUtensorMap* scales) {
    EncodeTiledFn enc = encode_tiled_fn();
    if (!enc) return false;
    if ((reinterpret_cast<uintptr_t>(w.codes) & 15) != 0 || (reinterpret_cast<uintptr_t>(w.scales) & 15) != 0) return false;
    if (w.Kp % 16 != 0) return false;
    {
        const cuuint64_t dims[2] = {(cuuint64_t)w.Kp, (cuuint64_t)w.N};
        const cuuint64_t strides[1] = {(cuuint64_t)w.Kp};
        const cuuint32_t box[2] = {(cuuint32_t)kItemK, 8u};
        const cuuint32_t estr[2] = {1u, 1u};
        if (enc(codes, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<int8_t*>(w.codes), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return false;
    }
    {
        const cuuint64_t dims[2] = {(cuuint64_t)w.nb, (cuuint64_t)w.N};
        const cuuint64_t strides[1] = {(cuuint64_t)w.nb * 4};
        const cuuint32_t box[2] = {4u, 8u};
        const cuuint32_t estr[2] = {1u, 1u};
        if (enc(scales, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(w.scales), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return false;
    }
    return true;
}

namespace {

template <bool PLAIN>
void launch_rows(GemvTmaParams& p, bool swiglu, bool gpt, cudaStream_t s) {
    if (swiglu) { if (p.M > 2) launch_tma<true, 2, false, PLAIN>(p, s); else launch_tma<true, 1, false, PLAIN>(p, s); }
    else if (gpt) { if (p.M > 2) launch_tma<false, 2, true, PLAIN>(p, s); else launch_tma<false, 1, true, PLAIN>(p, s); }
    else { if (p.M > 2) launch_tma<false, 2, false, PLAIN>(p, s); else launch_tma<false, 1, false, PLAIN>(p, s); }
}

}  // namespace

// Returns false when the shape is outside this kernel's domain: a ring beside the digits of one row, whole blocks (the FMA kernel rounds
// less than the digits do: 1.0e-7 against 2e-7 of the result, and other lengths stay with it).
bool launch_q8_gemv_tma(const Q8LinearArgs& a, cudaStream_t s) {
    const int K = a.w.K;
    const bool swiglu = a.w2.codes != nullptr, gpt = a.beta != nullptr || a.act != 0;
    if (K % 32 != 0 || g_dev_error == nullptr || (swiglu && (gpt || a.w2.K != K || a.w2.Kp != a.w.Kp || a.w2.N != a.w.N))) return false;
    if (ring_for(K, 1).depth == 0) return false;
    GemvTmaParams p = {};
    // rows that do not come in 16-byte pieces, the setting that leaves tensor copies out, a driver without them
    const bool pieces = ((reinterpret_cast<uintptr_t>(a.x) | reinterpret_cast<uintptr_t>(a.gamma) | reinterpret_cast<uintptr_t>(a.beta)) & 15) == 0 && (a.M == 1 || a.ldx % 4 == 0);
    bool plain = !pieces || g_gemv_mode < 2 || !q8_encode_weight_maps(a.w, &p.codes, &p.scales);
    if (!plain && swiglu) plain = !q8_encode_weight_maps(a.w2, &p.codes2, &p.scales2);
    p.w = a.w; p.w2 = a.w2;
    for (int m0 = 0; m0 < a.M;) {
        int rows = std::min(a.M - m0, 4);            // 8 MMA columns = 2 activation rows × (3 digits + 1 unused); 3-4 rows take a second MMA
        while (rows > 1 && ring_for(K, rows).depth == 0) rows--;
        p.x = a.x + (size_t)m0 * a.ldx; p.ldx = a.ldx; p.gamma = a.gamma; p.beta = a.gamma ? a.beta : nullptr; p.eps = a.eps;
        p.bias = a.bias; p.bias2 = a.bias2; p.act = a.act;
        p.residual = a.residual ? a.residual + (size_t)m0 * a.ldr : nullptr; p.ldr = a.ldr;
        p.out = a.out + (size_t)m0 * a.ldo; p.ldo = a.ldo;
        p.K = K; p.N = a.w.N; p.M = rows;
        p.error = g_dev_error;
        p.trace = trace_slot();
        if (plain) launch_rows<true>(p, swiglu, gpt, s); else launch_rows<false>(p, swiglu, gpt, s);
        m0 += rows;
    }
    return true;
}

}  // namespace dj
