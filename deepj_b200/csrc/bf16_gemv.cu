// Projections of 1-16 activation rows with bf16 weights, passes of up to four rows: out = stage(x) · Wᵀ, fp32 products and sums.
//
// HBM-bound while it streams, but one layer's weights are 8 ... 50 MB, 1 ... 8 µs, and a launch between two others costs 1.5 µs at
// least: the dependency wait and the way of the row into every SM.  Two things decide how much more it costs.
//   * Weights on their way before the wait.  One block of 8 warps per SM, each warp with a ring of 4 KB items, a tensor
//     copy each; with one row at most half of an SM's shared memory and registers, so that the next projection's
//     block moves in and fills its own rings while this one multiplies.  (A thread issues a copy every 45 ns: with
//     512 bytes each that was a third of the bandwidth.)
//   * Few instructions.  A launch runs most of its code once, and fetching 1 KB of code that another kernel has displaced takes 0.15 µs:
//     rolled loops, sizes divided on the host, unusual forms out of line.
// Measured inside decoding steps of width 2048, from the dependency wait to the last block's end (the kernel before this one, which
// held three steps of weights in registers: launch to launch): 46 MB gate and up 9.3 µs (12.6), 23 MB down 5.7 and 8.4 MB out
// 5.1 (8.5 on average), head of 131 MB 21.2 µs = 6.2 TB/s.  Tried: asking the items behind the ring into L2 ahead of the wait (2-8 per
// warp: 2-4 % slower steps).
// Without tensor maps (PLAIN: a driver that gives none, or the setting that leaves tensor copies out) the lanes of a warp fill its ring with
// cp.async, 16 bytes each; everything else is the same.
// An item is ROWS weight rows × COLS columns.  A block owns a run of row groups; the items of that run, group by group, are cut
// into equal parts, one per warp, so that narrow weights keep every warp busy too.  A warp sums a row group for as long as
// its part stays in it and leaves the sum in shared memory; the end of the kernel adds the parts of a group in warp order.
#include "row_operand.cuh"
#include "tc_common.cuh"

#include <algorithm>

namespace dj {
namespace {

constexpr int kRgItem = 4096;
constexpr int kRgSmemMax = 224 * 1024;           // dynamic shared memory of a block that has its SM to itself
constexpr int kRgSmemHalf = 111 * 1024;          // of two blocks that share one
constexpr int kRgMaxDepth = 6, kRgMaxWarps = 16;
constexpr int kRgSpinLimit = 1 << 22;            // polls of a barrier before the kernel gives up on it
constexpr int kRgMaxGroups = 512;                // row groups of a block, at most
constexpr int kErrRingWait = 333;                // device error code: a copy never arrived
constexpr int kPieces = 4;                       // 16-byte pieces of a row's gain, gate or base that a thread holds while the row is on its way

__device__ __forceinline__ float bf_lo(uint32_t u) { return __uint_as_float(u << 16); }
__device__ __forceinline__ float bf_hi(uint32_t u) { return __uint_as_float(u & 0xffff0000u); }

// How table-routed experts (blockIdx.y = token row) enter: not at all, as row groups of the token's experts one after another
// (one output row per slot), or one after another along the reduction (outputs are the mean over the slots).
constexpr int kPlain = 0, kExpertRows = 1, kExpertSum = 2;

struct RgParams {
    CUtensorMap map;                             // boxes of an item, four columns to an element
    const __nv_bfloat16* w; int wRows;           // the same weight, for the PLAIN form
    RowOperand a, b;
    int rows;                                    // activation rows of this pass, at most MR
    int N, Kp, K1p;                              // K1p: first column of segment b
    int items, groups;                           // items per row group and weight matrix, row groups per matrix
    int share, extra;                            // row groups of a block; the first `extra` blocks have one more
    int warps, depth, maxGroups;                 // warps with a ring; items in it; row groups that a warp can touch
    // where a warp's part begins, in blocks of `share` and of share + 1 row groups: item, and the row group and the item in it
    int first[2][kRgMaxWarps + 1];
    unsigned short firstGroup[2][kRgMaxWarps], firstItem[2][kRgMaxWarps];
    int vec;                                     // bits 0, 1: segment a, b travels in 16-byte pieces
    int len, normWarps, normStep; unsigned lenMagic;     // segment a's norm: pieces per group, warps of a group, pieces of a warp, for p / len
    const float* residual; int ldr;
    float* out; int ldo;
    int gluRow; float limit; float* glu; int ldglu;
    float softcap; const float* bias; int pair;
    int early;                                   // experts: the tables may be read before the dependency wait
    int trigger;                                 // the next kernel may start before this one's wait
    const float* tok; const float* table; int top, vocab, expertRows;
    int* error;
};

// Sums v[i] over the warp for V values at once (V a power of two): lane l ends up with the sum of v[l / (32 / V)].
template <int V>
__device__ __forceinline__ float warp_sum_many(float (&v)[V], int lane) {
#pragma unroll
    for (int h = V / 2, o = 16; h >= 1; h >>= 1, o >>= 1) {
        const bool upper = (lane & o) != 0;
#pragma unroll
        for (int i = 0; i < h; i++) {
            const float give = upper ? v[i] : v[i + h], keep = upper ? v[i + h] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
    }
#pragma unroll
    for (int o = 16 / V; o >= 1; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
    return v[0];
}
__device__ __forceinline__ bool bounded_wait(uint32_t bar, uint32_t parity, int& limit, int* error) {
    bool ready = mbar_try_wait(bar, parity);
#pragma unroll 1
    for (int spin = 0; !ready && spin < limit; spin++) ready = mbar_try_wait(bar, parity);
    if (!ready) {                                // never on a healthy device: flag it, stop waiting long, keep the control flow
        atomicCAS(error, 0, kErrRingWait);
        limit = 64;
    }
    return ready;
}

// A segment whose columns do not come in aligned 16-byte pieces: one by one.
__device__ __noinline__ void stage_columns(const RowOperand* seg, int m, float* scratch, float* xs, bool keep) {
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, len = seg->groups > 0 ? seg->k / seg->groups : seg->k;
    const float* x = seg->x + (size_t)m * seg->ldx;
#pragma unroll 4
    for (int k = tid; k < seg->k; k += nt) xs[k] = x[k];
    if (seg->groups > 0) {
        __syncthreads();
#pragma unroll 1
        for (int g = tid >> 5; g < seg->groups; g += nt >> 5) {
            float ss = 0.0f;
#pragma unroll 1
            for (int k = g * len + lane; k < (g + 1) * len; k += 32) ss = fmaf(xs[k], xs[k], ss);
            for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
            if (lane == 0) scratch[g] = 1.0f / sqrtf(ss / (float)len + seg->eps);
        }
        __syncthreads();
    }
#pragma unroll 1
    for (int k = tid; k < seg->k; k += nt) {
        float v = xs[k];
        if (seg->groups > 0) v = (v * scratch[k / len]) * seg->gamma[k];
        if (seg->gate) v *= sigmoid_f(seg->gate[(size_t)m * seg->ldg + k]);
        if (seg->base) {
            v = fmaf(seg->mult, v, seg->base[(size_t)m * seg->ldbase + k]);
            if (keep && seg->sum) seg->sum[(size_t)m * seg->ldsum + k] = v;
        }
        xs[k] = v;
    }
}
__device__ __noinline__ float4 gated4(float4 v, float4 g) {
    return make_float4(v.x * sigmoid_f(g.x), v.y * sigmoid_f(g.y), v.z * sigmoid_f(g.z), v.w * sigmoid_f(g.w));
}
__device__ __forceinline__ const float* more_of(const RowOperand& seg, int m) {
    return seg.gate ? seg.gate + (size_t)m * seg.ldg : seg.base ? seg.base + (size_t)m * seg.ldbase : nullptr;
}

template <int MR, int ROWS, int WARPS, int EXPERTS, bool PLAIN>
__global__ void __launch_bounds__(WARPS * 32, MR == 1 ? 2 : 1) k_bf16_gemv(const __grid_constant__ RgParams p) {
    constexpr int COLS = kRgItem / 2 / ROWS, V = MR * ROWS, THREADS = WARPS * 32;
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ __align__(8) unsigned long long s_bar[WARPS * kRgMaxDepth + 1];
    __shared__ short s_owner[kRgMaxGroups];      // of a row group: the sum of the warp in which it begins
    __shared__ __align__(16) int s_rest[WARPS];  // of a warp: the row group that it took up from the warp before it, -1: none
    // rings [warps][depth][4096], rows [MR][row], then the warps' sums [warps][maxGroups][V], whose bytes first serve the norm
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nIt = p.items * (EXPERTS == kExpertSum ? p.top : 1), row = nIt * COLS;
    const int live = MR == 1 ? 1 : p.rows;       // the others' columns hold anything, as do their sums, which nothing reads
    unsigned char* const ring = smem + (size_t)warp * p.depth * kRgItem;
    float* const xs = reinterpret_cast<float*>(smem + (size_t)p.warps * p.depth * kRgItem);
    float* const parts = xs + MR * row;
    const uint32_t ringAddr = smem_u32(ring), bars = smem_u32(&s_bar[warp * kRgMaxDepth]), xbar = smem_u32(&s_bar[WARPS * kRgMaxDepth]);
    if (lane < p.depth) mbar_init(bars + 8 * lane, PLAIN ? 32 : 1);
    if (tid == 0) mbar_init(xbar, 1);
    if (tid < WARPS) s_rest[tid] = -1;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    __syncwarp();

    // this block's row groups [g0, g0 + groups), this warp's items
    const int bx = blockIdx.x, more = bx < p.extra, g0 = bx * p.share + min(bx, p.extra), groups = p.share + more;
    const int m0 = EXPERTS == kPlain ? 0 : (int)blockIdx.y;
    int left = p.first[more][warp + 1] - p.first[more][warp], it = p.firstItem[more][warp];
    // the next item to request: row group, item of it, ring slot
    int fLeft = left, fi = it, fg = g0 + p.firstGroup[more][warp], fs = 0, id = 0, slot = -1, slotRow = 0;
    auto fetch = [&] {
        fLeft--;
        if (PLAIN || lane == 0) {
            int k = fi * COLS, n = fg * ROWS;
            if (EXPERTS != kPlain) {
                const int s = EXPERTS == kExpertRows ? fg / p.groups : fi / p.items;
                if (s != slot) { slot = s; slotRow = (int)p.table[(size_t)id * p.top + s] * p.expertRows; }
                if (EXPERTS == kExpertRows) n -= s * p.groups * ROWS; else k -= s * p.items * COLS;
            }
            const uint32_t bar = bars + 8 * fs;
            if (PLAIN) {
#pragma unroll 4
                for (int i = lane; i < kRgItem / 16; i += 32) {      // piece i % (COLS / 8) of the item's row i / (COLS / 8)
                    const int wr = slotRow + n + i / (COLS / 8), wk = k + i % (COLS / 8) * 8;
                    const bool on = wr >= 0 && wr < p.wRows && wk < p.Kp;
                    cp_async16_zfill(ringAddr + fs * kRgItem + i * 16, p.w + (on ? (size_t)wr * p.Kp + wk : 0), on);
                }
                cp_async_arrive(bar);
            } else {
                mbar_arrive_expect_tx(bar, kRgItem);                 // what lies outside the weight counts, and comes as zeros
                tma_box(ringAddr + fs * kRgItem, &p.map, k / 4, slotRow + n, bar);
            }
        }
        if (++fi == nIt) { fi = 0; fg++; }
        if (++fs == p.depth) fs = 0;
    };
    const bool ahead = EXPERTS == kPlain || p.early;
#pragma unroll 1
    for (int half = 0; half < 2; half++) {
        if (half == 1) {
            if (p.trigger) pdl_launch_dependents();
            pdl_wait();
            if (!p.trigger) pdl_launch_dependents();
        }
        if ((half == 0) != ahead) continue;
        if (EXPERTS != kPlain) id = min(max((int)p.tok[m0], 0), p.vocab - 1);
#pragma unroll 1
        for (int d = 0; d < p.depth && fLeft > 0; d++) fetch();
    }

    // segments: the rows' one or two, or one per slot of a sum over experts
    const int segs = EXPERTS == kExpertSum ? p.top : p.b.k > 0 ? 2 : 1;
    auto column = [&](int s) { return EXPERTS == kExpertSum ? s * p.items * COLS : s ? p.K1p : 0; };
    auto source = [&](int m, int s) { return EXPERTS == kExpertSum ? m0 * p.top + s : m0 + m; };
    if (tid == 0) {
        const uint32_t na = (p.vec & 1) ? p.a.k * 4 : 0, nb = (p.vec & 2) ? p.b.k * 4 : 0;
        mbar_arrive_expect_tx(xbar, live * (EXPERTS == kExpertSum ? segs * na : na + nb));
#pragma unroll 1
        for (int i = 0; i < live * segs; i++) {
            const int m = MR == 1 ? 0 : i / segs, s = i - m * segs;
            const bool second = EXPERTS != kExpertSum && s == 1;
            const RowOperand& seg = second ? p.b : p.a;
            const uint32_t bytes = second ? nb : na;
            if (bytes) bulk_g2s(smem_u32(xs + m * row + column(s)), seg.x + (size_t)source(m, s) * seg.ldx, bytes, xbar);
        }
    }
    // the gain, gate and base of row 0, and the first output's residual, on their way beside the row
    const int n4 = p.a.k >> 2;
    auto ld4 = [](const float* q, int i) { return reinterpret_cast<const float4*>(q)[i]; };
    float4 gain[kPieces], add[kPieces];
    const float* more0 = more_of(p.a, source(0, 0));
    const bool shaped = (p.vec & 1) && (p.a.groups > 0 || more0 != nullptr);
#pragma unroll
    for (int u = 0; u < kPieces; u++) {
        gain[u] = add[u] = make_float4(0, 0, 0, 0);
        if (shaped && tid + u * THREADS < n4) {
            if (p.a.groups > 0) gain[u] = ld4(p.a.gamma, tid + u * THREADS);
            if (more0) add[u] = ld4(more0, tid + u * THREADS);
        }
    }
    // output o of activation row m: weight row n, output row orow
    const int outs = groups * ROWS;
    auto place = [&](int o, int m, int& n, int& orow) {
        n = g0 * ROWS + o;
        orow = m0 + m;
        if (EXPERTS == kExpertRows) {
            orow = m0 * p.top;
            for (; n >= p.groups * ROWS; n -= p.groups * ROWS) orow++;
        }
    };
    float resid = 0.0f;
    if (p.residual && tid < outs) {
        int n, orow; place(tid, 0, n, orow);
        if (n < p.gluRow && n < p.N) resid = p.residual[(size_t)orow * p.ldr + n];
    }
    // columns between and behind the segments
#pragma unroll 1
    for (int i = 0; i < live * segs; i++) {
        const int m = MR == 1 ? 0 : i / segs, s = i - m * segs;
        const int stop = EXPERTS == kExpertSum ? column(s + 1) : s + 1 < segs ? p.K1p : row;
#pragma unroll 1
        for (int k = column(s) + (EXPERTS != kExpertSum && s == 1 ? p.b.k : p.a.k) + tid; k < stop; k += THREADS) xs[m * row + k] = 0.0f;
    }
    int limit = kRgSpinLimit;
    __syncthreads();                             // the barrier is set up for every warp
    bounded_wait(xbar, 0, limit, p.error);
    if (shaped) {
#pragma unroll 1
        for (int m = 0; m < live * (EXPERTS == kExpertSum ? segs : 1); m++) {
            float4* const x4 = reinterpret_cast<float4*>(EXPERTS == kExpertSum ? xs + column(m) : xs + m * row);
            const int src = EXPERTS == kExpertSum ? source(0, m) : source(m, 0);
            const float* mo = more_of(p.a, src);
            float scale = 0.0f;
            if (p.a.groups > 0) {
                if (m > 0) __syncthreads();      // the scratch is used again
                float* const part = parts + p.a.groups;
#pragma unroll 1
                for (int u = warp; u < p.a.groups * p.normWarps; u += WARPS) {
                    int lo = u * p.len, hi = lo + p.len;
                    if (p.normWarps > 1) {
                        int g = 0, r = u;
                        for (; r >= p.normWarps; r -= p.normWarps) g++;
                        lo = g * p.len + r * p.normStep; hi = min(lo + p.normStep, (g + 1) * p.len);
                    }
                    float ss = 0.0f;
#pragma unroll 1
                    for (int q = lo + lane; q < hi; q += 32) {
                        const float4 v = x4[q];
                        ss = fmaf(v.x, v.x, ss); ss = fmaf(v.y, v.y, ss); ss = fmaf(v.z, v.z, ss); ss = fmaf(v.w, v.w, ss);
                    }
                    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
                    if (lane == 0) part[u] = ss;
                }
                __syncthreads();
                auto finish = [&](float ss) { return 1.0f / sqrtf(ss / (float)(4 * p.len) + p.a.eps); };
                if (p.a.groups == 1) {           // every warp on its own
                    float ss = lane < WARPS ? part[lane] : 0.0f;
                    for (int o = WARPS / 2; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
                    scale = __shfl_sync(0xffffffffu, finish(ss), 0);
                } else {
#pragma unroll 1
                    for (int g = tid; g < p.a.groups; g += THREADS) {
                        float ss = 0.0f;
#pragma unroll 1
                        for (int r = 0; r < p.normWarps; r++) ss += part[g * p.normWarps + r];
                        parts[g] = finish(ss);
                    }
                    __syncthreads();
                }
            }
            float* const sum = p.a.sum && bx == 0 ? p.a.sum + (size_t)src * p.a.ldsum : nullptr;
            auto shape = [&](int q, float4 w, float4 b) {
                float4 v = x4[q];
                if (p.a.groups > 0) {
                    const float s = p.a.groups == 1 ? scale : parts[__umulhi((unsigned)q, p.lenMagic)];
                    v = make_float4((v.x * s) * w.x, (v.y * s) * w.y, (v.z * s) * w.z, (v.w * s) * w.w);
                }
                if (p.a.gate) v = gated4(v, b);
                if (p.a.base) {
                    v = make_float4(fmaf(p.a.mult, v.x, b.x), fmaf(p.a.mult, v.y, b.y), fmaf(p.a.mult, v.z, b.z), fmaf(p.a.mult, v.w, b.w));
                    if (sum) reinterpret_cast<float4*>(sum)[q] = v;
                }
                x4[q] = v;
            };
            int q = tid;
            if (m == 0) {
#pragma unroll
                for (int u = 0; u < kPieces; u++, q += THREADS) {
                    if (q >= n4) break;
                    shape(q, gain[u], add[u]);
                }
            }
#pragma unroll 1
            for (; q < n4; q += THREADS) shape(q, p.a.groups > 0 ? ld4(p.a.gamma, q) : make_float4(0, 0, 0, 0), mo ? ld4(mo, q) : make_float4(0, 0, 0, 0));
        }
    }
    if (p.vec != 3) {
#pragma unroll 1
        for (int i = 0; i < live * segs; i++) {
            const int m = MR == 1 ? 0 : i / segs, s = i - m * segs;
            const bool second = EXPERTS != kExpertSum && s == 1;
            if (p.vec & (second ? 2 : 1)) continue;
            stage_columns(second ? &p.b : &p.a, source(m, s), parts, xs + m * row + column(s), bx == 0);
            __syncthreads();
        }
    }
    __syncthreads();

    float acc[V];
#pragma unroll
    for (int i = 0; i < V; i++) acc[i] = 0.0f;
    int cs = 0, held = warp * p.maxGroups, g = p.firstGroup[more][warp];
    bool whole = it == 0;                        // the row group begins in this warp's part
    uint32_t phase = 0;
#pragma unroll 1
    for (; left > 0; left--) {
        bounded_wait(bars + 8 * cs, (phase >> cs) & 1, limit, p.error);
        phase ^= 1u << cs;
        const unsigned char* d = ring + cs * kRgItem + lane * 8;
        const float* xb = xs + it * COLS + lane * 4;
#pragma unroll
        for (int c = 0; c < COLS / 128; c++) {
            uint2 w[ROWS];
#pragma unroll
            for (int r = 0; r < ROWS; r++) w[r] = *reinterpret_cast<const uint2*>(d + c * 256 + r * (COLS * 2));
#pragma unroll
            for (int m = 0; m < MR; m++) {
                const float4 x = *reinterpret_cast<const float4*>(xb + m * row + c * 128);
#pragma unroll
                for (int r = 0; r < ROWS; r++) {
                    float s = acc[m * ROWS + r];
                    s = fmaf(bf_lo(w[r].x), x.x, s); s = fmaf(bf_hi(w[r].x), x.y, s);
                    s = fmaf(bf_lo(w[r].y), x.z, s); s = fmaf(bf_hi(w[r].y), x.w, s);
                    acc[m * ROWS + r] = s;
                }
            }
        }
        __syncwarp();                            // every lane has read the slot before lane 0 hands it to the copy engine again
        if (fLeft > 0) fetch();
        if (++cs == p.depth) cs = 0;
        if (++it == nIt || left == 1) {
            it = 0;
            const float sum = warp_sum_many<V>(acc, lane);
            if (lane % (32 / V) == 0) parts[held * V + lane / (32 / V)] = sum;
            if (lane == 0) {
                if (whole) s_owner[g] = (short)held; else s_rest[warp] = g;
            }
            whole = true;
            held++; g++;
#pragma unroll
            for (int i = 0; i < V; i++) acc[i] = 0.0f;
        }
    }
    __syncthreads();

    // every lane of a warp takes part (the gated pair's other half is the next lane's)
#pragma unroll 1
    for (int m = 0; m < live; m++) {
#pragma unroll 1
        for (int o = tid; o - lane < outs; o += THREADS) {
            const int gr = min(o, outs - 1) / ROWS, at = m * ROWS + o % ROWS;
            float v = parts[s_owner[gr] * V + at];
#pragma unroll
            for (int w = 1; w < WARPS; w++)      // in warp order
                if (s_rest[w] == gr) v += parts[w * p.maxGroups * V + at];
            const float up = __shfl_down_sync(0xffffffffu, v, 1);
            int n, orow; place(o, m, n, orow);
            if (o >= outs || n >= p.N) continue;
            if (n >= p.gluRow) {
                if (((n - p.gluRow) & 1) == 0) p.glu[(size_t)orow * p.ldglu + ((n - p.gluRow) >> 1)] = pair_f(v, up, p.limit, p.pair);
                continue;
            }
            if (EXPERTS == kExpertSum) v /= (float)p.top;
            if (p.bias) v += p.bias[n];
            if (p.residual) v += m == 0 && o == tid ? resid : p.residual[(size_t)orow * p.ldr + n];
            p.out[(size_t)orow * p.ldo + n] = softcap_f(v, p.softcap);
        }
    }
}

// Four columns to an element: a box may be 256 elements wide, an item is up to 1024 columns.
bool encode_items(CUtensorMap* map, const Bf16View& w, int cols, int rows) {
    EncodeTiledFn enc = encode_tiled_fn();
    if (!enc || ((uintptr_t)w.w & 15) != 0 || w.Kp % 8 != 0) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)w.Kp / 4, (cuuint64_t)w.N};
    const cuuint64_t strides[1] = {(cuuint64_t)w.Kp * 2};
    const cuuint32_t box[2] = {(cuuint32_t)cols / 4, (cuuint32_t)rows};
    const cuuint32_t estr[2] = {1u, 1u};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_INT64, 2, const_cast<__nv_bfloat16*>(w.w), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int MR, int ROWS, int WARPS, int EXPERTS, bool PLAIN = false>
bool launch_rg(RgParams& p, const Bf16View& w, int tokens, cudaStream_t s) {
    constexpr int COLS = kRgItem / 2 / ROWS;
    if constexpr (!PLAIN)
        if (g_gemv_mode < 2 || !encode_items(&p.map, w, COLS, ROWS)) return launch_rg<MR, ROWS, WARPS, EXPERTS, true>(p, w, tokens, s);
    p.w = w.w; p.wRows = w.N; p.Kp = w.Kp; p.error = g_dev_error;
    p.items = (w.Kp + COLS - 1) / COLS;
    p.groups = (p.N + ROWS - 1) / ROWS;
    const int groups = p.groups * (EXPERTS == kExpertRows ? p.top : 1), items = p.items * (EXPERTS == kExpertSum ? p.top : 1);
    int gx = 1;
    if (tokens == 1) {
        gx = std::min(groups, g_num_sms * ((groups + g_num_sms * kRgMaxGroups - 1) / (g_num_sms * kRgMaxGroups)));
    } else {                                     // the blocks of all token rows share the SMs: the fewest rounds for the work per block
        double best = 1e30;
        for (int g = 1; g <= std::min(groups, g_num_sms); g++) {
            const double cost = (double)(((long long)tokens * g + g_num_sms - 1) / g_num_sms) * ((groups + g - 1) / g + 1);
            if (cost < best) { best = cost; gx = g; }
        }
        gx = std::max(gx, (groups + kRgMaxGroups - 1) / kRgMaxGroups);
    }
    p.share = groups / gx; p.extra = groups % gx;
    // as deep a ring as half of an SM holds; where the rows leave no room for that, of a whole one, with fewer warps at last
    const int most = p.share + (p.extra > 0);
    const int scratch = std::max(2 * p.a.groups, 2 * p.b.groups) + kRgMaxWarps;
    size_t smem = 0;
    for (p.warps = WARPS, p.depth = 0; p.depth == 0 && p.warps > 0; p.warps /= 2) {
        const int perWarp = (most * items + p.warps - 1) / p.warps;
        p.maxGroups = std::min(most, (perWarp + items - 2) / items + 1);
        const size_t fixed = ((size_t)MR * items * COLS + std::max(scratch, p.warps * p.maxGroups * MR * ROWS)) * 4, step = (size_t)p.warps * kRgItem;
        auto fits = [&](size_t room) { return room > fixed ? (int)std::min<size_t>(kRgMaxDepth, (room - fixed) / step) : 0; };
        p.depth = std::min(MR == 1 && fits(kRgSmemHalf) >= 2 ? fits(kRgSmemHalf) : fits(kRgSmemMax), std::max(perWarp, 1));
        smem = fixed + p.depth * step;
        if (p.depth > 0) break;
    }
    // Three or four rows that leave rings to fewer than half of the warps are better off as two passes of two: 12288 → 4096 31.5 in place of 43.7 µs,
    // 13312 → 4096 36.5 in place of 86; with half of them and one item each (11008 → 4096 27.4) two passes take 31.
    if (p.depth == 0 || (MR == 4 && p.warps < WARPS / 2)) return false;
    for (int v = 0; v < 2; v++) {
        const int units = (p.share + v) * items, busy = std::min(p.warps, units);
        for (int i = 0; i <= kRgMaxWarps; i++) {
            const int u = i < busy ? (int)((long long)units * i / busy) : units;
            p.first[v][i] = u;
            if (i < kRgMaxWarps) { p.firstGroup[v][i] = (unsigned short)(u / items); p.firstItem[v][i] = (unsigned short)(u % items); }
        }
    }
    auto aligned = [](const RowOperand& r) {
        return (((uintptr_t)r.x | (uintptr_t)r.gate | (uintptr_t)r.base | (uintptr_t)r.sum | (uintptr_t)r.gamma) & 15) == 0 &&
               ((r.k | r.ldx | (r.gate ? r.ldg : 0) | (r.base ? r.ldbase : 0) | (r.sum ? r.ldsum : 0)) & 3) == 0 && (r.groups < 2 || r.k / r.groups % 4 == 0);
    };
    // the second segment is a plain copy or goes column by column
    p.vec = (aligned(p.a) ? 1 : 0) | (p.b.k == 0 || (aligned(p.b) && p.b.groups == 0 && !p.b.gate && !p.b.base) ? 2 : 0);
    if (p.a.groups > 0 && (p.vec & 1)) {
        p.len = p.a.k / p.a.groups / 4;
        p.normWarps = std::max(1, WARPS / p.a.groups);
        p.normStep = (p.len + p.normWarps - 1) / p.normWarps;
        p.lenMagic = (unsigned)((1ull << 32) / (unsigned)p.len + 1);
        if (p.len == 1) p.vec &= ~1;             // the multiplier would not fit
    }
    static bool attr = false;
    if (!attr) {
        DJ_CUDA_CHECK(cudaFuncSetAttribute(k_bf16_gemv<MR, ROWS, WARPS, EXPERTS, PLAIN>, cudaFuncAttributeMaxDynamicSharedMemorySize, kRgSmemMax));
        attr = true;
    }
    launch_k(k_bf16_gemv<MR, ROWS, WARPS, EXPERTS, PLAIN>, dim3((unsigned)gx, (unsigned)tokens), dim3(WARPS * 32), smem, s, true, p);
    return true;
}

// Columns that the fullest block multiplies, those of padding among them, with so many weight rows per item.
long long padded_work(int rows, int rowSlots, int N, int itemSlots, int Kp) {
    const int cols = kRgItem / 2 / rows, groups = rowSlots * ((N + rows - 1) / rows);
    return (long long)((groups + g_num_sms - 1) / g_num_sms) * rows * itemSlots * ((Kp + cols - 1) / cols) * cols;
}
// One activation row (or one per token).  Two weight rows of 1024 columns per item, or four of 512 where that is a twentieth
// less work (lengths such as 512 or 1408); eight of 256 where the padded slots of a sum would not fit otherwise.
template <int EXPERTS>
bool launch_one(RgParams& p, const Bf16View& w, int rowSlots, int itemSlots, int tokens, cudaStream_t s) {
    if (padded_work(4, rowSlots, p.N, itemSlots, w.Kp) * 20 < padded_work(2, rowSlots, p.N, itemSlots, w.Kp) * 19)
        if (launch_rg<1, 4, 8, EXPERTS>(p, w, tokens, s)) return true;
    if (launch_rg<1, 2, 8, EXPERTS>(p, w, tokens, s) || launch_rg<1, 4, 8, EXPERTS>(p, w, tokens, s)) return true;
    if constexpr (EXPERTS == kExpertSum) return launch_rg<1, 8, 8, EXPERTS>(p, w, tokens, s);
    return false;
}

}  // namespace

void launch_bf16_gemv(const Bf16LinearArgs& a, cudaStream_t s) {
    for (int m0 = 0; m0 < a.M;) {
        RgParams p = {};
        p.a = a.a; p.b = a.b; p.N = a.w.N; p.K1p = pad8(a.a.k);
        p.a.x += (size_t)m0 * p.a.ldx;
        if (p.a.gate) p.a.gate += (size_t)m0 * p.a.ldg;
        if (p.a.base) p.a.base += (size_t)m0 * p.a.ldbase;
        if (p.a.sum) p.a.sum += (size_t)m0 * p.a.ldsum;
        if (p.b.k > 0) {
            p.b.x += (size_t)m0 * p.b.ldx;
            if (p.b.gate) p.b.gate += (size_t)m0 * p.b.ldg;
        }
        p.residual = a.residual ? a.residual + (size_t)m0 * a.ldr : nullptr; p.ldr = a.ldr;
        p.out = a.out ? a.out + (size_t)m0 * a.ldo : nullptr; p.ldo = a.ldo;
        p.gluRow = a.gluRow; p.limit = a.limit; p.glu = a.glu ? a.glu + (size_t)m0 * a.ldglu : nullptr; p.ldglu = a.ldglu;
        p.softcap = a.softcap; p.bias = a.bias; p.pair = a.pair;
        p.trigger = a.trigger;
        // three rows take the pass of four: 4096 → 12288 23.7 µs against 39.3 as a pass of two and one of one
        int rows = std::min(a.M - m0, 4);
        p.rows = rows;
        // as many rows as the staging leaves a ring for
        if (rows >= 3 && !launch_rg<4, 4, 16, kPlain>(p, a.w, 1, s)) p.rows = rows = 2;
        if (rows == 2 && !launch_rg<2, 2, 8, kPlain>(p, a.w, 1, s)) rows = 1;
        if (rows == 1 && !launch_one<kPlain>(p, a.w, 1, 1, 1, s)) throw std::runtime_error("bf16 projection: reduction length too large");
        m0 += rows;
    }
}

void launch_bf16_expert_gemv(const Bf16ExpertArgs& e, float* y, cudaStream_t s) {
    RgParams p = {};
    p.tok = e.tok; p.table = e.table; p.top = e.top; p.vocab = e.vocab;
    p.a = e.x; p.N = 2 * e.ff; p.K1p = pad8(e.x.k);
    p.gluRow = 0; p.limit = e.limit; p.glu = y; p.ldglu = e.ff;
    p.early = e.early; p.expertRows = 2 * e.ff; p.trigger = 0;
    if (!launch_one<kExpertRows>(p, e.up, e.top, 1, e.M, s)) throw std::runtime_error("experts: reduction length too large");
    p.a = RowOperand(); p.a.x = y; p.a.ldx = e.ff; p.a.k = e.ff;
    p.N = e.d; p.gluRow = e.d; p.glu = nullptr;
    p.residual = e.residual; p.ldr = e.ldr; p.out = e.out; p.ldo = e.ldo;
    p.early = 1; p.expertRows = e.d; p.trigger = e.trigger;       // behind the kernel above, which reads the tables only
    if (!launch_one<kExpertSum>(p, e.down, 1, e.top, e.M, s)) throw std::runtime_error("experts: too many slots for their width");
}

}  // namespace dj
