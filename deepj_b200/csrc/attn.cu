// Single-token causal attention over a K/V cache resident in HBM — one kernel.
//
// Replaces, for one new token per sequence, the reference's split-heads / RoPE /
// per-head QKᵀ / mask / softmax / PV / merge chain (HeadOps.java:33-140,
// RotaryEmbedding.java:81-122).  Masked positions contribute exactly +0 to the
// reference's softmax, so attending over 0..pos only is the same function.
//
// grid (splits, heads, batch), flash-decoding: a block rotates its head's q in registers (interleaved pairs,
// x0·c − x1·s, x0·s + x1·c) and streams its slice of the cache once.  Cached rows of a head are contiguous, so a warp asks for
// the K and the V rows of 32 / (hd / 16) positions with one bulk copy each, into a ring of its own, the first of them before the
// dependency wait; hd/16 lanes per position, online softmax in fp32.  The block that owns the newest position takes k and v from the
// projection buffer instead, rotates k and appends both to the cache.  Up to eight splits of a head are a cluster, where all clusters fit onto the chip: each
// block leaves (acc[hd], m, l) in the first one's shared memory, one cluster barrier, done.  More splits leave them in a workspace, and the last
// block of a head to finish (a ticket counter that it resets) merges them: a fence, the ticket and the loads are 2 µs.
// HBM-bound with long contexts: the algorithmic traffic is the K and V rows of 0..pos.  Measured between the projections around
// it, against rows through registers and tickets for any split: 16 heads × 128, 300 positions 6.9 µs (10.3; the hand-overs are 2 of it),
// 25 × 64, 210 positions ≈ 5 (7.3), 32 × 128, 2060 positions 16.1 (16.5, with less of the L1 that register loads want beside it).
#include "../../include/deepj_cuda.h"
#include "kernels.h"
#include "kv_cache.cuh"
#include "tc_common.cuh"
#include <algorithm>
#include <cmath>
#include <cstdlib>

namespace dj {

namespace {

constexpr int kAttnWarps = 4;
constexpr int kMaxSplits = 256;             // split partials a head can have (the merge keeps their weights in shared memory)
constexpr int kClusterSplits = 8;           // up to so many splits are a cluster
constexpr int kAttnSpinLimit = 1 << 22;     // polls of a barrier before the kernel gives up on it
constexpr int kErrAttnWait = 332;           // device error code: a copy of cached rows never arrived

// Prompt chunk: row z = (sequence b, token t) of the projection buffer holds k and v of position pos[b] + t.
// A block per row, a thread per two interleaved pairs: rotate k (x0·c − x1·s, x0·s + x1·c — RotaryEmbedding.java:81-122), copy v.
// 2048 rows of 32 heads × 128 took 71 µs as a block of 64 threads per head and row, 24 this way (21 µs at the copy bandwidth).
// Chunks of 32 tokens and more let the attention kernel in at the end.  Let in at the start, its 150 … 300 blocks took as long as if some SMs had three
// of them and others none: 32 heads × 64, 300 tokens behind 3000, both kernels 333 µs, 255 this way; 8 heads, 2048 tokens behind 700 239 and 216.
// Shorter ones have little to wait for (2 tokens of 32 heads × 64 7.1 µs, 7.6 with the end).
constexpr int kLateTokens = 32;
template <typename KT>
__global__ void __launch_bounds__(256) k_kv_append(const float* __restrict__ qkv, int k_off, int v_off, int ld, KT* __restrict__ kcache,
                            KT* __restrict__ vcache, int maxSeq, const float* __restrict__ posbuf,
                            const float* __restrict__ cosT, const float* __restrict__ sinT, int H, int hd, int T) {
    pdl_wait();
    if (T < kLateTokens) pdl_launch_dependents();
    const int z = blockIdx.x, b = z / T, tok = z - b * T;
    const int p = (int)posbuf[b] + tok;
    if (p < 0 || p >= maxSeq) return;
    const float* row = qkv + (size_t)z * ld;
    const int per = hd >> 2, n = H * per;         // hd is a multiple of 16
#pragma unroll 2
    for (int i = threadIdx.x; i < n; i += 256) {
        const int h = i / per, e = i - h * per;
        const float4 k = *reinterpret_cast<const float4*>(row + k_off + 4 * i), v = *reinterpret_cast<const float4*>(row + v_off + 4 * i);
        const float2 c = *reinterpret_cast<const float2*>(cosT + (size_t)p * (hd >> 1) + 2 * e), s = *reinterpret_cast<const float2*>(sinT + (size_t)p * (hd >> 1) + 2 * e);
        const size_t dst = (((size_t)b * H + h) * maxSeq + p) * hd + 4 * e;
        KvIo<KT>::st4(kcache + dst, make_float4(k.x * c.x - k.y * s.x, k.x * s.x + k.y * c.x, k.z * c.y - k.w * s.y, k.z * s.y + k.w * c.y));
        KvIo<KT>::st4(vcache + dst, v);
    }
    if (T >= kLateTokens) pdl_launch_dependents();
}

// Ring items per warp, of 2 KB of K rows and their V rows: four blocks and a projection's beside them have to fit into an SM.  (fp16 rows in items of
// half the size and lanes that read eight bytes a time: 12 heads × 64, 64 sequences at 200 17.3 µs, in place of 13.5 through cp.async rings; 13.4 this way.
// 32 × 128, 24 tokens behind 500 52.5, 38.7 and 36.0.)
constexpr int kRingStages = 2;
struct AttnDecodeParams {
    const float* qkv; int q_off, k_off, v_off, ld;
    void* kcache; void* vcache; int maxSeq;
    const float* pos; const float* cosT; const float* sinT;
    float* ws; int* tickets; float* out; int ldo, H; float scale; int T, append;
    int* error;
};

// A lane holds 16-byte pieces c·LPP + gl of its position's rows (four elements in fp32, eight in fp16): its neighbours read the pieces beside them.
// CLUSTER: the splits of a head are one cluster, whose blocks leave their partials in the first one's shared memory.
template <int LPP, typename KT, bool CLUSTER>   // lanes per position = hd / 16; cache element type
__global__ void __launch_bounds__(kAttnWarps * 32, 4) k_attn_decode(const AttnDecodeParams p) {
    constexpr int HD = LPP * 16, half = HD / 2;
    constexpr int PIECE = 16 / (int)sizeof(KT), NP = 16 / PIECE;         // elements of a piece, pieces of a lane
    constexpr int PPW = 32 / LPP;                 // positions per warp iteration
    constexpr int GPI = 4 / (int)sizeof(KT), PPI = PPW * GPI;            // a ring item: so many groups of positions, 2 KB of K rows
    constexpr int G = kAttnWarps * PPI;           // positions per block iteration
    constexpr int kStages = kRingStages, kPlane = PPI * HD * (int)sizeof(KT);      // ring items per warp: K rows of PPI consecutive positions, then their V rows
    extern __shared__ __align__(128) unsigned char ring[];               // [warps][kStages][2][kPlane]
    __shared__ __align__(8) unsigned long long s_bar[kAttnWarps * kStages];
    __shared__ __align__(16) float s_acc[kAttnWarps][HD];
    __shared__ float s_m[kAttnWarps], s_l[kAttnWarps];
    __shared__ int s_last;
    __shared__ float s_w[CLUSTER ? 1 : kMaxSplits];
    __shared__ float s_part[CLUSTER ? kClusterSplits : 1][CLUSTER ? HD + 2 : 1];       // the cluster's partials, in its first block

    // row z of the projection / output buffers is token t of sequence b: T = 1 (and append) for a decode step;
    // T > 1 for a short prompt chunk, whose k/v rows the append kernel has already written
    const int split = blockIdx.x, splits = gridDim.x, h = blockIdx.y, z = blockIdx.z;
    const int b = p.T == 1 ? z : z / p.T, tok = z - b * p.T;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int group = lane / LPP, gl = lane % LPP;
    if constexpr (CLUSTER) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    const uint32_t bars = smem_u32(&s_bar[warp * kStages]), mine = smem_u32(ring) + warp * (kStages * 2 * kPlane);
    if (lane < kStages) mbar_init(bars + 8 * lane, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    __syncwarp();

    // The cache rows below the current position were written by earlier steps, not by the kernel this one depends
    // on, so the first rows are requested BEFORE the wait and stream in while the projection kernel drains.  The
    // position read here is re-read after the wait; in the (never observed) case that it moved, the early rows are
    // dropped and requested again.
    auto read_pos = [&]() { return min(max((int)__ldcg(p.pos + b) + tok, 0), p.maxSeq - 1); };
    int pos = read_pos(), at = 0, endc = 0;       // the warp's next position to request, the end of the block's cached ones
    bool ownsNew = false;                         // the new token's position is this block's: not in the cache yet, folded in apart
    auto slice = [&]() {
        const int seq = pos + 1, chunk = (seq + splits - 1) / splits, start = split * chunk, end = min(seq, start + chunk);
        ownsNew = p.append && pos >= start && pos < end;
        endc = ownsNew ? pos : end;
        at = start + warp * PPI;
    };
    const size_t plane = ((size_t)b * p.H + h) * p.maxSeq * HD;
    KT* const khead = static_cast<KT*>(p.kcache) + plane;
    KT* const vhead = static_cast<KT*>(p.vcache) + plane;
    int asked = 0, taken = 0, limit = kAttnSpinLimit;                    // items since the start; item i is in slot i % kStages
    auto request = [&]() {
        if (lane == 0) {
            const int slot = asked % kStages;
            const uint32_t bytes = min(PPI, endc - at) * HD * (int)sizeof(KT), bar = bars + 8 * slot, to = mine + slot * (2 * kPlane);
            mbar_arrive_expect_tx(bar, 2 * bytes);
            bulk_g2s(to, khead + (size_t)at * HD, bytes, bar);
            bulk_g2s(to + kPlane, vhead + (size_t)at * HD, bytes, bar);
        }
        asked++;
        at += G;
    };
    auto take = [&]() {                           // the next item has arrived
        const uint32_t bar = bars + 8 * (taken % kStages), parity = (taken / kStages) & 1;
        bool ready = mbar_try_wait(bar, parity);
#pragma unroll 1
        for (int spin = 0; !ready && spin < limit; spin++) ready = mbar_try_wait(bar, parity);
        if (!ready) {                             // never on a healthy device: flag it, stop waiting long, keep the control flow
            if (lane == 0) atomicCAS(p.error, 0, kErrAttnWait);
            limit = 64;
        }
        taken++;
    };
    slice();
    int base = at;
#pragma unroll 1
    for (int i = 0; i < kStages && at < endc && p.T == 1; i++) request();      // a chunk's own rows were written by the kernel before this one
    // the rotation tables are constants: the row of the early position is fetched before the wait too
    float2 cs[4], sn[4];                          // of two pairs each
    auto load_tables = [&]() {
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const size_t at = (size_t)pos * half + PIECE / 2 * (j / (4 / NP) * LPP + gl) + j % (4 / NP) * 2;
            cs[j] = *reinterpret_cast<const float2*>(p.cosT + at);
            sn[j] = *reinterpret_cast<const float2*>(p.sinT + at);
        }
    };
    load_tables();
    const int early = pos;
    pdl_wait();
    pdl_launch_dependents();
    // the query row does not depend on the position: its loads go out together with the position's
    const float* rowp = p.qkv + (size_t)z * p.ld + h * HD + PIECE * gl;
    auto load_row = [&](int off, float (&v)[16]) {
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float4 a = *reinterpret_cast<const float4*>(rowp + off + j / (4 / NP) * (PIECE * LPP) + j % (4 / NP) * 4);
            v[4 * j] = a.x; v[4 * j + 1] = a.y; v[4 * j + 2] = a.z; v[4 * j + 3] = a.w;
        }
    };
    float q[16], kx[16], vx[16];
    load_row(p.q_off, q);
    pos = read_pos();
    if (pos != early || p.T > 1) {
#pragma unroll 1
        while (taken < asked) take();
        __syncwarp();
        if (pos != early) load_tables();
        slice();
        base = at;
#pragma unroll 1
        for (int i = 0; i < kStages && at < endc; i++) request();
    }
    // interleaved pairs (x0, x1) → (x0·c − x1·s, x0·s + x1·c)
    auto rotate = [&](float (&v)[16]) {
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const float c = i & 1 ? cs[i / 2].y : cs[i / 2].x, s = i & 1 ? sn[i / 2].y : sn[i / 2].x, x0 = v[2 * i], x1 = v[2 * i + 1];
            v[2 * i] = x0 * c - x1 * s;
            v[2 * i + 1] = x0 * s + x1 * c;
        }
    };

    float m = -INFINITY, l = 0.0f, acc[16];
#pragma unroll
    for (int e = 0; e < 16; e++) acc[e] = 0.0f;
    const bool folds = ownsNew && warp == 0;      // warp-uniform
    if (folds) { load_row(p.k_off, kx); load_row(p.v_off, vx); }
    rotate(q);
    // one group of positions a time: the new token's first (lane group 0), then what the ring holds, GPI groups an item
    const KT* item = nullptr;
    int gi = 0;
#pragma unroll 1
    for (bool fresh = folds; fresh || base < endc; fresh = false) {
        const bool valid = fresh ? group == 0 : base + group < endc;
        if (fresh) {
            // k and v come from the projections; k is rotated, both are appended to the cache, and this step attends to what
            // later steps will read back (the rounded values of an fp16 cache)
            rotate(kx);
#pragma unroll
            for (int c = 0; c < NP; c++)
                if (valid) {
                    KvIo<KT>::st_piece(khead + (size_t)pos * HD + PIECE * (c * LPP + gl), kx + PIECE * c);
                    KvIo<KT>::st_piece(vhead + (size_t)pos * HD + PIECE * (c * LPP + gl), vx + PIECE * c);
                }
#pragma unroll
            for (int e = 0; e < 16; e++) { kx[e] = KvIo<KT>::stored(kx[e]); vx[e] = KvIo<KT>::stored(vx[e]); }
        } else {
            if (GPI == 1 || gi == 0) {
                item = reinterpret_cast<const KT*>(ring + (size_t)warp * (kStages * 2 * kPlane) + (taken % kStages) * (2 * kPlane)) + group * HD + PIECE * gl;
                take();
            }
#pragma unroll
            for (int c = 0; c < NP; c++) { KvIo<KT>::ld_piece(item + c * (PIECE * LPP), kx + PIECE * c); KvIo<KT>::ld_piece(item + PPI * HD + c * (PIECE * LPP), vx + PIECE * c); }
        }
        float d[4];
#pragma unroll
        for (int j = 0; j < 4; j++) d[j] = fmaf(q[4 * j + 3], kx[4 * j + 3], fmaf(q[4 * j + 2], kx[4 * j + 2], fmaf(q[4 * j + 1], kx[4 * j + 1], q[4 * j] * kx[4 * j])));
        float dot = (d[0] + d[1]) + (d[2] + d[3]);
#pragma unroll
        for (int o = LPP / 2; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
        if (valid) {
            const float sc = dot * p.scale, mn = fmaxf(m, sc), corr = expf(m - mn), pe = expf(sc - mn);
            l = l * corr + pe;
#pragma unroll
            for (int e = 0; e < 16; e++) acc[e] = fmaf(pe, vx[e], acc[e] * corr);
            m = mn;
        }
        if (!fresh && GPI > 1 && gi + 1 < GPI && base + PPW < endc) {
            gi++;
            base += PPW;
            item += PPW * HD;
        } else if (!fresh) {
            base += G - gi * PPW;
            gi = 0;
            __syncwarp();                         // the slot is read out before a later request may overwrite it
            if (at < endc) request();
        }
    }

    // the warp's groups → one row per warp → the block's
    {
        float M = m;
#pragma unroll
        for (int o = LPP; o < 32; o <<= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
        const float f = m > -INFINITY ? expf(m - M) : 0.0f;
        l *= f;
#pragma unroll
        for (int e = 0; e < 16; e++) acc[e] *= f;
#pragma unroll
        for (int o = LPP; o < 32; o <<= 1) {
            l += __shfl_xor_sync(0xffffffffu, l, o);
#pragma unroll
            for (int e = 0; e < 16; e++) acc[e] += __shfl_xor_sync(0xffffffffu, acc[e], o);
        }
        if (group == 0) {
#pragma unroll
            for (int j = 0; j < 4; j++)
                *reinterpret_cast<float4*>(&s_acc[warp][j / (4 / NP) * (PIECE * LPP) + PIECE * gl + j % (4 / NP) * 4]) = make_float4(acc[4 * j], acc[4 * j + 1], acc[4 * j + 2], acc[4 * j + 3]);
        }
        if (lane == 0) { s_m[warp] = M; s_l[warp] = l; }
    }
    __syncthreads();
    float M = fmaxf(fmaxf(s_m[0], s_m[1]), fmaxf(s_m[2], s_m[3])), L = 0.0f, w[kAttnWarps];
#pragma unroll
    for (int i = 0; i < kAttnWarps; i++) { w[i] = s_m[i] > -INFINITY ? expf(s_m[i] - M) : 0.0f; L = fmaf(s_l[i], w[i], L); }
    auto blocks = [&](int j) {                    // column j of the block's sum
        float a = 0.0f;
#pragma unroll
        for (int i = 0; i < kAttnWarps; i++) a = fmaf(s_acc[i][j], w[i], a);
        return a;
    };
    float* const orow = p.out + (size_t)z * p.ldo + h * HD;
    if (splits == 1) {
#pragma unroll 1
        for (int j = tid; j < HD; j += kAttnWarps * 32) orow[j] = blocks(j) / L;
        return;
    }
    if constexpr (CLUSTER) {
        __syncwarp();                                                    // (the barrier's .aligned forms want whole warps)
        asm volatile("barrier.cluster.wait.aligned;" ::: "memory");      // every block of the cluster is running
        uint32_t to;
        asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(to) : "r"(smem_u32(&s_part[split][0])));
        auto put = [&](int j, float v) { asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(to + 4 * j), "f"(v) : "memory"); };
#pragma unroll 1
        for (int j = tid; j < HD; j += kAttnWarps * 32) put(j, blocks(j));
        if (tid == 0) { put(HD, M); put(HD + 1, L); }
        __syncwarp();                                                    // heads of 16: half of the first warp has put a column
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        if (split != 0) return;
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        M = -INFINITY;
#pragma unroll 1
        for (int i = 0; i < splits; i++) M = fmaxf(M, s_part[i][HD]);
#pragma unroll 1
        for (int j = tid; j < HD; j += kAttnWarps * 32) {
            float a = 0.0f;
            L = 0.0f;
#pragma unroll 1
            for (int i = 0; i < splits; i++) {
                const float e = expf(s_part[i][HD] - M);                 // an empty split: exp(−inf) = 0
                a = fmaf(s_part[i][j], e, a);
                L = fmaf(s_part[i][HD + 1], e, L);
            }
            orow[j] = a / L;
        }
        return;
    }
    // ── the last block of this head merges the split partials ──
    const float* const records = p.ws + ((size_t)z * p.H + h) * splits * (HD + 2);
    float* const record = p.ws + (((size_t)z * p.H + h) * splits + split) * (HD + 2);
#pragma unroll 1
    for (int j = tid; j < HD; j += kAttnWarps * 32) record[j] = blocks(j);
    if (tid == 0) { record[HD] = M; record[HD + 1] = L; }
    __threadfence();
    __syncthreads();
    if (tid == 0) {
        const int ticket = atomicAdd(&p.tickets[z * p.H + h], 1);
        s_last = ticket == splits - 1;
        if (s_last) p.tickets[z * p.H + h] = 0;   // ready for the next launch
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    // every thread asks for its column of the first splits together with the (m, l) pairs: one load round trip for most
    constexpr int kBatch = 20;
    float first[kBatch];
#pragma unroll
    for (int i = 0; i < kBatch; i++) first[i] = tid < HD && i < splits ? __ldcg(records + (size_t)i * (HD + 2) + tid) : 0.0f;
    M = -INFINITY;
#pragma unroll 1
    for (int i = lane; i < splits; i += 32) M = fmaxf(M, __ldcg(records + (size_t)i * (HD + 2) + HD));
    for (int o = 16; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
    L = 0.0f;
#pragma unroll 1
    for (int i = lane; i < splits; i += 32) {     // every warp for itself; the first one leaves the weights
        const float e = expf(__ldcg(records + (size_t)i * (HD + 2) + HD) - M);
        L = fmaf(__ldcg(records + (size_t)i * (HD + 2) + HD + 1), e, L);
        if (warp == 0) s_w[i] = e;
    }
    for (int o = 16; o > 0; o >>= 1) L += __shfl_xor_sync(0xffffffffu, L, o);
    __syncthreads();
    for (int j = tid; j < HD; j += kAttnWarps * 32) {
        float a = 0.0f;
        if (j == tid) {
#pragma unroll
            for (int i = 0; i < kBatch; i++) if (i < splits) a = fmaf(first[i], s_w[i], a);
        }
#pragma unroll 8
        for (int i = j == tid ? kBatch : 0; i < splits; i++) a = fmaf(__ldcg(records + (size_t)i * (HD + 2) + j), s_w[i], a);
        orow[j] = a / L;
    }
}

// ───────────── prompt chunks: tiled causal attention ─────────────
// Row-wise decode attention re-reads every key once per query row.  For a chunk of T ≥ 32 tokens this kernel
// lets 32 consecutive query rows of one head share each 64-key tile of K and V through shared memory (fp32 on the
// CUDA cores, online softmax per row):  S = Q·Kᵀ (Q rotated and pre-scaled at load, the K tile's 16-byte chunks
// XOR-swizzled so that the 16-byte reads of a quarter warp never share a bank), mask, running max / sum, P through
// shared memory, O += P·V.
// grid (query tiles, heads, sequences), 256 threads: thread (rg, cg) = (t / 16, t % 16) owns rows 2rg, 2rg+1 —
// the 16 lanes of a row pair are contiguous, row reductions are half-warp shuffles.
constexpr int kPQ = 32, kPK = 64;

template <int HD, typename KT>
__global__ void __launch_bounds__(256, 2) k_attn_prefill_tiled(
        const float* __restrict__ qkv, int q_off, int ld, const KT* __restrict__ kcache, const KT* __restrict__ vcache,
        int maxSeq, const float* __restrict__ posbuf, const float* __restrict__ cosT, const float* __restrict__ sinT,
        float* __restrict__ out, int ldo, int H, float scale, int T) {
    extern __shared__ __align__(16) float sm[];
    float* Qs = sm;                                 // [32][HD]
    float* Ks = Qs + kPQ * HD;                      // [64][HD], 16-byte chunks XOR-swizzled by (key / 4) % 8
    float* Vs = Ks + kPK * HD;                      // [64][HD]
    float* Ps = Vs + kPK * HD;                      // [32][68]
    constexpr int kPsStride = kPK + 4;
    pdl_wait();
    pdl_launch_dependents();
    const int tid = threadIdx.x, rg = tid >> 4, cg = tid & 15;
    const int qt = blockIdx.x, h = blockIdx.y, b = blockIdx.z;
    const int t0 = qt * kPQ;
    int pos0 = (int)posbuf[b];
    pos0 = pos0 < 0 ? 0 : pos0;
    const int half = HD >> 1;
    // Q tile: rotate (interleaved pairs) at position pos0 + t and fold in the 1/sqrt(hd) scale
    for (int i = tid; i < kPQ * half; i += 256) {
        const int r = i / half, pr = i % half;
        const int t = t0 + r;
        float x0 = 0.0f, x1 = 0.0f;
        if (t < T && pos0 + t < maxSeq) {
            const float2 v = *reinterpret_cast<const float2*>(qkv + (size_t)(b * T + t) * ld + q_off + h * HD + 2 * pr);
            const float c = cosT[(size_t)(pos0 + t) * half + pr], s = sinT[(size_t)(pos0 + t) * half + pr];
            x0 = (v.x * c - v.y * s) * scale;
            x1 = (v.x * s + v.y * c) * scale;
        }
        Qs[r * HD + 2 * pr] = x0;
        Qs[r * HD + 2 * pr + 1] = x1;
    }
    const KT* kb = kcache + ((size_t)b * H + h) * maxSeq * HD;
    const KT* vb = vcache + ((size_t)b * H + h) * maxSeq * HD;
    const int lastKey = min(maxSeq - 1, pos0 + min(T, t0 + kPQ) - 1);       // newest key any row of this tile may see
    const int r0 = 2 * rg, r1 = 2 * rg + 1;
    const int lim0 = pos0 + t0 + r0, lim1 = pos0 + t0 + r1;                  // row r attends to keys ≤ lim
    constexpr int kOC = HD / 16;                                             // output columns per thread
    float o0[kOC], o1[kOC];
#pragma unroll
    for (int j = 0; j < kOC; j++) { o0[j] = 0.0f; o1[j] = 0.0f; }
    float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.0f, l1 = 0.0f;
    for (int k0 = 0; k0 <= lastKey; k0 += kPK) {
        __syncthreads();                            // the previous tile's K, V and P are no longer read (first round: Q is written)
        // K tile, transposed, and V tile
        for (int i = tid; i < kPK * (HD / 4); i += 256) {
            const int key = i / (HD / 4), d4 = i % (HD / 4);
            float4 kv = make_float4(0.f, 0.f, 0.f, 0.f), vv = kv;
            if (k0 + key <= lastKey) {
                kv = KvIo<KT>::ld4(kb + (size_t)(k0 + key) * HD + 4 * d4);
                vv = KvIo<KT>::ld4(vb + (size_t)(k0 + key) * HD + 4 * d4);
            }
            *reinterpret_cast<float4*>(Ks + key * HD + 4 * (d4 ^ ((key >> 2) & 7))) = kv;
            *reinterpret_cast<float4*>(Vs + key * HD + 4 * d4) = vv;
        }
        __syncthreads();
        // S = Q·Kᵀ for rows r0, r1 and keys 4cg … 4cg+3
        float s0[4] = {0.f, 0.f, 0.f, 0.f}, s1[4] = {0.f, 0.f, 0.f, 0.f};
        const int sw = cg & 7;                      // (key / 4) % 8 of this thread's four keys
#pragma unroll 4
        for (int c = 0; c < HD / 4; c++) {
            const float4 q0 = *reinterpret_cast<const float4*>(Qs + r0 * HD + 4 * c);
            const float4 q1 = *reinterpret_cast<const float4*>(Qs + r1 * HD + 4 * c);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float4 k4 = *reinterpret_cast<const float4*>(Ks + (4 * cg + j) * HD + 4 * (c ^ sw));
                s0[j] = fmaf(q0.x, k4.x, s0[j]); s0[j] = fmaf(q0.y, k4.y, s0[j]); s0[j] = fmaf(q0.z, k4.z, s0[j]); s0[j] = fmaf(q0.w, k4.w, s0[j]);
                s1[j] = fmaf(q1.x, k4.x, s1[j]); s1[j] = fmaf(q1.y, k4.y, s1[j]); s1[j] = fmaf(q1.z, k4.z, s1[j]); s1[j] = fmaf(q1.w, k4.w, s1[j]);
            }
        }
        float mx0 = -INFINITY, mx1 = -INFINITY;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int key = k0 + 4 * cg + j;
            if (key > lim0 || key > lastKey) s0[j] = -INFINITY;
            if (key > lim1 || key > lastKey) s1[j] = -INFINITY;
            mx0 = fmaxf(mx0, s0[j]); mx1 = fmaxf(mx1, s1[j]);
        }
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) { mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, o)); mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, o)); }
        const float mn0 = fmaxf(m0, mx0), mn1 = fmaxf(m1, mx1);
        const float c0 = mn0 > -INFINITY ? expf(m0 - mn0) : 1.0f, c1 = mn1 > -INFINITY ? expf(m1 - mn1) : 1.0f;
        float ps0 = 0.0f, ps1 = 0.0f;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float p0 = s0[j] > -INFINITY ? expf(s0[j] - mn0) : 0.0f, p1 = s1[j] > -INFINITY ? expf(s1[j] - mn1) : 0.0f;
            Ps[r0 * kPsStride + 4 * cg + j] = p0; Ps[r1 * kPsStride + 4 * cg + j] = p1;
            ps0 += p0; ps1 += p1;
        }
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) { ps0 += __shfl_xor_sync(0xffffffffu, ps0, o); ps1 += __shfl_xor_sync(0xffffffffu, ps1, o); }
        l0 = l0 * c0 + ps0; l1 = l1 * c1 + ps1;
        m0 = mn0; m1 = mn1;
#pragma unroll
        for (int j = 0; j < kOC; j++) { o0[j] *= c0; o1[j] *= c1; }
        __syncthreads();
        // O += P·V for rows r0, r1 and columns kOC·cg … kOC·cg + kOC − 1
        const int nk = min(kPK, lastKey - k0 + 1);
        for (int key = 0; key < nk; key++) {
            const float p0 = Ps[r0 * kPsStride + key], p1 = Ps[r1 * kPsStride + key];
            const float* vr = Vs + key * HD + kOC * cg;
#pragma unroll
            for (int j = 0; j < kOC; j += 4) {
                const float4 v4 = *reinterpret_cast<const float4*>(vr + j);
                o0[j] = fmaf(p0, v4.x, o0[j]); o0[j + 1] = fmaf(p0, v4.y, o0[j + 1]); o0[j + 2] = fmaf(p0, v4.z, o0[j + 2]); o0[j + 3] = fmaf(p0, v4.w, o0[j + 3]);
                o1[j] = fmaf(p1, v4.x, o1[j]); o1[j + 1] = fmaf(p1, v4.y, o1[j + 1]); o1[j + 2] = fmaf(p1, v4.z, o1[j + 2]); o1[j + 3] = fmaf(p1, v4.w, o1[j + 3]);
            }
        }
    }
    if (t0 + r0 < T && l0 > 0.0f) {
        float* dst = out + (size_t)(b * T + t0 + r0) * ldo + h * HD + kOC * cg;
#pragma unroll
        for (int j = 0; j < kOC; j++) dst[j] = o0[j] / l0;
    }
    if (t0 + r1 < T && l1 > 0.0f) {
        float* dst = out + (size_t)(b * T + t0 + r1) * ldo + h * HD + kOC * cg;
#pragma unroll
        for (int j = 0; j < kOC; j++) dst[j] = o1[j] / l1;
    }
}

template <int HD> constexpr size_t prefill_tiled_smem() { return (size_t)(kPQ * HD + kPK * HD + kPK * HD + kPQ * (kPK + 4)) * 4; }

}  // namespace

int attn_decode_splits(int B, int H, int maxSeq) {
    int want = (4 * g_num_sms) / (B * H);           // every CTA resident at once: a second, nearly empty wave would double the time
    int cap = (maxSeq + 63) / 64;
    int s = want < cap ? want : cap;
    if (s > 256) s = 256;                           // the merge keeps one weight per split in shared memory
    return s < 1 ? 1 : s;
}
size_t attn_decode_ws_floats(int B, int H, int hd, int splits) {
    return (size_t)B * H * splits * (hd + 2);
}

namespace {

template <typename KT>
void launch_attn_decode_t(const AttnDecodeArgs& a, cudaStream_t s) {
    int lpp = a.hd / 16;
    if (a.hd % 16 != 0 || (lpp != 1 && lpp != 2 && lpp != 4 && lpp != 8 && lpp != 16 && lpp != 32))
        throw std::runtime_error("attention: head dim " + std::to_string(a.hd) + " is not one of 16,32,64,128,256,512");
    const int T = a.T < 1 ? 1 : a.T;
    const long rows = (long)a.B * T;
    if (rows > 65535) throw std::runtime_error("attention: more than 65535 rows in one launch");
    dim3 grid(a.splits, a.H, (unsigned)rows), block(kAttnWarps * 32);
    if (a.splits > 1 && rows * a.H > kAttnTickets / 2) throw std::runtime_error("attention: rows × heads exceeds " + std::to_string(kAttnTickets / 2));
    KT* kc = static_cast<KT*>(a.kcache);
    KT* vc = static_cast<KT*>(a.vcache);
    if (T > 1) {
        // the chunk's keys (rotated) and values go into the cache first; the attention kernel then only reads
        launch_k(k_kv_append<KT>, dim3((unsigned)rows), dim3(256), 0, s, true, (const float*)a.qkv, a.k_off, a.v_off, a.ld, kc, vc, a.maxSeq,
                 a.pos, a.cosT, a.sinT, a.H, a.hd, T);
    }
    static const bool noTiled = getenv("DEEPJ_CUDA_NO_TILED_PREFILL") != nullptr;
    static const bool noMma = getenv("DEEPJ_CUDA_NO_MMA_PREFILL") != nullptr;
    if (T >= kPQ && !noTiled && !noMma && launch_attn_prefill_mma(a, s)) return;      // tensor-core tiles (attn_mma.cu)
    if (T >= kPQ && !noTiled && (a.hd == 64 || a.hd == 128)) {
        dim3 tg((T + kPQ - 1) / kPQ, a.H, a.B);
        if (a.hd == 128) {
            static bool attr = false;
            if (!attr) { DJ_CUDA_CHECK(cudaFuncSetAttribute(k_attn_prefill_tiled<128, KT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)prefill_tiled_smem<128>())); attr = true; }
            launch_k(k_attn_prefill_tiled<128, KT>, tg, dim3(256), prefill_tiled_smem<128>(), s, true, (const float*)a.qkv, a.q_off, a.ld,
                     (const KT*)kc, (const KT*)vc, a.maxSeq, a.pos, a.cosT, a.sinT, a.out, a.ldo, a.H, a.scale, T);
        } else {
            static bool attr = false;
            if (!attr) { DJ_CUDA_CHECK(cudaFuncSetAttribute(k_attn_prefill_tiled<64, KT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)prefill_tiled_smem<64>())); attr = true; }
            launch_k(k_attn_prefill_tiled<64, KT>, tg, dim3(256), prefill_tiled_smem<64>(), s, true, (const float*)a.qkv, a.q_off, a.ld,
                     (const KT*)kc, (const KT*)vc, a.maxSeq, a.pos, a.cosT, a.sinT, a.out, a.ldo, a.H, a.scale, T);
        }
        return;
    }
    AttnDecodeParams p = {a.qkv, a.q_off, a.k_off, a.v_off, a.ld, kc, vc, a.maxSeq, a.pos, a.cosT, a.sinT, a.ws, a.tickets, a.out, a.ldo, a.H, a.scale, T,
                          T == 1 ? 1 : 0, g_dev_error};
    const size_t smem = (size_t)kAttnWarps * kRingStages * 4096;
    // a few splits merge through the first block's shared memory instead of a ticket, a fence and a round trip to the partials,
    bool cluster = a.splits > 1 && a.splits <= kClusterSplits;
    auto go = [&](auto kernel) {
        DJ_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024));
        launch_k_cluster(kernel, grid, block, smem, s, dim3(cluster ? a.splits : 1), p);
    };
    // where all clusters are resident at once (187 of three, 142 of four, 93 of six): a second, nearly empty wave took 8 heads × 128, 24 sequences at 1000
    // from 20.5 µs to 33 (fp16; 35 and 41 in fp32)
    auto fits = [&](auto kernel) {
        if (!cluster) return false;
        static int resident[33][kClusterSplits + 1];                     // clusters by lanes per position and splits, 0 = not asked yet
        int& most = resident[lpp][a.splits];
        if (most == 0) {
            DJ_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024));
            cudaLaunchAttribute attr;
            attr.id = cudaLaunchAttributeClusterDimension;
            attr.val.clusterDim.x = a.splits; attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(a.splits); cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.attrs = &attr; cfg.numAttrs = 1;
            DJ_CUDA_CHECK(cudaOccupancyMaxActiveClusters(&most, kernel, &cfg));
        }
        return rows * a.H <= most;
    };
#define DJ_ATTN_CASE(L) case L: cluster = fits(k_attn_decode<L, KT, true>); if (cluster) go(k_attn_decode<L, KT, true>); else go(k_attn_decode<L, KT, false>); break;
    switch (lpp) {
        DJ_ATTN_CASE(1) DJ_ATTN_CASE(2) DJ_ATTN_CASE(4) DJ_ATTN_CASE(8) DJ_ATTN_CASE(16) DJ_ATTN_CASE(32)
    }
#undef DJ_ATTN_CASE
}

}  // namespace

void launch_attn_decode(const AttnDecodeArgs& a, cudaStream_t s) {
    if (a.kvHalf) launch_attn_decode_t<__half>(a, s);
    else launch_attn_decode_t<float>(a, s);
}

}  // namespace dj

// ───────────── attention without any allocation ─────────────
// Scratch for deepj_cuda_attn_decode_static: the split partials and the ticket counters
// live in this fixed array instead of the runtime's growable workspace.  Every GPU that
// loads the library holds these 2 MiB + 16 KiB until the process exits.
namespace {
constexpr size_t kStaticPartialFloats = 512 * 1024;     // 2 MiB of (acc[hd], m, l) records
constexpr size_t kStaticTickets = 4096;                 // batch × heads
static __device__ __align__(256) float g_attn_static_scratch[kStaticPartialFloats + kStaticTickets];

// The array's name is only a host-side handle; the device address comes from
// cudaGetSymbolAddress, asked once per device with that device current.
float* g_static_scratch_addr[64] = {};
}  // namespace

extern "C" int deepj_cuda_attn_decode_static(int32_t qkv, int32_t q_off, int32_t k_off, int32_t v_off, int32_t ld,
                                             int32_t kv, int32_t layer, int32_t pos, int32_t cos_table, int32_t sin_table,
                                             int32_t out, int32_t out_off, int32_t ldo, int32_t B, int32_t H, int32_t hd) {
    using namespace dj;
    try {
        cudaStream_t stream = runtime_stream();
        if (stream == nullptr) throw std::runtime_error("attn_decode_static: the library holds no buffers yet (nothing was allocated through it)");
        const int dev = runtime_device();
        if (dev < 0 || dev >= 64) throw std::runtime_error("attn_decode_static: device index out of range");
        // the library's device is made current for the length of this call and the caller's is put back on every way out
        struct DeviceGuard {
            int prev = -1; bool switched = false;
            ~DeviceGuard() { if (switched) cudaSetDevice(prev); }
        } guard;
        DJ_CUDA_CHECK(cudaGetDevice(&guard.prev));
        if (guard.prev != dev) { DJ_CUDA_CHECK(cudaSetDevice(dev)); guard.switched = true; }
        if (g_static_scratch_addr[dev] == nullptr) {
            // first call on this device: resolve the scratch array's device address
            float* p = nullptr;
            DJ_CUDA_CHECK(cudaGetSymbolAddress((void**)&p, g_attn_static_scratch));
            if (p == nullptr) throw std::runtime_error("attn_decode_static: scratch address is null");
            g_static_scratch_addr[dev] = p;
        }
        float* scratch = g_static_scratch_addr[dev];

        PoolKV kvb; PoolF32 bq, bp, bc, bs, bo;
        if (!pool_kv(kv, &kvb)) throw std::runtime_error("attn_decode_static: missing KV cache id=" + std::to_string(kv));
        if (!pool_f32(qkv, &bq) || !pool_f32(pos, &bp) || !pool_f32(cos_table, &bc) || !pool_f32(sin_table, &bs) || !pool_f32(out, &bo))
            throw std::runtime_error("attn_decode_static: missing GPU buffer");
        if (B < 1 || H < 1 || hd < 2 || B > kvb.B || H != kvb.H || hd != kvb.hd) throw std::runtime_error("attn_decode_static: shape does not match the KV cache");
        if (layer < 0 || layer >= kvb.layers) throw std::runtime_error("attn_decode_static: layer out of range");
        if (q_off < 0 || k_off < 0 || v_off < 0 || out_off < 0 || ld % 4 || q_off % 4 || k_off % 4 || v_off % 4)
            throw std::runtime_error("attn_decode_static: offsets and stride must be non-negative multiples of 4 floats");
        const int d = H * hd;
        const int maxOff = std::max(q_off, std::max(k_off, v_off));
        if (ld < maxOff + d || ldo < d) throw std::runtime_error("attn_decode_static: row stride smaller than the row");
        if (bq.floats < (size_t)(B - 1) * ld + maxOff + d || bp.floats < (size_t)B || bo.floats < (size_t)out_off + (size_t)(B - 1) * ldo + d ||
            bc.floats < (size_t)kvb.maxSeq * (hd / 2) || bs.floats < (size_t)kvb.maxSeq * (hd / 2))
            throw std::runtime_error("attn_decode_static: a buffer is smaller than the op needs");
        const int splits = attn_decode_splits(B, H, kvb.maxSeq);
        const size_t need = attn_decode_ws_floats(B, H, hd, splits);
        if (need > kStaticPartialFloats || (size_t)B * H > kStaticTickets)
            throw std::runtime_error("attn_decode_static: needs " + std::to_string(need) + " scratch floats and " + std::to_string((size_t)B * H) +
                                     " counters; the static scratch holds " + std::to_string(kStaticPartialFloats) + " and " +
                                     std::to_string(kStaticTickets) + " (use op 67 through deepj_cuda_flush_ops for larger shapes)");
        int* tickets = reinterpret_cast<int*>(scratch + kStaticPartialFloats);
        // the array keeps whatever the last call left: the counters must start at zero
        DJ_CUDA_CHECK(cudaMemsetAsync(tickets, 0, (size_t)B * H * sizeof(int), stream));
        AttnDecodeArgs a = {};
        a.qkv = bq.ptr; a.q_off = q_off; a.k_off = k_off; a.v_off = v_off; a.ld = ld;
        const size_t esz = kvb.half ? 2 : 4;
        const size_t plane = (size_t)kvb.layers * kvb.B * kvb.H * kvb.maxSeq * kvb.hd;
        const size_t layerOff = (size_t)layer * kvb.B * kvb.H * kvb.maxSeq * kvb.hd;
        a.kcache = static_cast<char*>(kvb.ptr) + layerOff * esz; a.vcache = static_cast<char*>(kvb.ptr) + (plane + layerOff) * esz;
        a.maxSeq = kvb.maxSeq; a.kvHalf = kvb.half;
        a.pos = bp.ptr; a.cosT = bc.ptr; a.sinT = bs.ptr;
        a.out = bo.ptr + out_off; a.ldo = ldo; a.B = B; a.H = H; a.hd = hd;
        a.scale = (float)(1.0 / std::sqrt((double)hd));
        a.splits = splits; a.ws = scratch; a.tickets = tickets;
        launch_attn_decode(a, stream);
        DJ_CUDA_CHECK(cudaStreamSynchronize(stream));
        return 0;
    } catch (const std::exception& e) {
        set_last_error(e.what());
        return 1;
    }
}

