// Many-row projections with bf16 weights on the 5th-generation tensor cores: out[M × N] = A[M × K] · W[N × K]ᵀ.
//
// The activation rows are staged to bf16 in the workspace by k_stage_rows (norm and gate applied in fp32 there); both
// operands then travel as 64-column boxes with 128-byte swizzle through the tensor-memory accelerator.  Persistent CTAs,
// one per SM, walk 128 × BN output tiles (rows of tiles fastest: CTAs that run together share a weight tile in L2):
//   warp 4   one thread keeps a ring of (A, W) stages full; the first stages' weights are on their way before the
//            dependency wait
//   warp 5   one thread issues tcgen05.mma 128 × BN × 16 into one of two accumulators in tensor memory
//   warps 0-3  drain the other accumulator: tcgen05.ld, a shared-memory transpose, row-contiguous stores with residual,
//            soft cap or the gated pair
// Grouped form (table-routed experts): `tileExpert` gives each 128-row tile its expert (−1: no tile), whose weight rows
// start at expert · N; `rowMap` scatters output rows.  Every wait is bounded (codes 211-214 in the device error word,
// 215-218 in the form for pairs of SMs, whose comment stands at the kernel).
#include "row_operand.cuh"
#include "tc_common.cuh"

#include <algorithm>

namespace dj {
namespace {

constexpr int kGM = 128, kGK = 64, kGThreads = 192;
constexpr int kABytes = kGM * kGK * 2;
constexpr int kEpiBytes = 4 * 32 * 33 * 4;

struct GemmTcParams {
    CUtensorMap a, w;
    int M, N, nK, mTiles, nTiles;
    const int* tileExpert; const int* rowMap;
    const float* lenPos; int lenT;               // rows = lenPos[0] + lenT, at most M (device-side length)
    const float* residual; int ldr;
    float* out; int ldo; __nv_bfloat16* outHalf; // outHalf: bf16 rows instead of fp32
    int gluRow; float limit; float* glu; int ldglu;
    float softcap; const float* bias; int pair;
    int* error;
};

// K-major, 128-byte swizzle: 8-row groups 1024 bytes apart, descriptor version 1, layout type 2
__device__ __forceinline__ uint64_t desc_sw128(uint32_t smem_addr) {
    return (uint64_t)((smem_addr >> 4) & 0x3fff) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}

template <int BN> struct GemmShape {
    static constexpr int kStageBytes = kABytes + BN * kGK * 2;
    static constexpr int kStages = BN == 256 ? 4 : BN == 128 ? 6 : 8;
    static constexpr size_t kSmem = (size_t)kStages * kStageBytes + kEpiBytes + 1024;
    static constexpr int kTmem = 2 * BN < 32 ? 32 : 2 * BN;
    // bf16 × bf16 → fp32, both K-major
    static constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(kGM >> 4) << 24);
};

// A warp's 32 rows of an accumulator (from column 0 of it) → the outputs of rows mBase … and columns n0 ….
template <int BN>
__device__ __forceinline__ void store_tile(const GemmTcParams& p, uint32_t acc, int mBase, int rows, int n0, float* stg, int warp, int lane) {
    int myRow = mBase + lane < rows ? mBase + lane : -1;      // output row of tile row `lane`
    if (myRow >= 0 && p.rowMap != nullptr) myRow = p.rowMap[myRow];
#pragma unroll 1
    for (int c0 = 0; c0 < BN && n0 + c0 < p.N; c0 += 32) {
        uint32_t v[32];
        tmem_ld32(acc + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0, v);
#pragma unroll
        for (int j = 0; j < 32; j++) stg[lane * 33 + j] = __uint_as_float(v[j]);
        __syncwarp();
        const int nb = n0 + c0, nn = nb + lane;
        if (p.outHalf != nullptr) {
#pragma unroll 8
            for (int i = 0; i < 32; i += 2) {
                const int r = i + (lane >> 4), row = __shfl_sync(0xffffffffu, myRow, r), c = 2 * (lane & 15);
                if (row >= 0 && nb + c < p.N)
                    *reinterpret_cast<__nv_bfloat162*>(p.outHalf + (size_t)row * p.ldo + nb + c) = __floats2bfloat162_rn(stg[r * 33 + c], stg[r * 33 + c + 1]);
            }
            __syncwarp();
            continue;
        }
        if (nb < p.gluRow) {
            const float myBias = p.bias != nullptr && nn < p.gluRow ? p.bias[nn] : 0.0f;
#pragma unroll 8
            for (int i = 0; i < 32; i++) {
                const int row = __shfl_sync(0xffffffffu, myRow, i);
                if (row >= 0 && nn < p.gluRow) {
                    float val = stg[i * 33 + lane] + myBias;
                    if (p.residual) val += p.residual[(size_t)row * p.ldr + nn];
                    p.out[(size_t)row * p.ldo + nn] = softcap_f(val, p.softcap);
                }
            }
        }
        if (nb + 32 > p.gluRow && p.gluRow < p.N) {
            const int pair = nb + 2 * (lane & 15);
#pragma unroll 4
            for (int i = 0; i < 32; i += 2) {
                const int r = i + (lane >> 4), row = __shfl_sync(0xffffffffu, myRow, r);
                if (row >= 0 && pair >= p.gluRow && pair < p.N) {
                    const float g = stg[r * 33 + 2 * (lane & 15)], u = stg[r * 33 + 2 * (lane & 15) + 1];
                    p.glu[(size_t)row * p.ldglu + ((pair - p.gluRow) >> 1)] = pair_f(g, u, p.limit, p.pair);
                }
            }
        }
        __syncwarp();
    }
}

template <int BN>
__global__ void __launch_bounds__(kGThreads, 1) k_bf16_gemm_tc(const __grid_constant__ GemmTcParams p) {
    using S = GemmShape<BN>;
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ __align__(8) unsigned long long s_bar[2 * S::kStages + 4];
    __shared__ uint32_t s_tmem;
    __shared__ volatile int s_abort;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t raw = smem_u32(smem), base = (raw + 1023u) & ~1023u;
    float* const stg = reinterpret_cast<float*>(smem + (base - raw) + (size_t)S::kStages * S::kStageBytes) + warp * (32 * 33);
    auto full = [&](int s) { return smem_u32(&s_bar[s]); };
    auto empty = [&](int s) { return smem_u32(&s_bar[S::kStages + s]); };
    auto accFull = [&](int a) { return smem_u32(&s_bar[2 * S::kStages + a]); };
    auto accEmpty = [&](int a) { return smem_u32(&s_bar[2 * S::kStages + 2 + a]); };
    if (tid == 0) {
        for (int s = 0; s < S::kStages; s++) { mbar_init(full(s), 1); mbar_init(empty(s), 1); }
        for (int a = 0; a < 2; a++) { mbar_init(accFull(a), 1); mbar_init(accEmpty(a), 128); }
        s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 4) tmem_alloc(smem_u32(&s_tmem), S::kTmem);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    int rows = p.M, mTiles = p.mTiles, tiles = p.mTiles * p.nTiles;
    auto read_length = [&] {                         // after the dependency wait
        if (p.lenPos != nullptr) {
            rows = min(p.M, max((int)p.lenPos[0], 0) + p.lenT);
            mTiles = (rows + kGM - 1) / kGM;
            tiles = mTiles * p.nTiles;
        }
    };

    if (warp == 4) {
        if (lane == 0) {
            int early = 0;                                   // stages whose weights were requested before the wait
            if (p.tileExpert == nullptr && p.lenPos == nullptr && (int)blockIdx.x < tiles) {
                const int n0 = ((int)blockIdx.x / p.mTiles) * BN;
                for (; early < S::kStages && early < p.nK; early++) {
                    mbar_arrive_expect_tx(full(early), S::kStageBytes);
                    tma_box(base + early * S::kStageBytes + kABytes, &p.w, early * kGK, n0, full(early));
                }
            }
            pdl_wait();
            pdl_launch_dependents();
            read_length();
            unsigned it = 0;
            bool ok = true;
            for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x) {
                const int mt = t % mTiles;
                int wrow = (t / mTiles) * BN;
                if (p.tileExpert != nullptr) {
                    const int e = p.tileExpert[mt];
                    if (e < 0) continue;
                    wrow += e * p.N;
                }
                for (int kt = 0; kt < p.nK; kt++, it++) {
                    const int s = it % S::kStages;
                    const uint32_t dst = base + s * S::kStageBytes;
                    if ((int)it >= early) {
                        if (it >= (unsigned)S::kStages && !mbar_wait(empty(s), (it / S::kStages - 1) & 1, &s_abort, p.error, 211)) { ok = false; break; }
                        mbar_arrive_expect_tx(full(s), S::kStageBytes);
                        tma_box(dst + kABytes, &p.w, kt * kGK, wrow, full(s));
                    }
                    tma_box(dst, &p.a, kt * kGK, mt * kGM, full(s));
                }
            }
            if (!ok)                                         // a wait ran out: let the copies in flight land before the block goes
                for (unsigned back = 1; back <= (unsigned)S::kStages && back <= it; back++) {
                    const unsigned j = it - back;
                    for (unsigned w = 0; w < (1u << 16) && !mbar_try_wait(full(j % S::kStages), (j / S::kStages) & 1); w++) {}
                }
        }
        __syncwarp();
    } else if (warp == 5) {
        if (lane == 0) {
            pdl_wait();
            pdl_launch_dependents();
            read_length();
            unsigned it = 0, n = 0;
            bool ok = true;
            for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x) {
                if (p.tileExpert != nullptr && p.tileExpert[t % mTiles] < 0) continue;
                const int a = n & 1;
                if (n >= 2 && !mbar_wait(accEmpty(a), (n / 2 - 1) & 1, &s_abort, p.error, 212)) break;
                tc_fence_after();
                for (int kt = 0; kt < p.nK; kt++, it++) {
                    const int s = it % S::kStages;
                    if (!mbar_wait(full(s), (it / S::kStages) & 1, &s_abort, p.error, 213)) { ok = false; break; }
                    tc_fence_after();
                    const uint32_t sa = base + s * S::kStageBytes, sw = sa + kABytes;
#pragma unroll
                    for (int k = 0; k < kGK / 16; k++)
                        umma_f16(tmem + (uint32_t)(a * BN), desc_sw128(sa + k * 32), desc_sw128(sw + k * 32), S::kIdesc, (kt | k) != 0);
                    umma_commit(empty(s));
                }
                if (ok) umma_commit(accFull(a));
                n++;
            }
        }
        __syncwarp();
    } else {
        pdl_wait();
        pdl_launch_dependents();
        read_length();
        unsigned n = 0;
        for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
            const int mt = t % mTiles, n0 = (t / mTiles) * BN;
            if (p.tileExpert != nullptr && p.tileExpert[mt] < 0) continue;
            const int a = n & 1;
            if (!__all_sync(0xffffffffu, mbar_wait(accFull(a), (n / 2) & 1, &s_abort, p.error, 214))) break;
            tc_fence_after();
            store_tile<BN>(p, tmem + (uint32_t)(a * BN), mt * kGM + warp * 32, rows, n0, stg, warp, lane);
            tc_fence_before();
            mbar_arrive(accEmpty(a));
            n++;
        }
    }
    __syncthreads();
    if (warp == 4) { tc_fence_after(); tmem_dealloc(tmem, S::kTmem); }
}

// ───────────── two SMs on one tile ─────────────
// A cluster of two CTAs multiplies 256 × 256 tiles with tcgen05.mma of cta_group::2: each CTA holds its own 128 rows of A and half of
// the weight rows, and the tensor cores read the other half from the neighbour.  Per k-step of 16 an SM's shared memory is written
// 8 KB and read 8 KB in 135 cycles instead of 12 and 12 KB, which at 128 bytes a cycle was what bound the single-CTA form.  2048 rows through
// [40960 … 44032 × 4096] and [4096 × 15104], four layers: 3.78 ms in place of 4.03; [8192 … 22016 × 4096], [4096 × 4096 and 11008], four layers:
// 2.84 in place of 3.09.  Counters at 2048 × 4096 → 16384 (932 TFLOP/s): tensor pipe busy 46 % of the
// time, 7.3 TB/s of operands into the SMs, L2 slices at 30 % of their rate, DRAM at 11 %: no unit is near its own.
// The barriers that the MMAs wait for are the first CTA's: both CTAs' copies complete on its `full`, both CTAs' epilogue warps arrive
// on its accEmpty; a commit arrives on both CTAs' `empty` and accFull.  Everything else is the kernel above.
constexpr int kPN = 256, kPStages = 6, kPBytes = kABytes + kPN / 2 * kGK * 2;
constexpr size_t kPSmem = (size_t)kPStages * kPBytes + kEpiBytes + 1024;
constexpr uint32_t kPIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kPN >> 3) << 17) | ((uint32_t)(2 * kGM >> 4) << 24);

__device__ __forceinline__ uint32_t in_first(uint32_t addr) {            // the same place in the cluster's first CTA
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(a) : "r"(addr));
    return a;
}
__device__ __forceinline__ void tma_box_pair(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar) : "memory");
}
__device__ __forceinline__ void umma_f16_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}"
                 ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void umma_commit_pair(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"((uint16_t)3) : "memory");
}
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__global__ void __launch_bounds__(kGThreads, 1) k_bf16_gemm_pair(const __grid_constant__ GemmTcParams p) {
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ __align__(8) unsigned long long s_bar[2 * kPStages + 4];
    __shared__ uint32_t s_tmem;
    __shared__ volatile int s_abort;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, rank = (int)(blockIdx.x & 1);
    const uint32_t raw = smem_u32(smem), base = (raw + 1023u) & ~1023u;
    float* const stg = reinterpret_cast<float*>(smem + (base - raw) + (size_t)kPStages * kPBytes) + warp * (32 * 33);
    auto full = [&](int s) { return smem_u32(&s_bar[s]); };
    auto empty = [&](int s) { return smem_u32(&s_bar[kPStages + s]); };
    auto accFull = [&](int a) { return smem_u32(&s_bar[2 * kPStages + a]); };
    auto accEmpty = [&](int a) { return smem_u32(&s_bar[2 * kPStages + 2 + a]); };
    if (tid == 0) {
        for (int s = 0; s < kPStages; s++) { mbar_init(full(s), 1); mbar_init(empty(s), 1); }
        for (int a = 0; a < 2; a++) { mbar_init(accFull(a), 1); mbar_init(accEmpty(a), 8); }
        s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 4) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_barrier();                                       // both CTAs' barriers stand before anything arrives on them
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    const int tiles = p.mTiles * p.nTiles, first = (int)(blockIdx.x >> 1), stride = (int)(gridDim.x >> 1);

    if (warp == 4) {
        if (lane == 0) {
            unsigned early = 0;                              // stages whose weights were requested before the wait
            auto weights = [&](unsigned it, int kt, int n0) {
                const int s = it % kPStages;
                if (rank == 0) mbar_arrive_expect_tx(full(s), 2 * kPBytes);
                tma_box_pair(base + s * kPBytes + kABytes, &p.w, kt * kGK, n0 + rank * (kPN / 2), in_first(full(s)));
            };
            if (first < tiles)
                for (; early < (unsigned)kPStages && early < (unsigned)p.nK; early++) weights(early, (int)early, (first / p.mTiles) * kPN);
            pdl_wait();
            pdl_launch_dependents();
            unsigned it = 0;
            bool ok = true;
            for (int t = first; t < tiles && ok; t += stride) {
                const int row = (t % p.mTiles) * (2 * kGM) + rank * kGM, n0 = (t / p.mTiles) * kPN;
                for (int kt = 0; kt < p.nK; kt++, it++) {
                    const int s = it % kPStages;
                    if (it >= early) {
                        if (it >= (unsigned)kPStages && !mbar_wait(empty(s), (it / kPStages - 1) & 1, &s_abort, p.error, 215)) { ok = false; break; }
                        weights(it, kt, n0);
                    }
                    tma_box_pair(base + s * kPBytes, &p.a, kt * kGK, row, in_first(full(s)));
                }
            }
            if (!ok && rank == 0)                            // a wait ran out: let both CTAs' copies in flight land before the blocks go
                for (unsigned back = 1; back <= (unsigned)kPStages && back <= it; back++) {
                    const unsigned j = it - back;
                    for (unsigned w = 0; w < (1u << 16) && !mbar_try_wait(full(j % kPStages), (j / kPStages) & 1); w++) {}
                }
        }
        __syncwarp();
    } else if (warp == 5) {
        if (lane == 0 && rank == 0) {
            pdl_wait();
            pdl_launch_dependents();
            unsigned it = 0, n = 0;
            bool ok = true;
            for (int t = first; t < tiles && ok; t += stride) {
                const int a = n & 1;
                if (n >= 2 && !mbar_wait(accEmpty(a), (n / 2 - 1) & 1, &s_abort, p.error, 216)) break;
                tc_fence_after();
                for (int kt = 0; kt < p.nK; kt++, it++) {
                    const int s = it % kPStages;
                    if (!mbar_wait(full(s), (it / kPStages) & 1, &s_abort, p.error, 217)) { ok = false; break; }
                    tc_fence_after();
                    const uint32_t sa = base + s * kPBytes, sw = sa + kABytes;
#pragma unroll
                    for (int k = 0; k < kGK / 16; k++)
                        umma_f16_pair(tmem + (uint32_t)(a * kPN), desc_sw128(sa + k * 32), desc_sw128(sw + k * 32), kPIdesc, (kt | k) != 0);
                    umma_commit_pair(empty(s));
                }
                if (ok) umma_commit_pair(accFull(a));
                n++;
            }
        }
        __syncwarp();
    } else {
        pdl_wait();
        pdl_launch_dependents();
        unsigned n = 0;
        for (int t = first; t < tiles; t += stride) {
            const int a = n & 1;
            if (!__all_sync(0xffffffffu, mbar_wait(accFull(a), (n / 2) & 1, &s_abort, p.error, 218))) break;
            tc_fence_after();
            store_tile<kPN>(p, tmem + (uint32_t)(a * kPN), (t % p.mTiles) * (2 * kGM) + rank * kGM + warp * 32, p.M, (t / p.mTiles) * kPN, stg, warp, lane);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(in_first(accEmpty(a))) : "memory");
            n++;
        }
    }
    __syncthreads();
    cluster_barrier();                                       // neither CTA's memory is used from outside any more
    if (warp == 4) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}

bool encode_rows(CUtensorMap* map, const void* base, size_t K, size_t pitch, size_t rows, int boxRows) {
    EncodeTiledFn enc = encode_tiled_fn();
    if (!enc) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)pitch * 2};
    const cuuint32_t box[2] = {(cuuint32_t)kGK, (cuuint32_t)boxRows};
    const cuuint32_t estr[2] = {1u, 1u};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int BN>
bool run(GemmTcParams& p, const void* a, int aK, int aPitch, size_t aRows, const Bf16View& w, cudaStream_t s) {
    using S = GemmShape<BN>;
    if (!encode_rows(&p.a, a, aK, aPitch, aRows, kGM) || !encode_rows(&p.w, w.w, w.Kp, w.Kp, w.N, BN)) return false;
    static bool attr = false;
    if (!attr) {
        DJ_CUDA_CHECK(cudaFuncSetAttribute(k_bf16_gemm_tc<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::kSmem));
        attr = true;
    }
    p.nTiles = (p.N + BN - 1) / BN;
    const int grid = std::min(p.mTiles * p.nTiles, g_num_sms);
    launch_k(k_bf16_gemm_tc<BN>, dim3((unsigned)grid), dim3(kGThreads), S::kSmem, s, true, p);
    return true;
}

bool run_pair(GemmTcParams& p, const void* a, int aK, int aPitch, size_t aRows, const Bf16View& w, cudaStream_t s) {
    if (!encode_rows(&p.a, a, aK, aPitch, aRows, kGM) || !encode_rows(&p.w, w.w, w.Kp, w.Kp, w.N, kPN / 2)) return false;
    static bool attr = false;
    if (!attr) {
        DJ_CUDA_CHECK(cudaFuncSetAttribute(k_bf16_gemm_pair, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPSmem));
        attr = true;
    }
    p.mTiles = (p.M + 2 * kGM - 1) / (2 * kGM); p.nTiles = (p.N + kPN - 1) / kPN;
    const int pairs = std::min(p.mTiles * p.nTiles, g_num_sms / 2);
    launch_k_cluster(k_bf16_gemm_pair, dim3((unsigned)(2 * pairs)), dim3(kGThreads), kPSmem, s, dim3(2), p);
    return true;
}
// Rounds of pairs, in the units of the widths below.  What the pairs save is operand traffic, which bounds long reductions.  Over 32 … 3000 rows and
// 512 … 40000 outputs, where their rounds cost as much as those of the best single width, they take 1.00 of its time up to lengths of 1024, 0.99 at
// 2048, 0.96 at 4096 and beyond, and there the narrow widths fall behind by up to half.  Counted at 0.85 for all lengths they were taken for
// short ones where single tiles fill the SMs better: 640 × 2048 → 40000 254 in place of 219 µs, 768 × 512 → 4096 39.4 and 35.0, 300 × 512 → 8192 38.4 and 30.9.
constexpr int kPairLong = 3584;
double pair_cost(int M, int N, int Kp) {
    const long tiles = (long)((M + 2 * kGM - 1) / (2 * kGM)) * ((N + kPN - 1) / kPN);
    return (double)((tiles + g_num_sms / 2 - 1) / (g_num_sms / 2)) * (kPN + 24) * (Kp >= kPairLong ? 0.92 : 1.0);
}

// the tile width with the least work per SM, wider tiles first
int pick_width(int mTiles, int N, double* cost = nullptr) {
    int best = 256; double bestCost = 1e30;
    for (int bn : {256, 128, 64}) {
        const long tiles = (long)mTiles * ((N + bn - 1) / bn);
        const double c = (double)((tiles + g_num_sms - 1) / g_num_sms) * (bn + 24);
        if (c < bestCost) { bestCost = c; best = bn; }
    }
    if (cost != nullptr) *cost = bestCost;
    return best;
}
bool run_width(int bn, GemmTcParams& p, const void* a, int aK, int aPitch, size_t aRows, const Bf16View& w, cudaStream_t s) {
    return bn == 256 ? run<256>(p, a, aK, aPitch, aRows, w, s) : bn == 128 ? run<128>(p, a, aK, aPitch, aRows, w, s) : run<64>(p, a, aK, aPitch, aRows, w, s);
}

}  // namespace

// Plain form: stages a.M rows into a.ws, then multiplies.  Grouped form (tileExpert): the staged rows are in a.ws already,
// a.M of them in whole 128-row tiles, a.w holds every expert's a.nPer rows.  False when the shape does not qualify.
bool launch_bf16_gemm_tc(const Bf16LinearArgs& a, const GroupedRows* g, cudaStream_t s) {
    if (g_dev_error == nullptr || encode_tiled_fn() == nullptr || a.w.Kp % 8 != 0 || ((uintptr_t)a.ws & 15) != 0) return false;
    GemmTcParams p;
    p.M = a.M; p.N = g ? g->rowsPerExpert : a.w.N; p.nK = (a.w.Kp + kGK - 1) / kGK; p.mTiles = (a.M + kGM - 1) / kGM;
    p.tileExpert = g ? g->tileExpert : nullptr; p.rowMap = g ? g->rowMap : nullptr;
    p.residual = a.residual; p.ldr = a.ldr; p.out = a.out; p.ldo = a.ldo;
    p.gluRow = a.gluRow; p.limit = a.limit; p.glu = a.glu; p.ldglu = a.ldglu; p.softcap = a.softcap; p.bias = a.bias; p.pair = a.pair;
    p.error = g_dev_error;
    p.lenPos = nullptr; p.lenT = 0; p.outHalf = nullptr;
    if (!g) launch_stage_rows(a.a, a.b, a.w.Kp, a.M, nullptr, 1, a.ws, true, s);
    double cost;
    const int width = pick_width(p.mTiles, p.N, &cost);
    if (!g && pair_cost(a.M, p.N, a.w.Kp) <= cost && run_pair(p, a.ws, a.w.Kp, a.w.Kp, a.M, a.w, s)) return true;
    return run_width(width, p, a.ws, a.w.Kp, a.w.Kp, a.M, a.w, s);
}

void launch_bf16_gemm_rows(const __nv_bfloat16* rows, int lda, int K, const float* pos, int T, int maxRows, const Bf16View& w, __nv_bfloat16* out, int ldo,
                           cudaStream_t s) {
    GemmTcParams p = {};
    p.M = maxRows; p.N = w.N; p.nK = (K + kGK - 1) / kGK; p.mTiles = (maxRows + kGM - 1) / kGM;
    p.lenPos = pos; p.lenT = T; p.outHalf = out; p.ldo = ldo; p.gluRow = w.N; p.error = g_dev_error;
    if (lda % 8 != 0 || w.Kp % 8 != 0 || (w.N & 1) != 0 || g_dev_error == nullptr || !run_width(pick_width(p.mTiles, p.N), p, rows, K, lda, maxRows, w, s))
        throw std::runtime_error("bf16 product over cached rows: the shape does not qualify");
}

}  // namespace dj

// Which way `rows` rows of a many-row bf16 product go: out[0] = 1 for pairs of SMs and 0 for single ones, out[1] the tile width.
extern "C" int deepj_cuda_bf16_route(int32_t rows, int32_t K, int32_t N, int32_t* out) {
    if (rows < 1 || K < 1 || N < 1 || out == nullptr) { dj::set_last_error("bf16_route: bad arguments"); return 1; }
    double cost;
    const int width = dj::pick_width((rows + dj::kGM - 1) / dj::kGM, N, &cost);
    out[0] = dj::pair_cost(rows, N, dj::pad8(K)) <= cost;
    out[1] = out[0] ? dj::kPN : width;
    return 0;
}
