// gd_mlp.cu -- BF16 training and inference kernels of the collision surrogate.
//
// Network (per cell; x is the cell's distribution over the compact nodes):
//   h0 = W0 x + b0                      encoder      n_in  -> 256
//   h1 = GELU(W1 h0 + b1)               MLP          256   -> 512
//   h2 = GELU(W2 h1 + b2)                            512   -> 512
//   z  = W3 h2 + b3 + h0                (residual)   512   -> 256
//   y  = W4 z + b4                      decoder      256   -> n_out
// Every matrix product is C = A B^T on the tcgen05 tensor cores (BF16
// operands staged by TMA, FP32 accumulation in tensor memory) with the bias,
// GELU, GELU derivative or residual applied in the epilogue.  Weights are FP32
// masters with BF16 copies; Adam updates the masters.  Batch rows are cells;
// the public entry points take and return the library's [node][cell] layout.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "gd_internal.h"
#include "gd_tc.cuh"

namespace gd {
namespace {

using namespace tc;
using bf16 = __nv_bfloat16;

// GEMM tile of GM rows x GN columns (see gemm_nt), K steps of GK.
constexpr int GM = 128, GK = 64;
constexpr uint32_t kA = GM * GK * 2;
constexpr int kGThreads = 192;
constexpr uint32_t gemm_stage(int gn) { return kA + (uint32_t)gn * GK * 2; }
constexpr int kGMaxStages = 4;
// the epilogue warps' 32 x 32 tiles (rows of 33), then the stages
constexpr uint32_t kEpiTile = 32 * 33 * 4, kEpiBytes = (4 * kEpiTile + 1023) / 1024 * 1024;
constexpr size_t gemm_smem(int gn, int stages) { return 1024 + kEpiBytes + (size_t)stages * gemm_stage(gn); }

enum { EPI_NONE = 0, EPI_GELU = 1, EPI_DGELU = 2, EPI_NODE = 3 };

struct GemmArgs {
    int M, N, K;
    int stages, kps;    // stages of shared memory and K steps of each, set by gemm_nt
    const float *bias;  // [N] or null
    const float *add;   // [M][ld32] added after the bias, or null
    const float *aux;   // EPI_DGELU: pre-activation [M][ld32]
    float *pre_out;     // EPI_GELU: pre-activation out [M][ld32], or null
    float *c32;         // [M][ld32] or null
    bf16 *c16;          // [M][ld16] or null
    bf16 *c16t;         // the transpose, [N][ldt], or null
    int ld32, ld16, ldt;
    // EPI_NODE: c32 is [column][ld32], each row's values times its scale (the
    // network's output in the library's layout): columns < n_out, times
    // out_gain and, when scale2 is set, scale2[row]^2
    const float *scale2;
    float out_gain;
    int n_out;
    int *err;
    // failure-detection test hook: > 0 makes every CTA wait this many polls on
    // a barrier that nothing arrives at (before any copy or MMA is issued),
    // record the time-out, free its tensor memory and return; < 0 makes its
    // epilogue do so, with copies and MMAs in flight
    int stall_polls;
};

__device__ __forceinline__ float gelu(float x) { return 0.5f * x * (1.f + erff(x * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad(float x)
{
    return 0.5f * (1.f + erff(x * 0.70710678118654752f)) + x * 0.39894228040143268f * expf(-0.5f * x * x);
}

// After a time-out: the producer (thread 0, which has begun that many stages of the
// ring) waits for its last copies and for the MMAs that read them, the MMA thread (32)
// for the arrivals of its last accumulators.
__device__ __noinline__ void drain(int thread, int begun, int stages, uint64_t *full, uint64_t *empty, uint64_t *accf, int *err)
{
    if (thread == 0)
        for (int j = max(0, begun - stages); j < begun; j++) {
            mbar_wait(smem_u32(full + j % stages), (uint32_t)(j / stages) & 1u, err);
            mbar_wait(smem_u32(empty + j % stages), (uint32_t)(j / stages) & 1u, err);
        }
    if (thread == 32)
        for (int j = max(0, begun - 2); j < begun; j++)
            mbar_wait(smem_u32(accf + (j & 1)), (uint32_t)(j >> 1) & 1u, err);
}

// The products of one launch: G of one K, their tiles one after another.
template <int G>
struct GemmSet {
    CUtensorMap a[G], b[G];
    GemmArgs g[G];
    int end[G];  // of each product's tiles
};

// extra: the row's value of p.add (or of p.aux)
template <int EPI>
__device__ __forceinline__ void epilogue_value(const GemmArgs &p, size_t o32, float bias, float extra, float &x)
{
    if (p.bias) x += bias;
    if (EPI == EPI_DGELU) {
        x *= gelu_grad(extra);
    } else {
        if (p.add) x += extra;
        if (EPI == EPI_GELU) {
            if (p.pre_out) p.pre_out[o32] = x;
            x = gelu(x);
        }
    }
}

// C[M][N] = sum_k A[m][k] B[n][k] (A: M x K, B: N x K, both K-major BF16), in
// 128 x GN tiles, gridDim.x CTAs taking them in turn; warp 0 issues TMA, warp 1
// the MMAs into one of two accumulators, warps 2..5 read the other (row m = thread)
// and apply the epilogue.  A warp turns its 32 x 32 values in shared memory, so
// that its lanes hold 32 columns of a row and every access of C and of the added or
// multiplied arrays is one segment (a row per lane before: 32 segments of 16 bytes);
// the added or multiplied values are requested before the accumulator is awaited.
// TR: c16t is written.
template <int EPI, int GN, int G, bool TR>
__global__ void __launch_bounds__(kGThreads, 1) gemm_nt_kernel(const __grid_constant__ GemmSet<G> set)
{
    // K, the stages, err and the test hook are the first product's
    const GemmArgs p = set.g[0];
    constexpr uint32_t kStageBytes = gemm_stage(GN), kIdesc = umma_idesc_bf16(GM, GN);
    extern __shared__ __align__(1024) unsigned char dsmem[];
    unsigned char *epi = reinterpret_cast<unsigned char *>(
        (reinterpret_cast<uintptr_t>(dsmem) + 1023) & ~static_cast<uintptr_t>(1023));
    unsigned char *base = epi + kEpiBytes;
    __shared__ __align__(8) uint64_t full_bar[kGMaxStages], empty_bar[kGMaxStages], accf_bar[2], acce_bar[2], stall_bar;
    __shared__ uint32_t tmem_holder;
    __shared__ int abort_flag, gave_up;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int begun = 0;  // the producer's stages, the MMA thread's accumulators
    const int num_k = p.K / GK, GS = p.stages, KPS = p.kps, late = max(0, -p.stall_polls);
    const int tiles = set.end[G - 1];
    // product, first row and first column of a tile
    auto locate = [&](int t, int *g, int *m0, int *n0) {
        *g = 0;
        if (G > 1) {
            while (t >= set.end[*g]) (*g)++;
            if (*g > 0) t -= set.end[*g - 1];
        }
        const int mt = (set.g[*g].M + GM - 1) / GM;
        *m0 = t % mt * GM;
        *n0 = t / mt * GN;
    };

    if (threadIdx.x == 0) abort_flag = *(volatile int *)p.err;
    __syncthreads();
    if (abort_flag) return;
    if (threadIdx.x == 0) {
        gave_up = 0;
        for (int s = 0; s < GS; s++) {
            mbar_init(smem_u32(&full_bar[s]), 1);
            mbar_init(smem_u32(&empty_bar[s]), 1);
        }
        for (int b = 0; b < 2; b++) {
            mbar_init(smem_u32(&accf_bar[b]), 1);
            mbar_init(smem_u32(&acce_bar[b]), 4);  // the four epilogue warps
        }
        mbar_init(smem_u32(&stall_bar), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_holder)),
                     "r"(2 * GN)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    }
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_holder;

    if (p.stall_polls > 0) {
        // test hook: a bounded wait that must run out (stall_bar never
        // completes a phase); nothing has been issued yet, so the CTA can go
        // straight to the common exit below, which frees the tensor memory
        if (threadIdx.x == 32) mbar_wait_limit(smem_u32(&stall_bar), 0u, p.err, (uint32_t)p.stall_polls);
        __syncthreads();
        if (threadIdx.x == 0) abort_flag = *(volatile int *)p.err;
        __syncthreads();
    }

    if (abort_flag) {
        // every thread skips the work alike and meets the barrier below
    } else if (warp == 0) {
        if (lane == 0) {
            bool ok = true;
            int s = 0;
            uint32_t ph = 0;
            for (int t = blockIdx.x; ok && t < tiles; t += gridDim.x) {
                int g, m0, n0;
                locate(t, &g, &m0, &n0);
                for (int k = 0; k < num_k; k += KPS) {
                    if (!mbar_wait(smem_u32(&empty_bar[s]), ph ^ 1u, p.err)) {
                        ok = false;
                        break;
                    }
                    uint32_t st = smem_u32(base) + (uint32_t)(s * KPS) * kStageBytes;
                    const uint32_t fb = smem_u32(&full_bar[s]);
                    const int kn = min(KPS, num_k - k);
                    mbar_expect_tx(fb, (uint32_t)kn * kStageBytes);
                    for (int q = 0; q < kn; q++, st += kStageBytes) {
                        tma_load_2d(st, &set.a[g], (k + q) * GK, m0, fb);
                        tma_load_2d(st + kA, &set.b[g], (k + q) * GK, n0, fb);
                    }
                    begun++;
                    if (++s == GS) {
                        s = 0;
                        ph ^= 1u;
                    }
                }
            }
            if (!ok) gave_up = 1;
        }
    } else if (warp == 1) {
        if (lane == 0) {
            bool ok = true;
            int s = 0, i = 0;
            uint32_t ph = 0;
            for (int t = blockIdx.x; ok && t < tiles; t += gridDim.x, i++) {
                const int buf = i & 1;
                if (!mbar_wait(smem_u32(&acce_bar[buf]), ((uint32_t)(i >> 1) & 1u) ^ 1u, p.err)) {
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                for (int k = 0; k < num_k; k += KPS) {
                    if (!mbar_wait(smem_u32(&full_bar[s]), ph, p.err)) {
                        ok = false;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    uint32_t st = smem_u32(base) + (uint32_t)(s * KPS) * kStageBytes;
                    const int kn = min(KPS, num_k - k);
                    for (int q = 0; q < kn; q++, st += kStageBytes) {
#pragma unroll
                        for (int kk = 0; kk < GK / 16; kk++) {
                            const uint32_t off = (uint32_t)kk * 32u;
                            umma_bf16(tmem + (uint32_t)(buf * GN), umma_desc(st + off), umma_desc(st + kA + off),
                                      kIdesc, (k + q > 0 || kk > 0) ? 1u : 0u);
                        }
                    }
                    umma_commit(smem_u32(&empty_bar[s]));
                    if (++s == GS) {
                        s = 0;
                        ph ^= 1u;
                    }
                }
                if (ok) {
                    umma_commit(smem_u32(&accf_bar[buf]));
                    begun++;
                }
            }
            if (!ok) gave_up = 1;
        }
    } else {
        const int quad = warp & 3;
        float *tile = reinterpret_cast<float *>(epi + quad * kEpiTile);
        int i = 0;
        for (int t = blockIdx.x; t < tiles; t += gridDim.x, i++) {
            int g, m0, n0;
            locate(t, &g, &m0, &n0);
            const GemmArgs p = set.g[g];  // a copy: stores to C cannot change it
            const float *ex = EPI == EPI_DGELU ? p.aux : p.add;
            const int mw = m0 + quad * 32, m = mw + lane, rows = min(32, p.M - mw);  // the warp's first row, the lane's
            float s = 0.f;
            if (EPI == EPI_NODE && m < p.M)
                s = (p.scale2 ? __ldg(p.scale2 + m) * __ldg(p.scale2 + m) : 1.f) * p.out_gain;
            float extra[32];
            auto load_extra = [&](int n) {
                if constexpr (EPI == EPI_NONE || EPI == EPI_DGELU) {
                    if (!ex) return;
#pragma unroll
                    for (int r = 0; r < 32; r++)
                        extra[r] = r < rows && n < p.N ? ex[(size_t)(mw + r) * p.ld32 + n] : 0.f;
                }
            };
            load_extra(n0 + lane);
            const int buf = i & 1;
            bool ok = true;
            if (lane == 0)
                ok = mbar_wait_limit(late ? smem_u32(&stall_bar) : smem_u32(&accf_bar[buf]), (uint32_t)(i >> 1) & 1u, p.err,
                                     late ? (uint32_t)late : kWaitPolls);
            if (__shfl_sync(0xffffffffu, ok ? 1 : 0, 0) == 0) {
                gave_up = 1;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t taddr = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(buf * GN);
#pragma unroll 1
            for (int c0 = 0; c0 < GN; c0 += 32) {
                const int n = n0 + c0 + lane;
                const float bias = p.bias && n < p.N ? __ldg(p.bias + n) : 0.f;
                float v[32];
                tmem_ld32(taddr + (uint32_t)c0, v);
                if (c0 + 32 == GN) {
                    // the accumulator is read: the next tile but one may use it
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(smem_u32(&acce_bar[buf]));
                }
                if (EPI == EPI_NODE) {
                    // lanes hold 32 rows of a column: the output's layout
#pragma unroll
                    for (int j = 0; j < 32; j++) {
                        float x = v[j];
                        epilogue_value<EPI>(p, 0, __shfl_sync(0xffffffffu, bias, j), 0.f, x);
                        if (m < p.M && n0 + c0 + j < p.n_out) p.c32[(size_t)(n0 + c0 + j) * p.ld32 + m] = x * s;
                    }
                } else {
                    if (c0 > 0) load_extra(n);
#pragma unroll
                    for (int j = 0; j < 32; j++) tile[lane * 33 + j] = v[j];
                    __syncwarp();
                    if (n < p.N) {
#pragma unroll
                        for (int r = 0; r < 32; r++) {
                            if (r >= rows) continue;
                            float x = tile[r * 33 + lane];
                            epilogue_value<EPI>(p, (size_t)(mw + r) * p.ld32 + n, bias, extra[r], x);
                            if (p.c32) p.c32[(size_t)(mw + r) * p.ld32 + n] = x;
                            if (p.c16) p.c16[(size_t)(mw + r) * p.ld16 + n] = __float2bfloat16_rn(x);
                            if (TR) tile[r * 33 + lane] = x;
                        }
                    }
                    __syncwarp();
                    if (TR) {
#pragma unroll
                        for (int j = 0; j < 32; j++)
                            if (n0 + c0 + j < p.N && m < p.M)
                                p.c16t[(size_t)(n0 + c0 + j) * p.ldt + m] = __float2bfloat16_rn(tile[lane * 33 + j]);
                        __syncwarp();
                    }
                }
            }
        }
    }
    __syncthreads();
    if (gave_up) {
        // a wait of this CTA timed out: the copies in flight land, the MMAs that
        // read them and the arrivals on their way are done before it leaves (waits
        // that run out by themselves too)
        drain(threadIdx.x, begun, GS, full_bar, empty_bar, accf_bar, p.err);
        __syncthreads();
    }
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * GN) : "memory");
    }
}

// C[M][N] = A_hi B_hi^T + A_hi B_lo^T + A_lo B_hi^T (FP32) for K-major BF16
// operands: the FP32-equivalent product of two BF16 hi/lo splits, in one
// launch.  The tensor cores' FP32 accumulation loses bits over long sums, so
// the K range runs in chunks of kchunk 64-column steps: each chunk goes into
// one of two tensor-memory accumulators, and the epilogue adds the chunks, in
// chunk order, into FP32 sums it holds in registers (one row and 128 columns
// per thread).  One 128 x 128 tile per CTA; warp 0 issues TMA, warp 1 the
// MMAs (three per 16-column K step), warps 2..5 the epilogue.  Every wait is
// bounded.
constexpr int XM = 128, XN = 128, XS = 3;
constexpr uint32_t kXA = XM * GK * 2, kXB = XN * GK * 2, kXStage = 2 * kXA + 2 * kXB;  // 64 KB
constexpr uint32_t kXIdesc = umma_idesc_bf16(XM, XN);
constexpr size_t kX3Smem = XS * kXStage + 1024;

struct Gemm3Args {
    int M, N, K, kchunk;  // K and kchunk in elements (multiples of 64)
    float *c;
    int ldc;
    int *err;
    int stall_polls;  // failure-detection test hook, as in GemmArgs
};

__global__ void __launch_bounds__(kGThreads, 1)
    gemm3_nt_kernel(const __grid_constant__ CUtensorMap tAh, const __grid_constant__ CUtensorMap tAl,
                    const __grid_constant__ CUtensorMap tBh, const __grid_constant__ CUtensorMap tBl, Gemm3Args p)
{
    extern __shared__ __align__(1024) unsigned char dsmem[];
    unsigned char *base = reinterpret_cast<unsigned char *>(
        (reinterpret_cast<uintptr_t>(dsmem) + 1023) & ~static_cast<uintptr_t>(1023));
    __shared__ __align__(8) uint64_t full_bar[XS], empty_bar[XS], accf_bar[2], acce_bar[2], stall_bar;
    __shared__ uint32_t tmem_holder;
    __shared__ int abort_flag, gave_up;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int begun = 0;  // as in gemm_nt_kernel
    const int m0 = blockIdx.x * XM, n0 = blockIdx.y * XN;
    const int num_k = p.K / GK, kcs = p.kchunk / GK, late = max(0, -p.stall_polls);
    const int nchunks = (num_k + kcs - 1) / kcs;

    if (threadIdx.x == 0) abort_flag = *(volatile int *)p.err;
    __syncthreads();
    if (abort_flag) return;
    if (threadIdx.x == 0) {
        gave_up = 0;
        for (int s = 0; s < XS; s++) {
            mbar_init(smem_u32(&full_bar[s]), 1);
            mbar_init(smem_u32(&empty_bar[s]), 1);
        }
        for (int b = 0; b < 2; b++) {
            mbar_init(smem_u32(&accf_bar[b]), 1);
            mbar_init(smem_u32(&acce_bar[b]), 4);  // the four epilogue warps
        }
        mbar_init(smem_u32(&stall_bar), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_holder)),
                     "r"(2 * XN)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    }
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_holder;

    if (p.stall_polls > 0) {
        // test hook: a bounded wait that must run out before anything is issued
        if (threadIdx.x == 32) mbar_wait_limit(smem_u32(&stall_bar), 0u, p.err, (uint32_t)p.stall_polls);
        __syncthreads();
        if (threadIdx.x == 0) abort_flag = *(volatile int *)p.err;
        __syncthreads();
    }

    if (abort_flag) {
        // every thread skips the work alike and meets the barrier below
    } else if (warp == 0) {
        if (lane == 0) {
            for (int k = 0; k < num_k; k++) {
                const int s = k % XS;
                const uint32_t ph = (uint32_t)(k / XS) & 1u;
                if (!mbar_wait(smem_u32(&empty_bar[s]), ph ^ 1u, p.err)) {
                    gave_up = 1;
                    break;
                }
                unsigned char *st = base + (size_t)s * kXStage;
                const uint32_t fb = smem_u32(&full_bar[s]);
                mbar_expect_tx(fb, kXStage);
                tma_load_2d(smem_u32(st), &tAh, k * GK, m0, fb);
                tma_load_2d(smem_u32(st + kXA), &tAl, k * GK, m0, fb);
                tma_load_2d(smem_u32(st + 2 * kXA), &tBh, k * GK, n0, fb);
                tma_load_2d(smem_u32(st + 2 * kXA + kXB), &tBl, k * GK, n0, fb);
                begun++;
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            bool ok = true;
            int k = 0;
            for (int c = 0; ok && c < nchunks; c++) {
                const int buf = c & 1;
                if (!mbar_wait(smem_u32(&acce_bar[buf]), ((uint32_t)(c >> 1) & 1u) ^ 1u, p.err)) {
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t d_tmem = tmem + (uint32_t)(buf * XN);
                const int kend = min(num_k, k + kcs);
                for (const int kbeg = k; k < kend; k++) {
                    const int s = k % XS;
                    if (!mbar_wait(smem_u32(&full_bar[s]), (uint32_t)(k / XS) & 1u, p.err)) {
                        ok = false;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t st = smem_u32(base + (size_t)s * kXStage);
                    const uint32_t aH = st, aL = st + kXA, bH = st + 2 * kXA, bL = st + 2 * kXA + kXB;
#pragma unroll
                    for (int kk = 0; kk < GK / 16; kk++) {
                        const uint32_t off = (uint32_t)kk * 32u;
                        umma_bf16(d_tmem, umma_desc(aH + off), umma_desc(bH + off), kXIdesc,
                                  (k > kbeg || kk > 0) ? 1u : 0u);
                        umma_bf16(d_tmem, umma_desc(aH + off), umma_desc(bL + off), kXIdesc, 1u);
                        umma_bf16(d_tmem, umma_desc(aL + off), umma_desc(bH + off), kXIdesc, 1u);
                    }
                    umma_commit(smem_u32(&empty_bar[s]));
                }
                if (ok) {
                    umma_commit(smem_u32(&accf_bar[buf]));
                    begun++;
                }
            }
            if (!ok) gave_up = 1;
        }
    } else {
        const int quad = warp & 3;
        const int m = m0 + quad * 32 + lane;
        float sum[XN];
#pragma unroll
        for (int j = 0; j < XN; j++) sum[j] = 0.f;
        bool ok = true;
        for (int c = 0; ok && c < nchunks; c++) {
            const int buf = c & 1;
            bool w = true;
            if (lane == 0)
                w = mbar_wait_limit(late ? smem_u32(&stall_bar) : smem_u32(&accf_bar[buf]), (uint32_t)(c >> 1) & 1u, p.err,
                                    late ? (uint32_t)late : kWaitPolls);
            if (__shfl_sync(0xffffffffu, w ? 1 : 0, 0) == 0) {
                ok = false;
                gave_up = 1;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t taddr = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(buf * XN);
#pragma unroll
            for (int c0 = 0; c0 < XN; c0 += 32) {
                float v[32];
                tmem_ld32(taddr + (uint32_t)c0, v);
#pragma unroll
                for (int j = 0; j < 32; j++) sum[c0 + j] += v[j];
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&acce_bar[buf]));
        }
        if (ok && m < p.M) {
            float *row = p.c + (size_t)m * p.ldc;
#pragma unroll
            for (int j = 0; j < XN; j += 4) {
                const int n = n0 + j;
                if (n + 4 <= p.N) {
                    *reinterpret_cast<float4 *>(row + n) = make_float4(sum[j], sum[j + 1], sum[j + 2], sum[j + 3]);
                } else {
#pragma unroll
                    for (int q = 0; q < 4; q++)
                        if (n + q < p.N) row[n + q] = sum[j + q];
                }
            }
        }
    }
    __syncthreads();
    if (gave_up) {
        drain(threadIdx.x, begun, XS, full_bar, empty_bar, accf_bar, p.err);
        __syncthreads();
    }
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * XN) : "memory");
    }
}

// out[c][r] = in[r][c] for BF16 [R][C] (row strides ldi, ldo)
__global__ void transpose_bf16_kernel(const bf16 *__restrict__ in, int R, int Cc, int ldi, bf16 *__restrict__ out,
                                      int ldo)
{
    __shared__ bf16 tile[32][34];
    const int r0 = blockIdx.y * 32, c0 = blockIdx.x * 32;
    for (int y = threadIdx.y; y < 32; y += blockDim.y) {
        const int r = r0 + y, c = c0 + threadIdx.x;
        tile[y][threadIdx.x] = (r < R && c < Cc) ? in[(size_t)r * ldi + c] : __float2bfloat16_rn(0.f);
    }
    __syncthreads();
    for (int y = threadIdx.y; y < 32; y += blockDim.y) {
        const int c = c0 + y, r = r0 + threadIdx.x;
        if (c < Cc && r < R) out[(size_t)c * ldo + r] = tile[threadIdx.x][y];
    }
}

// FP32 [R][C] (ld ldi) -> BF16 [R][C_pad] (ld ldo), zero columns C..C_pad
__global__ void to_bf16_kernel(const float *__restrict__ in, int R, int Cc, int ldi, int C_pad, bf16 *__restrict__ out,
                               int ldo)
{
    const int64_t total = (int64_t)R * C_pad;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
        const int r = (int)(t / C_pad), c = (int)(t % C_pad);
        out[(size_t)r * ldo + c] = __float2bfloat16_rn(c < Cc ? in[(size_t)r * ldi + c] : 0.f);
    }
}

// Sum over r < rows of src[r][col] (or of the squares), one chain in the order
// of r: a block of 32 columns x 32 warps copies the rows ahead into a ring of
// shared memory while the first warp adds.  Bound by the chain of additions (4
// cycles each); a thread per column that loads as it adds waits for memory
// instead (3648 rows: 240 -> 17 us; 1024 rows: 60 -> 6.5 us).  Four-byte copies
// alone: 22 and 8.4 us.
constexpr int kOrdPer = 4, kOrdRows = 32 * kOrdPer, kOrdStages = 6;  // rows per thread and per stage
constexpr size_t kOrdSmem = (size_t)kOrdStages * kOrdRows * 32 * sizeof(float);
template <bool SQUARE>
__device__ __forceinline__ float ordered_sum(const float *__restrict__ src, int rows, size_t ld, int col, bool live)
{
    extern __shared__ __align__(16) float ord_ring[];  // [stage][row][column]
    const int x = threadIdx.x, y = threadIdx.y;
    const int chunks = (rows + kOrdRows - 1) / kOrdRows;
    // a block whose columns all exist, in rows of 16-byte alignment, copies 16
    // bytes per thread (four rows per warp) instead of 4
    const int col0 = col - x;
    const bool wide = __all_sync(0xffffffffu, live) && (ld & 3) == 0 &&
                      ((reinterpret_cast<uintptr_t>(src) + 4 * (size_t)col0) & 15) == 0;
    const int per = wide ? 1 : kOrdPer, x0 = wide ? 4 * (x & 7) : x, y0 = wide ? 4 * y + (x >> 3) : y;
    const float *p = src + (size_t)y0 * ld + (wide ? col0 + x0 : live ? col : 0);
    const size_t step = (size_t)(kOrdRows / per) * ld;
    const uint32_t ring = smem_u32(ord_ring + 32 * y0 + x0), ring_end = ring + (uint32_t)kOrdSmem;
    uint32_t dst = ring;
    int row = y0;
    auto fetch = [&]() {
        if (wide) {
            if (row < rows)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(p) : "memory");
            p += step;
            row += kOrdRows;
        } else {
#pragma unroll
            for (int k = 0; k < kOrdPer; k++, p += step, row += 32)
                if (row < rows)
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst + k * 32 * 128), "l"(p)
                                 : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        dst += kOrdRows * 128;
        if (dst == ring_end) dst = ring;
    };
    float s = 0.f;
    for (int c = 0; c < kOrdStages - 1; c++) fetch();
    for (int c = 0; c < chunks; c++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kOrdStages - 2) : "memory");
        __syncthreads();  // chunk c is in, and everyone is done with chunk c - 1
        fetch();
        if (y == 0) {
            const int n = min(kOrdRows, rows - c * kOrdRows);
            const float *t = ord_ring + (c % kOrdStages) * kOrdRows * 32 + x;
            const uint32_t at = smem_u32(t);
            auto ld16 = [&](int r, float *u) {
#pragma unroll
                for (int q = 0; q < 16; q++)
                    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(u[q]) : "r"(at + (r + q) * 128));
            };
            auto add16 = [&](const float *u) {
#pragma unroll
                for (int q = 0; q < 16; q++) {
                    if (SQUARE) s += u[q] * u[q];
                    else s += u[q];
                }
            };
            int r = 0;
            if (n == kOrdRows) {
                float u[16], w[16];
                ld16(0, u);
#pragma unroll
                for (; r < kOrdRows; r += 32) {
                    ld16(r + 16, w);
                    add16(u);
                    if (r + 32 < kOrdRows) ld16(r + 32, u);
                    add16(w);
                }
            }
            for (; r < n; r++) {
                const float u = t[r * 32];
                if (SQUARE) s += u * u;
                else s += u;
            }
        }
    }
    return s;
}

template <typename... P, typename... A>
int launch_ordered(void (*kern)(P...), dim3 grid, cudaStream_t st, A... a)
{
    GD_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kOrdSmem));
    kern<<<grid, dim3(32, 32), kOrdSmem, st>>>(a...);
    GD_CUDA(cudaGetLastError());
    return GD_OK;
}

// Per-cell scale: mean of x over the n nodes (fixed order), or 1; in the blocks of
// a second row, the sum of squares of d over m nodes.  Block = 32 cells x 32 warps.
__global__ void __launch_bounds__(1024) cell_sums_kernel(const float *__restrict__ x, int n, int ldx, int use_mean,
                                                         float *__restrict__ scale, const float *__restrict__ d, int m,
                                                         int ldd, float *__restrict__ squares, int B)
{
    const int r = blockIdx.x * 32 + threadIdx.x;
    const bool live = r < B;
    if (blockIdx.y == 0) {
        const float s = use_mean ? ordered_sum<false>(x, n, ldx, r, live) / (float)n : 1.f;
        if (live && threadIdx.y == 0) scale[r] = s;
    } else {
        const float s = ordered_sum<true>(d, m, ldd, r, live);
        if (live && threadIdx.y == 0) squares[r] = s;
    }
}

__device__ __forceinline__ float inv_or_zero(float s) { return s != 0.f ? 1.f / s : 0.f; }

// Loss denominators per cell from the sums of squares in den: scaled like the
// targets for the relative losses, or n for the mean squared error; with mean set
// their mean over the batch (fixed order).  One block of 256 threads, beside those
// that copy the input.
struct DenArgs {
    float *den;  // null: nothing to do
    int pw;
    float inv_gain;
    int mse, n, mean;
};
__device__ __forceinline__ void denominators(const DenArgs &a, int B, const float *__restrict__ scale, double *s)
{
    const int t = threadIdx.y * 32 + threadIdx.x;
    double sum = 0.0;
    for (int i = t; i < B; i += 256) {
        const float sc = (a.pw ? inv_or_zero(scale[i] * scale[i]) : 1.f) * a.inv_gain;
        const float v = a.mse ? (float)a.n : a.den[i] * sc * sc;
        a.den[i] = v;
        sum += v;
    }
    if (!a.mean) return;
    s[t] = sum;
    __syncthreads();
    for (int k = 128; k > 0; k >>= 1) {
        if (t < k) s[t] += s[t + k];
        __syncthreads();
    }
    const float m = (float)(s[0] / B);
    for (int i = t; i < B; i += 256) a.den[i] = m;
}

// node-major FP32 x[i][r] (ld) -> cell-major BF16 xb[r][i] * gain / scale[r] (pad to
// n_p), for training also its transpose xt[i][r].  Block = 64 nodes x 32 cells: eight loads in flight per thread and whole
// 128-byte rows on both sides (4096 cells, 3648 nodes: 39 -> 15 us).
template <bool TRANSPOSE>
__global__ void gather_in_kernel(const float *__restrict__ x, int n, int ld, int B, const float *__restrict__ scale,
                                 float gain, bf16 *__restrict__ xb, bf16 *__restrict__ xt, int n_p, DenArgs den)
{
    __shared__ __align__(8) float tile[64][33];
    if ((int)blockIdx.y == n_p / 64) {  // the row past the nodes: the denominators
        if (blockIdx.x == 0) denominators(den, B, scale, reinterpret_cast<double *>(&tile[0][0]));
        return;
    }
    const int i0 = blockIdx.y * 64, r0 = blockIdx.x * 32, r = r0 + threadIdx.x;
    const float s = r < B ? inv_or_zero(scale[r]) * gain : 0.f;
    float v[8];
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const int i = i0 + threadIdx.y + 8 * k;
        v[k] = i < n && r < B ? __ldg(x + (size_t)i * ld + r) : 0.f;
    }
#pragma unroll
    for (int k = 0; k < 8; k++) {
        v[k] *= s;
        tile[threadIdx.y + 8 * k][threadIdx.x] = v[k];
        if (TRANSPOSE && r < B) xt[(size_t)(i0 + threadIdx.y + 8 * k) * B + r] = __float2bfloat16_rn(v[k]);
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const int y = threadIdx.y + 8 * k, c = 2 * threadIdx.x;
        if (r0 + y < B)
            *reinterpret_cast<__nv_bfloat162 *>(xb + (size_t)(r0 + y) * n_p + i0 + c) =
                __floats2bfloat162_rn(tile[c][y], tile[c + 1][y]);
    }
}

// Loss of cell r: the sum of the node tiles' errors / den[r].
__device__ __forceinline__ float cell_loss(const float *__restrict__ err_part, int tiles, int B,
                                           const float *__restrict__ den, int r)
{
    float e = 0.f;
#pragma unroll 8
    for (int k = 0; k < tiles; k++) e += __ldg(err_part + (size_t)k * B + r);
    return e / fmaxf(den[r], 1e-30f);
}
__global__ void row_err_kernel(const float *__restrict__ err_part, int tiles, int B, const float *__restrict__ den,
                               float *__restrict__ row_err)
{
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r < B) row_err[r] = cell_loss(err_part, tiles, B, den, r);
}

// The cells' losses and their mean over the batch (fixed order), by one block of 1024.
struct MeanLoss {
    const float *err_part;
    int tiles;
    const float *den;
    float *row_err, *out;
};
__device__ __forceinline__ void mean_loss(const MeanLoss &m, int B, double *s)
{
    const int t = threadIdx.y * 32 + threadIdx.x;
    double a = 0.0;
    for (int r = t; r < B; r += 1024) {
        const float e = cell_loss(m.err_part, m.tiles, B, m.den, r);
        m.row_err[r] = e;
        a += e;
    }
    s[t] = a;
    __syncthreads();
    for (int k = 512; k > 0; k >>= 1) {
        if (t < k) s[t] += s[t + k];
        __syncthreads();
    }
    if (t == 0) *m.out = (float)(s[0] / B);
}

// The layers' bias gradients: column sums gb[n] = sum_r d[r][n], r < R (fixed
// order).  Block = 32 columns x 32 warps, layer by layer; one block past them the
// batch's loss.
struct ColSums {
    const float *d[5];
    float *out[5];
    int n[5], end[5];  // columns; end of the layer's blocks
};
__global__ void __launch_bounds__(1024) colsum_kernel(const __grid_constant__ ColSums c, int R, MeanLoss loss)
{
    if ((int)blockIdx.x == c.end[4]) {
        extern __shared__ __align__(16) float ord_ring[];
        mean_loss(loss, R, reinterpret_cast<double *>(ord_ring));
        return;
    }
    int g = 0;
    while ((int)blockIdx.x >= c.end[g]) g++;
    const int n = ((int)blockIdx.x - (g > 0 ? c.end[g - 1] : 0)) * 32 + threadIdx.x;
    const bool live = n < c.n[g];
    const float s = ordered_sum<false>(c.d[g], R, c.n[g], n, live);
    if (live && threadIdx.y == 0) c.out[g][n] = s;
}

// Output gradient dy = 2 (y - t') / den / B with t'[r][i] = t[i][r] inv_gain /
// scale[r]^2 (the scale only when pw): FP32 dy and BF16 dyb [r][n_p], its transpose
// dyt [n_p][B] when set, and per 64 nodes the sum of (y - t')^2 in
// err_part[node tile][r].  Block = 64 nodes x 32 cells.
__global__ void loss_grad_kernel(const float *__restrict__ y, const float *__restrict__ t, int ldt, int n, int n_p,
                                 int B, const float *__restrict__ scale, int pw, float inv_gain,
                                 const float *__restrict__ den, float *__restrict__ dy, bf16 *__restrict__ dyb,
                                 bf16 *__restrict__ dyt, float *__restrict__ err_part)
{
    __shared__ float tile[64][33];
    const int i0 = blockIdx.y * 64, r0 = blockIdx.x * 32, tx = threadIdx.x, ty = threadIdx.y;
    {
        const int r = r0 + tx;
        const float s = r < B ? (pw ? inv_or_zero(scale[r] * scale[r]) : 1.f) * inv_gain : 0.f;
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const int i = i0 + ty + 8 * k;
            tile[ty + 8 * k][tx] = i < n && r < B ? __ldg(t + (size_t)i * ldt + r) * s : 0.f;
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const int yy = ty + 8 * k, r = r0 + yy, i = i0 + 2 * tx;
        if (r >= B) continue;  // the whole warp
        const float dr = fmaxf(den[r], 1e-30f);
        const float2 v = *reinterpret_cast<const float2 *>(y + (size_t)r * n_p + i);
        float2 g = make_float2(0.f, 0.f);
        float e = 0.f;
        if (i < n) {
            const float d = v.x - tile[2 * tx][yy];
            e += d * d;
            g.x = 2.f * d / dr / (float)B;
        }
        if (i + 1 < n) {
            const float d = v.y - tile[2 * tx + 1][yy];
            e += d * d;
            g.y = 2.f * d / dr / (float)B;
        }
        *reinterpret_cast<float2 *>(dy + (size_t)r * n_p + i) = g;
        *reinterpret_cast<__nv_bfloat162 *>(dyb + (size_t)r * n_p + i) = __floats2bfloat162_rn(g.x, g.y);
        tile[2 * tx][yy] = g.x;
        tile[2 * tx + 1][yy] = g.y;
        for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
        if (tx == 0) err_part[(size_t)blockIdx.y * B + r] = e;
    }
    if (!dyt) return;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 8; k++)
        if (r0 + tx < B) dyt[(size_t)(i0 + ty + 8 * k) * B + r0 + tx] = __float2bfloat16_rn(tile[ty + 8 * k][tx]);
}

// Adam (decoupled weight decay) on the FP32 masters of all layers; writes the BF16
// copies and their transposes (bound by its bytes, 32 per weight, from L2: one
// launch instead of fourteen, 55 -> 20 us).  Block = 32 x 32 of a weight matrix, or
// 1024 of a bias; threads 32 x 8.
struct AdamSet {
    struct {
        float *w, *b, *mw, *vw, *mb, *vb;
        const float *gw, *gb;
        bf16 *wb, *wt;
        int out, in, wend, bend;  // ends of the weight's and of the bias's blocks
    } l[5];
    float lr, b1, b2, c1, c2, eps, wd;
};
__device__ __forceinline__ float adam(const AdamSet &a, float *w, const float *g, float *m, float *v, size_t i, float wd)
{
    const float gi = g[i];
    const float mi = __fmaf_rn(1.f - a.b1, gi, __fmul_rn(a.b1, m[i]));
    const float vi = __fmaf_rn(__fmul_rn(1.f - a.b2, gi), gi, __fmul_rn(a.b2, v[i]));
    m[i] = mi;
    v[i] = vi;
    const float upd = __fmaf_rn(wd, w[i], (mi / a.c1) / (sqrtf(vi / a.c2) + a.eps));
    const float wn = __fmaf_rn(-a.lr, upd, w[i]);
    w[i] = wn;
    return wn;
}
__global__ void adam_kernel(const __grid_constant__ AdamSet a)
{
    __shared__ float tile[32][33];
    int k = 0;
    while ((int)blockIdx.x >= a.l[k].bend) k++;
    const auto &l = a.l[k];
    const int blk = (int)blockIdx.x - (k > 0 ? a.l[k - 1].bend : 0), nw = l.wend - (k > 0 ? a.l[k - 1].bend : 0);
    if (blk >= nw) {
        const int i0 = (blk - nw) * 1024;
        for (int i = i0 + threadIdx.y * 32 + threadIdx.x; i < min(i0 + 1024, l.out); i += 256)
            adam(a, l.b, l.gb, l.mb, l.vb, i, 0.f);
        return;
    }
    // out and in are multiples of 32
    const int cols = l.in / 32, o0 = blk / cols * 32, i0 = blk % cols * 32;
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const int y = threadIdx.y + 8 * q;
        const size_t i = (size_t)(o0 + y) * l.in + i0 + threadIdx.x;
        const float wn = adam(a, l.w, l.gw, l.mw, l.vw, i, a.wd);
        l.wb[i] = __float2bfloat16_rn(wn);
        tile[y][threadIdx.x] = wn;
    }
    if (!l.wt) return;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const int y = threadIdx.y + 8 * q;
        l.wt[(size_t)(i0 + y) * l.out + o0 + threadIdx.x] = __float2bfloat16_rn(tile[threadIdx.x][y]);
    }
}

using EncodeTiled = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                 const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiled encoder()
{
    static EncodeTiled fn = nullptr;
    if (!fn) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiled>(p);
    }
    return fn;
}

// 2-D map over a K-major BF16 matrix [rows][K] (row stride K), box 64 x box_rows
int make_map(CUtensorMap *m, const bf16 *ptr, int rows, int K, int box_rows)
{
    EncodeTiled fn = encoder();
    if (!fn) return set_error(GD_ERR_CUDA, "cuTensorMapEncodeTiled is not available");
    const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    const cuuint64_t str[1] = {(cuuint64_t)K * 2};
    const cuuint32_t box[2] = {GK, (cuuint32_t)box_rows}, es[2] = {1, 1};
    CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<bf16 *>(ptr), dims, str, box, es,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return set_error(GD_ERR_CUDA, "tensor map encoding failed (" + std::to_string((int)r) + ")");
    return GD_OK;
}

// One of the products of a launch.
struct Product {
    const bf16 *A, *B;
    GemmArgs a;
};

template <int EPI, int GN, int G>
int launch_gemm(const Product *pr, int kps, int stages, int ctas, cudaStream_t st)
{
    GemmSet<G> set;
    int end = 0;
    for (int g = 0; g < G; g++) {
        int rc = make_map(&set.a[g], pr[g].A, pr[g].a.M, pr[g].a.K, GM);
        if (!rc) rc = make_map(&set.b[g], pr[g].B, pr[g].a.N, pr[g].a.K, GN);
        if (rc) return rc;
        set.g[g] = pr[g].a;
        set.g[g].kps = kps;
        set.g[g].stages = stages;
        set.end[g] = end += (pr[g].a.M + GM - 1) / GM * ((pr[g].a.N + GN - 1) / GN);
    }
    const size_t smem = gemm_smem(GN, stages * kps);
    // one product, not the output's layout: with or without the transpose
    auto kern = gemm_nt_kernel<EPI, GN, G, false>;
    if constexpr (G == 1 && EPI != EPI_NODE)
        if (pr[0].a.c16t) kern = gemm_nt_kernel<EPI, GN, G, true>;
    GD_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kern<<<std::min(end, ctas), kGThreads, smem, st>>>(set);
    GD_CUDA(cudaGetLastError());
    return GD_OK;
}

// C = A B^T with A [M][K], B [N][K] (BF16, row stride K), K % 64 == 0, for G
// products of one K in one launch; output strides ld32, ld16 multiples of 4.
//
// Tile width, K steps per stage and stages.  A K of up to 8 steps (every layer
// but the first and the weights' gradients): 32 columns and two CTAs per SM,
// since a CTA's fixed costs and its epilogue bound it (1024 x 512, K = 512: 10 us;
// 13 with 64 columns, 20 with 128, 34 with 256; 4096 x 3648, K = 256: 26 us, 36
// with 64, 33 with 128).  A longer K is bound by the handshakes and copies of its
// stages: four steps in each, in the narrowest tiles that one wave holds (1024 x
// 256, K = 3648: 17 us with 32 columns, 18 with 64, 27 with 128, one step per
// stage 24; 4096 x 256: 22 us with 64 columns, 32 with 32).
template <int G>
int gemm_nt(int epi, const Product *pr, cudaStream_t st)
{
    int dev = 0, sms = 0;
    GD_CUDA(cudaGetDevice(&dev));
    GD_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const int K = pr[0].a.K;
    for (int g = 0; g < G; g++) {
        const GemmArgs &a = pr[g].a;
        if (a.K != K || K % GK || K <= 0 || a.M <= 0 || a.N <= 0 || (epi != EPI_NODE && ((a.ld32 & 3) || (a.ld16 & 3))))
            return set_error(GD_ERR_INVALID_ARG, "GEMM shape: K a multiple of 64, strides multiples of 4");
    }
    const int num_k = K / GK;
    auto tiles = [&](int gn) {
        int n = 0;
        for (int g = 0; g < G; g++) n += (pr[g].a.M + GM - 1) / GM * ((pr[g].a.N + gn - 1) / gn);
        return n;
    };
    if (num_k <= 8) {
        if (epi == EPI_NONE) return launch_gemm<EPI_NONE, 32, G>(pr, 2, 2, 2 * sms, st);
        if (G == 1 && epi == EPI_GELU) return launch_gemm<EPI_GELU, 32, 1>(pr, 2, 2, 2 * sms, st);
        if (G == 1 && epi == EPI_DGELU) return launch_gemm<EPI_DGELU, 32, 1>(pr, 2, 2, 2 * sms, st);
        if (G == 1 && epi == EPI_NODE) return launch_gemm<EPI_NODE, 32, 1>(pr, 2, 2, 2 * sms, st);
    } else if (epi == EPI_NONE) {
        const int steps = (num_k + 3) / 4;  // stages of four
        if (tiles(32) <= sms) return launch_gemm<EPI_NONE, 32, G>(pr, 4, std::min(steps, 2), sms, st);
        if (tiles(64) <= sms) return launch_gemm<EPI_NONE, 64, G>(pr, 4, std::min(steps, 2), sms, st);
        if (tiles(128) <= sms) return launch_gemm<EPI_NONE, 128, G>(pr, 2, 3, sms, st);
        return launch_gemm<EPI_NONE, 256, G>(pr, 2, 2, sms, st);
    }
    return set_error(GD_ERR_INVALID_ARG, "unknown GEMM epilogue for this K");
}

int gemm_nt(int epi, const bf16 *A, const bf16 *B, const GemmArgs &a, cudaStream_t st)
{
    const Product p{A, B, a};
    return gemm_nt<1>(epi, &p, st);
}

int transpose(const bf16 *in, int R, int Cc, int ldi, bf16 *out, int ldo, cudaStream_t st)
{
    dim3 b(32, 8), g((Cc + 31) / 32, (R + 31) / 32);
    transpose_bf16_kernel<<<g, b, 0, st>>>(in, R, Cc, ldi, out, ldo);
    GD_CUDA(cudaGetLastError());
    return GD_OK;
}

int pad64(int n) { return (n + 63) / 64 * 64; }

}  // namespace

// C[M][N] (FP32, row stride ldc) = A_hi B_hi^T + A_hi B_lo^T + A_lo B_hi^T for
// K-major BF16 [M][K] and [N][K] operands, in one launch, the tensor cores
// summing at most k_chunk products per FP32 accumulation (the chunks added in
// FP32 in chunk order); the collision-matrix path computes the loss with it.
int gemm_bf16x3_nt_f32(const void *Ah, const void *Al, int M, const void *Bh, const void *Bl, int N, int K, float *C,
                       int ldc, int *err, cudaStream_t st, int stall_polls, int k_chunk)
{
    if (K % GK || K <= 0 || M <= 0 || N <= 0 || (ldc & 3) || k_chunk <= 0 || k_chunk % GK ||
        (reinterpret_cast<uintptr_t>(C) & 15))
        return set_error(GD_ERR_INVALID_ARG, "GEMM shape: K and the chunk multiples of 64, ldc a multiple of 4");
    CUtensorMap tAh, tAl, tBh, tBl;
    int rc = make_map(&tAh, static_cast<const bf16 *>(Ah), M, K, XM);
    if (!rc) rc = make_map(&tAl, static_cast<const bf16 *>(Al), M, K, XM);
    if (!rc) rc = make_map(&tBh, static_cast<const bf16 *>(Bh), N, K, XN);
    if (!rc) rc = make_map(&tBl, static_cast<const bf16 *>(Bl), N, K, XN);
    if (rc) return rc;
    Gemm3Args a{M, N, K, k_chunk, C, ldc, err, stall_polls};
    dim3 grid((M + XM - 1) / XM, (N + XN - 1) / XN);
    GD_CUDA(cudaFuncSetAttribute(gemm3_nt_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kX3Smem));
    gemm3_nt_kernel<<<grid, kGThreads, kX3Smem, st>>>(tAh, tAl, tBh, tBl, a);
    GD_CUDA(cudaGetLastError());
    return GD_OK;
}

}  // namespace gd

using gd::bf16;

struct gd_mlp {
    struct Layer {
        int out = 0, in = 0;  // padded
        float *w = nullptr, *b = nullptr, *gw = nullptr, *gb = nullptr;
        float *mw = nullptr, *vw = nullptr, *mb = nullptr, *vb = nullptr;
        bf16 *wb = nullptr, *wt = nullptr;  // BF16 copy [out][in] and its transpose [in][out]
    };
    int n_in = 0, n_out = 0, n_in_p = 0, n_out_p = 0, cap = 0, flags = 0;
    int device = 0;
    float in_gain = 1.f, out_gain = 1.f;  // global input / output normalisation
    Layer L[5];
    int64_t step = 0;
    int stall_next = 0;  // gd_mlp_inject_timeout: polls for the next forward's first GEMM (late: negative)
    // activations, [cap][features]
    bf16 *xb = nullptr, *h0b = nullptr, *h1b = nullptr, *h2b = nullptr, *zb = nullptr;
    float *h0 = nullptr, *a1 = nullptr, *a2 = nullptr, *y = nullptr;
    float *dy = nullptr, *dz = nullptr, *da2 = nullptr, *da1 = nullptr, *dh0 = nullptr;
    bf16 *dyb = nullptr, *dzb = nullptr, *da2b = nullptr, *da1b = nullptr;
    // transposes [features][batch]: the operands of the weights' gradients
    bf16 *xt = nullptr, *h0t = nullptr, *h1t = nullptr, *h2t = nullptr, *zt = nullptr;
    bf16 *dyt = nullptr, *dzt = nullptr, *da2t = nullptr, *da1t = nullptr, *dh0t = nullptr;
    float *scale = nullptr, *den = nullptr, *row_err = nullptr, *err_part = nullptr;
    int *err = nullptr;
    std::vector<void *> allocs;
};

namespace {

int mlp_alloc(gd_mlp *h, void **p, size_t bytes)
{
    cudaError_t e = cudaMalloc(p, bytes);
    if (e != cudaSuccess) return gd::cuda_error(e, "surrogate allocation");
    h->allocs.push_back(*p);
    return GD_OK;
}

template <typename T>
int alloc_n(gd_mlp *h, T **p, size_t n)
{
    return mlp_alloc(h, reinterpret_cast<void **>(p), n * sizeof(T));
}

void layer_dims(const gd_mlp *h, int k, int *out, int *in)
{
    const int dims[5][2] = {{256, h->n_in_p}, {512, 256}, {512, 512}, {256, 512}, {h->n_out_p, 256}};
    *out = dims[k][0];
    *in = dims[k][1];
}

int refresh_bf16(gd_mlp *h, cudaStream_t st)
{
    for (int k = 0; k < 5; k++) {
        gd_mlp::Layer &l = h->L[k];
        const int64_t n = (int64_t)l.out * l.in;
        gd::to_bf16_kernel<<<(int)std::min<int64_t>((n + 255) / 256, 4096), 256, 0, st>>>(l.w, l.out, l.in, l.in, l.in,
                                                                                           l.wb, l.in);
        GD_CUDA(cudaGetLastError());
        if (k > 0) {
            int rc = gd::transpose(l.wb, l.out, l.in, l.in, l.wt, l.out, st);
            if (rc) return rc;
        }
    }
    return GD_OK;
}

gd::GemmArgs args(int M, int N, int K, int *err)
{
    gd::GemmArgs a{};
    a.M = M;
    a.N = N;
    a.K = K;
    a.err = err;
    return a;
}

// network input: per-cell scales and the BF16 cell-major copy of x (with train its
// transpose too), and, when d [n_out][ldd] is set, the loss denominators of its
// sums of squares in h->den
int load_input(gd_mlp *h, const float *x, int ldx, int B, bool train, const float *d, int ldd, cudaStream_t st)
{
    const bool loss = d != nullptr;
    if (h->flags & GD_MLP_LOSS_MSE) d = nullptr;
    int rc = gd::launch_ordered(gd::cell_sums_kernel, dim3((B + 31) / 32, d ? 2 : 1), st, x, h->n_in, ldx,
                                (int)(h->flags & GD_MLP_SCALE_INPUT), h->scale, d, h->n_out, ldd, h->den, B);
    if (rc) return rc;
    const int mse = (h->flags & GD_MLP_LOSS_MSE) ? 1 : 0;
    const gd::DenArgs den{loss ? h->den : nullptr, (h->flags & GD_MLP_SCALE_OUTPUT) ? 1 : 0, 1.f / h->out_gain, mse,
                          h->n_out, !mse && (h->flags & GD_MLP_LOSS_BATCH)};
    dim3 blk(32, 8), grd((B + 31) / 32, h->n_in_p / 64 + (loss ? 1 : 0));
    auto gather = train ? gd::gather_in_kernel<true> : gd::gather_in_kernel<false>;
    gather<<<grd, blk, 0, st>>>(x, h->n_in, ldx, B, h->scale, h->in_gain, h->xb, h->xt, h->n_in_p, den);
    GD_CUDA(cudaGetLastError());
    return GD_OK;
}

// forward on rows [0, B) of h->xb; the output times its scales into out
// [n_out][ld_out], or, when out is null, unscaled into h->y ([B][n_out_p]); with
// train also the layers' transposes
int forward(gd_mlp *h, int B, float *out, int ld_out, bool train, cudaStream_t st)
{
    using namespace gd;
    int rc;
    auto transposed = [&](GemmArgs &a, bf16 *t) {
        if (train) a.c16t = t;
        a.ldt = B;
    };
    GemmArgs a = args(B, 256, h->n_in_p, h->err);
    a.stall_polls = h->stall_next;  // a pending time-out injection fires here, once
    h->stall_next = 0;
    a.bias = h->L[0].b;
    a.c32 = h->h0;
    a.ld32 = 256;
    a.c16 = h->h0b;
    a.ld16 = 256;
    transposed(a, h->h0t);
    if ((rc = gemm_nt(EPI_NONE, h->xb, h->L[0].wb, a, st))) return rc;
    a = args(B, 512, 256, h->err);
    a.bias = h->L[1].b;
    a.pre_out = train ? h->a1 : nullptr;
    a.ld32 = 512;
    a.c16 = h->h1b;
    a.ld16 = 512;
    transposed(a, h->h1t);
    if ((rc = gemm_nt(EPI_GELU, h->h0b, h->L[1].wb, a, st))) return rc;
    a = args(B, 512, 512, h->err);
    a.bias = h->L[2].b;
    a.pre_out = train ? h->a2 : nullptr;
    a.ld32 = 512;
    a.c16 = h->h2b;
    a.ld16 = 512;
    transposed(a, h->h2t);
    if ((rc = gemm_nt(EPI_GELU, h->h1b, h->L[2].wb, a, st))) return rc;
    a = args(B, 256, 512, h->err);
    a.bias = h->L[3].b;
    a.add = h->h0;
    a.ld32 = 256;
    a.c16 = h->zb;
    a.ld16 = 256;
    transposed(a, h->zt);
    if ((rc = gemm_nt(EPI_NONE, h->h2b, h->L[3].wb, a, st))) return rc;
    a = args(B, h->n_out_p, 256, h->err);
    a.bias = h->L[4].b;
    if (out) {
        a.c32 = out;
        a.ld32 = ld_out;
        a.n_out = h->n_out;
        a.scale2 = (h->flags & GD_MLP_SCALE_OUTPUT) ? h->scale : nullptr;
        a.out_gain = h->out_gain;
        return gemm_nt(EPI_NODE, h->zb, h->L[4].wb, a, st);
    }
    a.c32 = h->y;
    a.ld32 = h->n_out_p;
    return gemm_nt(EPI_NONE, h->zb, h->L[4].wb, a, st);
}

// all gradients; the batch's mean loss into loss when set
int backward(gd_mlp *h, int B, float *loss, cudaStream_t st)
{
    using namespace gd;
    int rc;
    auto transposed = [&](GemmArgs &a, bf16 *t) {
        a.c16t = t;
        a.ldt = B;
    };
    // y = W4 z + b4
    GemmArgs a = args(B, 256, h->n_out_p, h->err);
    a.c32 = h->dz;
    a.ld32 = 256;
    a.c16 = h->dzb;
    a.ld16 = 256;
    transposed(a, h->dzt);
    if ((rc = gemm_nt(EPI_NONE, h->dyb, h->L[4].wt, a, st))) return rc;
    // z = W3 h2 + b3 + h0
    a = args(B, 512, 256, h->err);
    a.aux = h->a2;
    a.c32 = h->da2;
    a.ld32 = 512;
    a.c16 = h->da2b;
    a.ld16 = 512;
    transposed(a, h->da2t);
    if ((rc = gemm_nt(EPI_DGELU, h->dzb, h->L[3].wt, a, st))) return rc;
    // h2 = GELU(W2 h1 + b2)
    a = args(B, 512, 512, h->err);
    a.aux = h->a1;
    a.c32 = h->da1;
    a.ld32 = 512;
    a.c16 = h->da1b;
    a.ld16 = 512;
    transposed(a, h->da1t);
    if ((rc = gemm_nt(EPI_DGELU, h->da2b, h->L[2].wt, a, st))) return rc;
    // h1 = GELU(W1 h0 + b1); dh0 also receives dz through the residual
    a = args(B, 256, 512, h->err);
    a.add = h->dz;
    a.c32 = h->dh0;
    a.ld32 = 256;
    transposed(a, h->dh0t);
    if ((rc = gemm_nt(EPI_NONE, h->da1b, h->L[1].wt, a, st))) return rc;
    // all weights' gradients in one launch: dW[o][i] = sum_b dY[b][o] X[b][i], A =
    // dY^T [out][B], B = X^T [in][B]
    const bf16 *dYt[5] = {h->dh0t, h->da1t, h->da2t, h->dzt, h->dyt};
    const bf16 *Xt[5] = {h->xt, h->h0t, h->h1t, h->h2t, h->zt};
    const float *dY[5] = {h->dh0, h->da1, h->da2, h->dz, h->dy};
    Product pr[5];
    ColSums cs;
    for (int k = 0; k < 5; k++) {
        const gd_mlp::Layer &l = h->L[k];
        pr[k] = Product{dYt[k], Xt[k], args(l.out, l.in, B, h->err)};
        pr[k].a.c32 = l.gw;
        pr[k].a.ld32 = l.in;
        cs.d[k] = dY[k];
        cs.out[k] = l.gb;
        cs.n[k] = l.out;
        cs.end[k] = (k > 0 ? cs.end[k - 1] : 0) + (l.out + 31) / 32;
    }
    if ((rc = gemm_nt<5>(EPI_NONE, pr, st))) return rc;
    const MeanLoss ml{h->err_part, h->n_out_p / 64, h->den, h->row_err, loss};
    return launch_ordered(colsum_kernel, dim3(cs.end[4] + (loss ? 1 : 0)), st, cs, B, ml);
}

// output gradient for targets t (the denominators in h->den) and the loss's parts;
// without train the cells' losses
int loss_grad(gd_mlp *h, const float *t, int ldt, int B, bool train, cudaStream_t st)
{
    const int pw = (h->flags & GD_MLP_SCALE_OUTPUT) ? 1 : 0;
    const float inv_gain = 1.f / h->out_gain;
    dim3 blk(32, 8), grd((B + 31) / 32, h->n_out_p / 64);
    gd::loss_grad_kernel<<<grd, blk, 0, st>>>(h->y, t, ldt, h->n_out, h->n_out_p, B, h->scale, pw, inv_gain, h->den,
                                              h->dy, h->dyb, train ? h->dyt : nullptr, h->err_part);
    if (!train)
        gd::row_err_kernel<<<(B + 1023) / 1024, 1024, 0, st>>>(h->err_part, h->n_out_p / 64, B, h->den, h->row_err);
    GD_CUDA(cudaGetLastError());
    return GD_OK;
}

int check_err(gd_mlp *h, cudaStream_t st)
{
    int flag = 0;
    GD_CUDA(cudaMemcpyAsync(&flag, h->err, sizeof(int), cudaMemcpyDeviceToHost, st));
    GD_CUDA(cudaStreamSynchronize(st));
    if (flag) {
        // clear the record so that later calls start clean
        GD_CUDA(cudaMemsetAsync(h->err, 0, sizeof(int), st));
        GD_CUDA(cudaStreamSynchronize(st));
        return gd::set_error(GD_ERR_CUDA, "surrogate GEMM: a pipeline wait timed out");
    }
    return GD_OK;
}

}  // namespace

extern "C" int gd_mlp_create(int n_in, int n_out, int batch_cap, int flags, uint64_t seed, gd_mlp **out)
{
    using namespace gd;
    if (!out) return set_error(GD_ERR_INVALID_ARG, "NULL argument");
    *out = nullptr;
    if (n_in < 1 || n_out < 1 || n_in > (1 << 16) || n_out > (1 << 16) || batch_cap < 64 || batch_cap % 64 ||
        (flags & ~(GD_MLP_SCALE_INPUT | GD_MLP_SCALE_OUTPUT | GD_MLP_LOSS_MSE | GD_MLP_LOSS_BATCH)))
        return set_error(GD_ERR_INVALID_ARG,
                         "need 1 <= n_in, n_out <= 65536, batch_cap a positive multiple of 64 and known flags");
    if ((flags & GD_MLP_SCALE_OUTPUT) && !(flags & GD_MLP_SCALE_INPUT))
        return set_error(GD_ERR_INVALID_ARG, "GD_MLP_SCALE_OUTPUT needs GD_MLP_SCALE_INPUT");
    {
        // parameters (FP32 master, gradient, two Adam moments, BF16 copy and
        // transpose) and activations, for the memory limit
        const double np = 256.0 * pad64(n_in) + 512.0 * 256 + 512.0 * 512 + 256.0 * 512 + 256.0 * pad64(n_out);
        const double acts = (double)batch_cap * (6.0 * pad64(n_in) + 14.0 * pad64(n_out) + 12000.0);
        const size_t limit = memory_limit();
        if (limit && np * 20.0 + acts > (double)limit)
            return set_error(GD_ERR_OUT_OF_MEMORY, "the surrogate network exceeds the library's memory limit");
    }
    gd_mlp *h = new gd_mlp();
    h->n_in = n_in;
    h->n_out = n_out;
    h->n_in_p = pad64(n_in);
    h->n_out_p = pad64(n_out);
    h->cap = batch_cap;
    h->flags = flags;
    cudaGetDevice(&h->device);
    int rc = GD_OK;
    // 64-bit LCG; uniform(-1/sqrt(fan_in), 1/sqrt(fan_in)) on the true inputs
    uint64_t state = seed * 6364136223846793005ull + 1442695040888963407ull;
    auto uni = [&]() {
        state = state * 6364136223846793005ull + 1442695040888963407ull;
        return (float)(((state >> 11) + 0.5) * (1.0 / 9007199254740992.0));
    };
    for (int k = 0; k < 5 && !rc; k++) {
        gd_mlp::Layer &l = h->L[k];
        layer_dims(h, k, &l.out, &l.in);
        const size_t n = (size_t)l.out * l.in;
        if (!rc) rc = alloc_n(h, &l.w, n);
        if (!rc) rc = alloc_n(h, &l.gw, n);
        if (!rc) rc = alloc_n(h, &l.mw, n);
        if (!rc) rc = alloc_n(h, &l.vw, n);
        if (!rc) rc = alloc_n(h, &l.b, l.out);
        if (!rc) rc = alloc_n(h, &l.gb, l.out);
        if (!rc) rc = alloc_n(h, &l.mb, l.out);
        if (!rc) rc = alloc_n(h, &l.vb, l.out);
        if (!rc) rc = alloc_n(h, &l.wb, n);
        if (!rc) rc = alloc_n(h, &l.wt, n);
        if (rc) break;
        const int fan_in = k == 0 ? n_in : l.in;
        const float bound = 1.f / std::sqrt((float)fan_in);
        std::vector<float> w(n, 0.f);
        for (int o = 0; o < l.out; o++)
            for (int i = 0; i < l.in; i++) {
                const bool real = (k != 0 || i < n_in) && (k != 4 || o < n_out);
                const float r = (2.f * uni() - 1.f) * bound;
                w[(size_t)o * l.in + i] = real ? r : 0.f;
            }
        if (cudaMemcpy(l.w, w.data(), n * sizeof(float), cudaMemcpyHostToDevice) != cudaSuccess ||
            cudaMemset(l.b, 0, l.out * sizeof(float)) != cudaSuccess ||
            cudaMemset(l.mw, 0, n * sizeof(float)) != cudaSuccess ||
            cudaMemset(l.vw, 0, n * sizeof(float)) != cudaSuccess ||
            cudaMemset(l.mb, 0, l.out * sizeof(float)) != cudaSuccess ||
            cudaMemset(l.vb, 0, l.out * sizeof(float)) != cudaSuccess)
            rc = set_error(GD_ERR_CUDA, "surrogate weight upload");
    }
    const size_t c = h->cap;
    if (!rc) rc = alloc_n(h, &h->xb, c * h->n_in_p);
    if (!rc) rc = alloc_n(h, &h->h0b, c * 256);
    if (!rc) rc = alloc_n(h, &h->h1b, c * 512);
    if (!rc) rc = alloc_n(h, &h->h2b, c * 512);
    if (!rc) rc = alloc_n(h, &h->zb, c * 256);
    if (!rc) rc = alloc_n(h, &h->h0, c * 256);
    if (!rc) rc = alloc_n(h, &h->a1, c * 512);
    if (!rc) rc = alloc_n(h, &h->a2, c * 512);
    if (!rc) rc = alloc_n(h, &h->y, c * h->n_out_p);
    if (!rc) rc = alloc_n(h, &h->dy, c * h->n_out_p);
    if (!rc) rc = alloc_n(h, &h->dyb, c * h->n_out_p);
    if (!rc) rc = alloc_n(h, &h->dz, c * 256);
    if (!rc) rc = alloc_n(h, &h->dzb, c * 256);
    if (!rc) rc = alloc_n(h, &h->da2, c * 512);
    if (!rc) rc = alloc_n(h, &h->da2b, c * 512);
    if (!rc) rc = alloc_n(h, &h->da1, c * 512);
    if (!rc) rc = alloc_n(h, &h->da1b, c * 512);
    if (!rc) rc = alloc_n(h, &h->dh0, c * 256);
    if (!rc) rc = alloc_n(h, &h->xt, c * h->n_in_p);
    if (!rc) rc = alloc_n(h, &h->h0t, c * 256);
    if (!rc) rc = alloc_n(h, &h->h1t, c * 512);
    if (!rc) rc = alloc_n(h, &h->h2t, c * 512);
    if (!rc) rc = alloc_n(h, &h->zt, c * 256);
    if (!rc) rc = alloc_n(h, &h->dyt, c * h->n_out_p);
    if (!rc) rc = alloc_n(h, &h->dzt, c * 256);
    if (!rc) rc = alloc_n(h, &h->da2t, c * 512);
    if (!rc) rc = alloc_n(h, &h->da1t, c * 512);
    if (!rc) rc = alloc_n(h, &h->dh0t, c * 256);
    if (!rc) rc = alloc_n(h, &h->err_part, c * (h->n_out_p / 64));
    if (!rc) rc = alloc_n(h, &h->scale, c);
    if (!rc) rc = alloc_n(h, &h->den, c);
    if (!rc) rc = alloc_n(h, &h->row_err, c);
    if (!rc) rc = alloc_n(h, &h->err, 1);
    if (!rc && cudaMemset(h->err, 0, sizeof(int)) != cudaSuccess) rc = set_error(GD_ERR_CUDA, "memset");
    if (!rc) rc = refresh_bf16(h, nullptr);
    if (!rc && cudaDeviceSynchronize() != cudaSuccess) rc = set_error(GD_ERR_CUDA, "surrogate set-up");
    if (rc) {
        for (void *p : h->allocs) cudaFree(p);
        delete h;
        return rc;
    }
    *out = h;
    return GD_OK;
}

extern "C" int gd_mlp_set_io_scale(gd_mlp *h, float in_gain, float out_gain)
{
    if (!h) return gd::set_error(GD_ERR_INVALID_ARG, "NULL argument");
    if (!(in_gain > 0.f) || !(out_gain > 0.f) || !std::isfinite(in_gain) || !std::isfinite(out_gain))
        return gd::set_error(GD_ERR_INVALID_ARG, "input and output gains must be finite and > 0");
    h->in_gain = in_gain;
    h->out_gain = out_gain;
    return GD_OK;
}

extern "C" int gd_mlp_destroy(gd_mlp *h)
{
    if (!h) return GD_OK;
    gd::DeviceGuard ds(h->device);
    for (void *p : h->allocs) cudaFree(p);
    delete h;
    return GD_OK;
}

extern "C" int gd_mlp_info(const gd_mlp *h, gd_mlp_info_t *info)
{
    if (!h || !info) return gd::set_error(GD_ERR_INVALID_ARG, "NULL argument");
    info->n_in = h->n_in;
    info->n_out = h->n_out;
    info->n_in_padded = h->n_in_p;
    info->n_out_padded = h->n_out_p;
    info->batch_cap = h->cap;
    info->flags = h->flags;
    info->steps = h->step;
    info->in_gain = h->in_gain;
    info->out_gain = h->out_gain;
    int64_t s = 0;
    double fl = 0.0;
    for (int k = 0; k < 5; k++) {
        s += (int64_t)h->L[k].out * h->L[k].in + h->L[k].out;
        fl += 2.0 * h->L[k].out * h->L[k].in;
    }
    info->num_params = s;
    info->forward_flop_per_cell = fl;
    return GD_OK;
}

extern "C" int gd_mlp_forward(gd_mlp *h, const float *x, int ldx, int batch, float *y, int ldy, gd_stream stream)
{
    using namespace gd;
    if (!h || !x || !y || batch < 1 || batch > h->cap || ldx < batch || ldy < batch)
        return set_error(GD_ERR_INVALID_ARG, "bad surrogate forward arguments (1 <= batch <= cap, ld >= batch)");
    gd::DeviceGuard ds(h->device);
    cudaStream_t st = (cudaStream_t)stream;
    int rc = load_input(h, x, ldx, batch, false, nullptr, 0, st);
    if (!rc) rc = forward(h, batch, y, ldy, false, st);
    return rc;
}

extern "C" int gd_mlp_train_step(gd_mlp *h, const float *x, int ldx, const float *t, int ldt, const float *tden,
                                 int ldd, int batch, float lr, float weight_decay, float *loss, gd_stream stream)
{
    using namespace gd;
    if (!h || !x || !t || batch < 64 || batch > h->cap || batch % 64 || ldx < batch || ldt < batch ||
        (tden && ldd < batch))
        return set_error(GD_ERR_INVALID_ARG, "bad surrogate training arguments (batch a multiple of 64, <= cap)");
    gd::DeviceGuard ds(h->device);
    cudaStream_t st = (cudaStream_t)stream;
    int rc = load_input(h, x, ldx, batch, true, tden ? tden : t, tden ? ldd : ldt, st);
    if (!rc) rc = forward(h, batch, nullptr, 0, true, st);
    if (!rc) rc = loss_grad(h, t, ldt, batch, true, st);
    if (rc) return rc;
    if ((rc = backward(h, batch, loss, st))) return rc;
    h->step++;
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    const float c1 = 1.f - (float)std::pow(0.9, (double)h->step), c2 = 1.f - (float)std::pow(0.999, (double)h->step);
    AdamSet ad;
    ad.lr = lr;
    ad.b1 = b1;
    ad.b2 = b2;
    ad.c1 = c1;
    ad.c2 = c2;
    ad.eps = eps;
    ad.wd = weight_decay;
    int blocks = 0;
    for (int k = 0; k < 5; k++) {
        gd_mlp::Layer &l = h->L[k];
        const int wend = blocks + l.out / 32 * (l.in / 32);
        blocks = wend + (l.out + 1023) / 1024;
        ad.l[k] = {l.w, l.b, l.mw, l.vw, l.mb, l.vb, l.gw, l.gb, l.wb, k > 0 ? l.wt : nullptr, l.out, l.in, wend, blocks};
    }
    adam_kernel<<<blocks, dim3(32, 8), 0, st>>>(ad);
    GD_CUDA(cudaGetLastError());
    return GD_OK;
}

extern "C" int gd_mlp_loss(gd_mlp *h, const float *x, int ldx, const float *t, int ldt, const float *tden, int ldd,
                           int batch, float *row_loss, gd_stream stream)
{
    using namespace gd;
    if (!h || !x || !t || !row_loss || batch < 1 || batch > h->cap || ldx < batch || ldt < batch ||
        (tden && ldd < batch))
        return set_error(GD_ERR_INVALID_ARG, "bad surrogate loss arguments");
    gd::DeviceGuard ds(h->device);
    cudaStream_t st = (cudaStream_t)stream;
    int rc = load_input(h, x, ldx, batch, false, tden ? tden : t, tden ? ldd : ldt, st);
    if (!rc) rc = forward(h, batch, nullptr, 0, false, st);
    if (!rc) rc = loss_grad(h, t, ldt, batch, false, st);
    if (rc) return rc;
    GD_CUDA(cudaMemcpyAsync(row_loss, h->row_err, (size_t)batch * sizeof(float), cudaMemcpyDeviceToDevice, st));
    return GD_OK;
}

extern "C" int gd_mlp_check(gd_mlp *h, gd_stream stream)
{
    if (!h) return gd::set_error(GD_ERR_INVALID_ARG, "NULL argument");
    gd::DeviceGuard ds(h->device);
    return check_err(h, (cudaStream_t)stream);
}

// FP32 parameter block: for each layer k = 0..4, W_k [out][in] then b_k [out],
// with n_in and n_out padded to multiples of 64 (padding entries are zero).
static int copy_params(gd_mlp *h, float *host, bool to_host, bool grads)
{
    gd::DeviceGuard ds(h->device);
    size_t off = 0;
    for (int k = 0; k < 5; k++) {
        gd_mlp::Layer &l = h->L[k];
        const size_t nw = (size_t)l.out * l.in;
        float *w = grads ? l.gw : l.w, *b = grads ? l.gb : l.b;
        cudaError_t e = to_host ? cudaMemcpy(host + off, w, nw * 4, cudaMemcpyDeviceToHost)
                                : cudaMemcpy(w, host + off, nw * 4, cudaMemcpyHostToDevice);
        off += nw;
        if (e == cudaSuccess)
            e = to_host ? cudaMemcpy(host + off, b, l.out * 4, cudaMemcpyDeviceToHost)
                        : cudaMemcpy(b, host + off, l.out * 4, cudaMemcpyHostToDevice);
        off += l.out;
        if (e != cudaSuccess) return gd::cuda_error(e, "surrogate parameter copy");
    }
    return GD_OK;
}

extern "C" int gd_mlp_get_params(gd_mlp *h, float *host)
{
    if (!h || !host) return gd::set_error(GD_ERR_INVALID_ARG, "NULL argument");
    return copy_params(h, host, true, false);
}

extern "C" int gd_mlp_set_params(gd_mlp *h, const float *host)
{
    if (!h || !host) return gd::set_error(GD_ERR_INVALID_ARG, "NULL argument");
    int rc = copy_params(h, const_cast<float *>(host), false, false);
    if (rc) return rc;
    gd::DeviceGuard ds(h->device);
    if ((rc = refresh_bf16(h, nullptr))) return rc;
    if (cudaDeviceSynchronize() != cudaSuccess) return gd::set_error(GD_ERR_CUDA, "surrogate parameter refresh");
    return GD_OK;
}

extern "C" int gd_mlp_get_grads(gd_mlp *h, float *host)
{
    if (!h || !host) return gd::set_error(GD_ERR_INVALID_ARG, "NULL argument");
    return copy_params(h, host, true, true);
}

extern "C" int gd_mlp_inject_timeout(gd_mlp *h, int polls)
{
    using namespace gd;
    if (!h || polls < 1 || polls > (1 << 20))
        return set_error(GD_ERR_INVALID_ARG, "gd_mlp_inject_timeout: need a network and 1 <= polls <= 2^20");
    h->stall_next = polls;
    return GD_OK;
}

extern "C" int gd_mlp_inject_late_timeout(gd_mlp *h, int polls)
{
    const int rc = gd_mlp_inject_timeout(h, polls);
    if (!rc) h->stall_next = -polls;
    return rc;
}
