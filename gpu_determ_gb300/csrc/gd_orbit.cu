// gd_orbit.cu -- FP32 gain, all eight reflections of a pair sum at once (sm_103a).
//
// Same sums as gd_gain.cu, in the pair-product form (collision_integral.cu:75-188):
// for every pair sum s the products P_s[n], their contraction C_s[m] with one
// weight row per distinct |g|, and C_s[m] added to the outputs (s +- g)/2.
// What differs is what one warp instruction covers and what is left out:
//
//  - The lattice is symmetric under the reflections x_a -> n_a - 1 - x_a, which
//    leave the weights unchanged.  The nodes are numbered row = 8 o + e (orbit o,
//    bit a of e set in the upper half of axis a), so the reflection r maps row t
//    to t ^ r.  One table entry, written for the pair sum D in the low octant,
//    serves all its reflections: a warp's lanes are (r, cell), lane addresses
//    are (entry ^ r), and each access of shared memory or of the packed f is one
//    contiguous row of 8 reflections x CPT cells.
//  - Products whose nodes lie outside the sphere, groups without a target in
//    it and weights of absent products are not in the tables (20^3, R = 4.8:
//    3.0e6 products, 2.4e6 group rows and 4.1e7 weight terms per cell; the class
//    boxes hold 9.3e6, 3.9e6 and 1.4e8).
//  - The outputs stay in registers for a whole part of the walk: a warp
//    owns groups of four neighbouring orbits and reads each C row once per
//    target.  No output
//    is read back or written in between, and no two warps share one, so every
//    sum has a fixed order and results are bitwise reproducible.
//
// The walk is cut into parts of about equal work, the same for every batch, and the
// parts' sums are added in a fixed order: a cell's gain has the same bits alone and
// in any batch.  A CTA takes one tile of CPT cells and one part.  f of the tile,
// the P rows and the C rows of a step sit in shared memory.  A step is as many D
// as fit these rows, or a part of one D's offsets (by shell |n|, its C rows then
// accumulate over the parts).  Contraction works on blocks of four rows of
// neighbouring |g|, whose shells overlap: one P row is read for four rows (1.2
// times the terms, a third of the shared-memory reads).  What a warp has to do
// is one linear stream of 512-byte chunks (products, contraction blocks,
// targets, step by step), copied ahead into a ring of shared memory by bulk
// copies, so that no table read waits for L2 or takes load slots.  The tables
// hold shared-memory offsets ready for use: an access costs one logic operation
// and the load.
//
// Bound: shared-memory wavefronts of the three phases (all read one row per
// operation, the outputs' phase at the rate of the load unit) for 60 % of the
// time, the rest the warps' own control flow, some 400 instructions per warp and
// step.  It replaces gain_pair_kernel (gd_gain.cu) on every lattice whose rows
// fit: 12^3 (R = 4.8), 1501 cells 20.3 -> 1.40 ms; 16^3 (whole box), 256 cells
// 22.6 -> 3.83 ms; 20^3 (R = 4.8), one cell 10.5 -> 0.18 ms, 4096 cells 70.6 ms
// (as many parts as the batch needs to fill the chip: 1.28, 3.79, 0.18 and 67.2 ms,
// but other bits in other batches);
// its error against FP64 is a third to a half as large (relative L2 of the gain 6.0e-8
// against 1.8e-7 at 20^3, 6.3e-8 against 1.27e-7 in the 16^3 box: sums of the targets
// of a step, then of steps, then of parts).  Measured and not better: 8, 12, 20 or 24 warps; groups of eight
// slots with one target a round (73.4 ms at 20^3); chunk-free dense streams (78 ms:
// a check per record costs more than the padding).
#include "gd_internal.h"
#include "gd_tc.cuh"
#include "gd_workers.h"

#include <algorithm>
#include <array>
#include <cmath>
#include <cstring>
#include <memory>

namespace gd {
namespace {

constexpr int kOWarps = 16;
constexpr int kOThreads = 32 * kOWarps;
constexpr int kORows = 4;                        // rows of a contraction block
constexpr uint32_t kOChunk = 512;                // bytes of a stream chunk
constexpr uint32_t kORing = 4 * kOChunk;         // a warp's ring: three chunks in flight
constexpr uint32_t kOBars = kOWarps * kORing;    // offset of the rings' barriers
constexpr uint32_t kOF = kOBars + 1024;          // offset of f
constexpr uint32_t kOQuad = 80;                  // bytes of a contraction quad
constexpr int kOMatrixNodes = 512;               // BF16x3 matrices stay below this (orbit_serves)
constexpr size_t kOScratch = (size_t)2 << 30;    // scratch of a launch: larger batches run in slices of cells
constexpr int kOSlots = 4;                       // output slots gathered side by side
constexpr int kOParts = 152;                     // parts of the walk, each summed by itself (orbit_build)
constexpr int kOGroup = 16;                      // rounds (two targets per slot, 32 bytes) of a group in a step: at most a chunk

struct OrbitArgs {
    const float *ft;              // [tile][row][CPT]
    const unsigned char *stream;  // per warp: the chunks of every step
    const int *start;             // [part][warp] position of its stream, in 16-byte units
    const int *bounds;            // [parts + 1] step bounds
    const int *row_node;
    float *part;                  // [part][tile][row][CPT], or null (one part): write gain
    float *gain;
    const float2 *scale;          // [cells_pad] power-of-two factors of f and back
    int *err;                     // set to 1 when a copy is not seen to land
    int norb, ns, ncells, ld;
    uint32_t p_at, zero_at;       // shared-memory offsets of the P rows and of the zero C row
    // failure-detection test hook: > 0 makes every warp wait this many polls, its
    // first copies in flight, on a barrier that nothing arrives at
    int stall_polls;
};

// Two FP32 operations per instruction where a lane holds two cells.
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c)
{
    float2 d;
    asm("{\n\t.reg .b64 x, y, z, w;\n\t"
        "mov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmov.b64 z, {%6, %7};\n\t"
        "fma.rn.f32x2 w, x, y, z;\n\tmov.b64 {%0, %1}, w;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return d;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b)
{
    float2 d;
    asm("{\n\t.reg .b64 x, y, w;\n\t"
        "mov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\t"
        "add.rn.f32x2 w, x, y;\n\tmov.b64 {%0, %1}, w;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}

// A gain of f 2^-k back to that of f (two factors: 4^k may exceed FP32's range).
__device__ __forceinline__ float unscale(float v, float s) { return __fmul_rn(__fmul_rn(v, s), s); }

template <int CPT>
struct Vec;
template <>
struct Vec<8> {
    using T = float2;
    static __device__ __forceinline__ T zero() { return make_float2(0.f, 0.f); }
    static __device__ __forceinline__ T mac(T a, T b, T c) { return fma2(a, b, c); }
    static __device__ __forceinline__ T mac(float w, T b, T c)
    {
        return make_float2(__fmaf_rn(w, b.x, c.x), __fmaf_rn(w, b.y, c.y));
    }
    static __device__ __forceinline__ T add(T a, T b) { return add2(a, b); }
    static __device__ __forceinline__ T mul(T a, T b) { return make_float2(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y)); }
};
template <>
struct Vec<4> {
    using T = float;
    static __device__ __forceinline__ T zero() { return 0.f; }
    static __device__ __forceinline__ T mac(T a, T b, T c) { return __fmaf_rn(a, b, c); }
    static __device__ __forceinline__ T add(T a, T b) { return __fadd_rn(a, b); }
    static __device__ __forceinline__ T mul(T a, T b) { return __fmul_rn(a, b); }
};

template <typename T>
__device__ __forceinline__ T lds(uint32_t addr);
template <>
__device__ __forceinline__ float lds<float>(uint32_t addr)
{
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr));
    return v;
}
template <>
__device__ __forceinline__ float2 lds<float2>(uint32_t addr)
{
    float2 v;
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr));
    return v;
}
template <>
__device__ __forceinline__ float4 lds<float4>(uint32_t addr)
{
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
    return v;
}
template <>
__device__ __forceinline__ uint4 lds<uint4>(uint32_t addr)
{
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}
template <>
__device__ __forceinline__ uint32_t lds<uint32_t>(uint32_t addr)
{
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ void sts(uint32_t addr, float v) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory"); }
__device__ __forceinline__ void sts(uint32_t addr, float2 v)
{
    asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(addr), "f"(v.x), "f"(v.y) : "memory");
}

template <int CPT, int NSLOT>
__global__ void __launch_bounds__(kOThreads, 1) orbit_gain_kernel(const __grid_constant__ OrbitArgs a)
{
    using V = Vec<CPT>;
    using T = typename V::T;
    constexpr uint32_t kRow = 32 * sizeof(T);  // bytes of a P or C row
    // rings, their barriers, f (and eight zero rows), P and C
    extern __shared__ __align__(1024) unsigned char smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t lb = lane * (uint32_t)sizeof(T);  // r * (CPT cells) + cell, in bytes
    const int r = lane >> 2;
    const uint32_t sm = (uint32_t)__cvta_generic_to_shared(smem), slb = sm + lb;

    // f of the tile, and eight zero rows, on their way before anything else
    const float *ft = a.ft + (size_t)blockIdx.x * a.ns * CPT;
    for (int i = threadIdx.x; i < (a.ns + 8) * CPT / 4; i += kOThreads) {
        if (i < a.ns * CPT / 4)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sm + kOF + i * 16), "l"(ft + 4 * i) : "memory");
        else
            *reinterpret_cast<float4 *>(smem + kOF + i * 16) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    const int s0 = a.bounds[blockIdx.y], s1 = a.bounds[blockIdx.y + 1];
    const uint32_t first = (uint32_t)__ldg(a.start + blockIdx.y * kOWarps + warp) * 16u;
    if (s0 < s1) {
        const uint32_t ring = sm + warp * kORing, bar = sm + kOBars + warp * 32;
        if (lane == 0) {
            for (int k = 0; k < 4; k++) tc::mbar_init(bar + 8 * k, 1);
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        __syncwarp();
        // the ring: chunk c sits at (c % 4) chunks
        const unsigned char *src = a.stream + (first & ~(kOChunk - 1));
        uint32_t issued = 0, taken = 0;
        uint32_t at = 0, room = 0;  // the stream's position, and the bytes to its chunk's end
        bool ok = true;
        auto fetch = [&]() {
            if (lane == 0) {
                const uint32_t b = bar + 8 * (issued & 3);
                tc::mbar_expect_tx(b, kOChunk);
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                                 ring + (issued & 3) * kOChunk),
                             "l"(src), "r"(kOChunk), "r"(b)
                             : "memory");
            }
            src += kOChunk;
            issued++;
        };
        // `bytes` of the stream at `at`, moving to the next chunk when this one has
        // less left: it has landed, the one before it is done with and its place
        // takes the third chunk ahead
        auto need = [&](uint32_t bytes) -> bool {
            if (room < bytes) {
                __syncwarp();
                fetch();
                ok = __all_sync(0xffffffffu, tc::mbar_wait(bar + 8 * (taken & 3), (taken >> 2) & 1, a.err)) && ok;
                at = ring + (taken & 3) * kOChunk;
                taken++;
                room = kOChunk;
            }
            return ok;
        };
        auto skip = [&](uint32_t bytes) {
            at += bytes;
            room -= bytes;
        };
        for (int k = 0; k < 3; k++) fetch();
        if (a.stall_polls > 0) {
            const uint32_t never = sm + kOBars + 32 * kOWarps + 8 * warp;
            if (lane == 0) {
                tc::mbar_init(never, 1);
                tc::mbar_wait_limit(never, 0u, a.err, (uint32_t)a.stall_polls);
            }
            ok = false;
        }
        if (warp == 0) sts(slb + a.zero_at, V::zero());  // padding targets read this row
        need(1);
        skip(first & (kOChunk - 1));
        T acc[NSLOT];
#pragma unroll
        for (int j = 0; j < NSLOT; j++) acc[j] = V::zero();
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();

        // C rows of a step into this warp's outputs: a count of rounds per group of
        // four slots, then the rounds: two offsets (of row and octant, the lane's
        // own by exclusive or) for each of the four, so that eight independent
        // loads are in flight
        auto gather = [&]() {
            constexpr uint32_t kCounts = (NSLOT / kOSlots + 15) & ~15;
            if (!need(kCounts)) return;
            uint32_t cw[(NSLOT / kOSlots + 3) / 4];
#pragma unroll
            for (int k = 0; k < (NSLOT / kOSlots + 3) / 4; k++) cw[k] = lds<uint32_t>(at + 4 * k);
            skip(kCounts);
#pragma unroll
            for (int g = 0; g < NSLOT / kOSlots; g++) {
                const int n = (cw[g / 4] >> (8 * (g & 3))) & 255;
                if (n == 0) continue;
                if (!need(32 * n)) return;
                room -= 32 * n;
                T s0 = V::zero(), s1 = V::zero(), s2 = V::zero(), s3 = V::zero();
                uint4 u = lds<uint4>(at), v = lds<uint4>(at + 16);
#pragma unroll 1
                for (int q = 0; q < n; q++) {
                    const T a0 = lds<T>(sm + (u.x ^ lb)), b0 = lds<T>(sm + (u.y ^ lb)), a1 = lds<T>(sm + (u.z ^ lb)),
                            b1 = lds<T>(sm + (u.w ^ lb)), a2 = lds<T>(sm + (v.x ^ lb)), b2 = lds<T>(sm + (v.y ^ lb)),
                            a3 = lds<T>(sm + (v.z ^ lb)), b3 = lds<T>(sm + (v.w ^ lb));
                    at += q + 1 < n ? 32 : 0;
                    u = lds<uint4>(at);  // the next round's (after the last: its own again)
                    v = lds<uint4>(at + 16);
                    s0 = V::add(s0, V::add(a0, b0));
                    s1 = V::add(s1, V::add(a1, b1));
                    s2 = V::add(s2, V::add(a2, b2));
                    s3 = V::add(s3, V::add(a3, b3));
                }
                at += 32;
                acc[4 * g] = V::add(acc[4 * g], s0);
                acc[4 * g + 1] = V::add(acc[4 * g + 1], s1);
                acc[4 * g + 2] = V::add(acc[4 * g + 2], s2);
                acc[4 * g + 3] = V::add(acc[4 * g + 3], s3);
            }
        };

        bool targets = false;
        for (int st = s0; st < s1; st++) {
            if (targets) gather();
            // products: rows of four pairs, then rows of at most two; a missing pair
            // reads the zero rows; low bits of the first offset: the axes on which
            // D is its own mirror, whose reflections repeat D
            uint4 hd = make_uint4(0, 0, 0, 0);  // rows of four, rows of two, first row of two, blocks (bit 31: targets)
            if (need(16)) {
                hd = lds<uint4>(at);
                skip(16);
            }
            uint32_t prow = slb + a.p_at + warp * kRow;
            for (uint32_t left = hd.x; left > 0;) {
                if (!need(32)) break;
                const uint32_t n = min(left, room / 32);
                left -= n;
                room -= 32 * n;
#pragma unroll 1
                for (uint32_t k = 0; k < n; k++, prow += kOWarps * kRow, at += 32) {
                    const uint4 u = lds<uint4>(at), w = lds<uint4>(at + 16);
                    const uint32_t self = u.x & 7u;
                    const T x0 = lds<T>(sm + ((u.x & ~7u) ^ lb)), y0 = lds<T>(sm + (u.y ^ lb)), x1 = lds<T>(sm + (u.z ^ lb)),
                            y1 = lds<T>(sm + (u.w ^ lb)), x2 = lds<T>(sm + (w.x ^ lb)), y2 = lds<T>(sm + (w.y ^ lb)),
                            x3 = lds<T>(sm + (w.z ^ lb)), y3 = lds<T>(sm + (w.w ^ lb));
                    T p = V::add(V::mac(x0, y0, V::mul(x1, y1)), V::mac(x2, y2, V::mul(x3, y3)));
                    if (self && (self & (uint32_t)r)) p = V::zero();
                    sts(prow, p);
                }
            }
            prow = slb + a.p_at + (hd.z + warp) * kRow;
            for (uint32_t left = hd.y; ok && left > 0;) {
                if (!need(16)) break;
                const uint32_t n = min(left, room / 16);
                left -= n;
                room -= 16 * n;
#pragma unroll 1
                for (uint32_t k = 0; k < n; k += 2, prow += 2 * kOWarps * kRow, at += 32) {
                    // two rows at a time (the second past the last: not stored)
                    const uint4 u = lds<uint4>(at), w = lds<uint4>(k + 1 < n ? at + 16 : at);
                    const T x0 = lds<T>(sm + ((u.x & ~7u) ^ lb)), y0 = lds<T>(sm + (u.y ^ lb)), x1 = lds<T>(sm + (u.z ^ lb)),
                            y1 = lds<T>(sm + (u.w ^ lb)), x2 = lds<T>(sm + ((w.x & ~7u) ^ lb)), y2 = lds<T>(sm + (w.y ^ lb)),
                            x3 = lds<T>(sm + (w.z ^ lb)), y3 = lds<T>(sm + (w.w ^ lb));
                    T p = V::mac(x0, y0, V::mul(x1, y1)), p2 = V::mac(x2, y2, V::mul(x3, y3));
                    if ((u.x | w.x) & 7u) {
                        if (u.x & (uint32_t)r) p = V::zero();
                        if (w.x & (uint32_t)r) p2 = V::zero();
                    }
                    sts(prow, p);
                    if (k + 1 < n) sts(prow + kOWarps * kRow, p2);
                }
                if (n & 1) {
                    at -= 16;
                    prow -= kOWarps * kRow;
                }
            }
            if (__syncthreads_or(!ok)) {
                ok = false;
                break;
            }
            // contraction: blocks {quads, C offset, 1: its sums continue those of an
            // earlier part}, each quad four entries {P offset; the four rows' weights}
            for (uint32_t b = hd.w & 0x7fffffffu; b > 0; b--) {
                if (!need(16)) break;
                const uint4 h = lds<uint4>(at);
                skip(16);
                const uint32_t cr = slb + h.y;
                T c0 = V::zero(), c1 = V::zero(), c2 = V::zero(), c3 = V::zero();
                if (h.z) {
                    c0 = lds<T>(cr);
                    c1 = lds<T>(cr + kRow);
                    c2 = lds<T>(cr + 2 * kRow);
                    c3 = lds<T>(cr + 3 * kRow);
                }
                for (uint32_t left = h.x; left > 0;) {
                    if (!need(kOQuad)) break;
                    const uint32_t n = min(left, room / kOQuad);
                    left -= n;
                    room -= kOQuad * n;
                    uint4 o = lds<uint4>(at);
#pragma unroll 1
                    for (uint32_t q = 0; q < n; q++) {
                        const float4 w0 = lds<float4>(at + 16), w1 = lds<float4>(at + 32), w2 = lds<float4>(at + 48),
                                     w3 = lds<float4>(at + 64);
                        const T p0 = lds<T>(o.x + slb), p1 = lds<T>(o.y + slb), p2 = lds<T>(o.z + slb), p3 = lds<T>(o.w + slb);
                        at += q + 1 < n ? kOQuad : 0;
                        o = lds<uint4>(at);  // the next quad's (after the last: its own again)
#define GD_MAC(wv, pv)           \
    c0 = V::mac((wv).x, pv, c0); \
    c1 = V::mac((wv).y, pv, c1); \
    c2 = V::mac((wv).z, pv, c2); \
    c3 = V::mac((wv).w, pv, c3)
                        GD_MAC(w0, p0);
                        GD_MAC(w1, p1);
                        GD_MAC(w2, p2);
                        GD_MAC(w3, p3);
#undef GD_MAC
                    }
                    at += kOQuad;
                }
                if (!ok) break;
                sts(cr, c0);
                sts(cr + kRow, c1);
                sts(cr + 2 * kRow, c2);
                sts(cr + 3 * kRow, c3);
            }
            targets = (hd.w >> 31) != 0;
            if (__syncthreads_or(!ok)) {
                ok = false;
                break;
            }
        }
        if (ok && targets) gather();
        // the copies in flight land before the CTA leaves
        for (; taken != issued; taken++) tc::mbar_wait(bar + 8 * (taken & 3), (taken >> 2) & 1, a.err);
        if (!ok) return;  // recorded in err
        // lane (r, cells): output row 8 o + r
        const int cell = blockIdx.x * CPT + (lane & 3) * (CPT / 4);
        float *part = a.part + ((size_t)blockIdx.y * gridDim.x + blockIdx.x) * (size_t)(a.ns * CPT) + (lane & 3) * (CPT / 4);
#pragma unroll
        for (int j = 0; j < NSLOT; j++) {
            const int o = (j / kOSlots * kOWarps + warp) * kOSlots + j % kOSlots;
            if (o >= a.norb) continue;
            if (a.part) {
                *reinterpret_cast<T *>(part + (8 * o + r) * CPT) = acc[j];
            } else {
                float *g = a.gain + (size_t)__ldg(a.row_node + 8 * o + r) * a.ld + cell;
                const float *v = reinterpret_cast<const float *>(&acc[j]);
#pragma unroll
                for (int q = 0; q < CPT / 4; q++)
                    if (cell + q < a.ncells) g[q] = unscale(v[q], a.scale[cell + q].y);
            }
        }
    } else {  // a part without steps (more parts than work): zero sums
        asm volatile("cp.async.wait_all;" ::: "memory");
        float *part = a.part + ((size_t)blockIdx.y * gridDim.x + blockIdx.x) * (size_t)(a.ns * CPT);
        for (int t = threadIdx.x; t < a.ns * CPT; t += kOThreads) part[t] = 0.f;
    }
}

// scale[cell] = {2^-k, 2^k} for max|f| of the cell in [2^k, 2^(k+1)) where that
// is beyond 2^+-40 (products could leave FP32's range), {1, 1} for the others,
// {1, NaN} for a cell with a non-finite f.  Block = 32 cells x 32 node strides (16 MB
// of loads in flight at 4096 cells), for few cells 4 x 256 (one cell: 10 -> 6 us).
__global__ void __launch_bounds__(1024) orbit_scale_kernel(const float *__restrict__ f, int ld, int ncells, int ns,
                                                           float2 *__restrict__ scale, int cells_pad)
{
    __shared__ unsigned red[1024];
    const int w = blockDim.x, x = threadIdx.x, y = threadIdx.y, cell = blockIdx.x * w + x;
    unsigned m = 0;  // bit patterns of |f| order like the values, infinity and NaN above all
    if (cell < ncells)
#pragma unroll 8
        for (int p = y; p < ns; p += blockDim.y) m = max(m, __float_as_uint(__ldg(f + (size_t)p * ld + cell)) & 0x7fffffffu);
    red[y * w + x] = m;
    for (int h = blockDim.y / 2; h > 0; h /= 2) {
        __syncthreads();
        if (y < h) red[y * w + x] = m = max(m, red[(y + h) * w + x]);
    }
    if (y == 0 && cell < cells_pad) {
        const int e = (int)(m >> 23);  // 0: zero or subnormal, 255: not finite
        int k = e == 0 ? -126 : min(126, e - 127);
        if (m == 0 || abs(k) <= 40) k = 0;
        scale[cell] = e == 255 ? make_float2(1.f, __int_as_float(0x7fc00000))
                               : make_float2(__int_as_float((127 - k) << 23), __int_as_float((127 + k) << 23));
    }
}

// ft[tile][row][CPT] from f[node][cell]: the packed rows the product loads
// read; cells past ncells are zero.  Block = 32 cells x 8 rows.
__global__ void orbit_pack_kernel(const float *__restrict__ f, int ld, int ncells, int ns, int cpt,
                                  const int *__restrict__ row_node, const float2 *__restrict__ scale,
                                  float *__restrict__ ft, int cells_pad)
{
    const int cell = blockIdx.x * 32 + threadIdx.x, row = blockIdx.y * 8 + threadIdx.y;
    if (row >= ns || cell >= cells_pad) return;
    float v = cell < ncells ? f[(size_t)__ldg(row_node + row) * ld + cell] : 0.f;
    v = __fmul_rn(v, scale[cell].x);
    ft[((size_t)(cell / cpt) * ns + row) * cpt + cell % cpt] = v;
}

// gain[node][cell] = sum over the parts of [part][tile][row][cpt]: each of the block's
// eight y rows adds a contiguous eighth of the parts in order, four cells of a row
// per thread, and the eight are added in order.
__global__ void __launch_bounds__(256) orbit_reduce_kernel(const float4 *__restrict__ part, int nparts, int ns, int cpt,
                                                           int ncells, int ld, const int *__restrict__ row_node,
                                                           const float2 *__restrict__ scale, float *__restrict__ gain)
{
    __shared__ float4 red[8][32];
    const int x = threadIdx.x, y = threadIdx.y, per = cpt / 4, n = ns * per;  // quads of a row, of a tile
    const int i = blockIdx.y * 32 + x, tile = blockIdx.x;
    const int k0 = nparts * y / 8, k1 = nparts * (y + 1) / 8;
    const size_t step = (size_t)gridDim.x * n;
    const float4 *p = part + (size_t)tile * n + min(i, n - 1);
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
    for (int k = k0; k < k1; k++) {
        const float4 v = __ldg(p + (size_t)k * step);
        s.x += v.x;
        s.y += v.y;
        s.z += v.z;
        s.w += v.w;
    }
    red[y][x] = s;
    __syncthreads();
    if (y != 0 || i >= n) return;
    for (int k = 1; k < 8; k++) {
        const float4 v = red[k][x];
        s.x += v.x;
        s.y += v.y;
        s.z += v.z;
        s.w += v.w;
    }
    const int cell = tile * cpt + i % per * 4;
    float *g = gain + (size_t)__ldg(row_node + i / per) * ld + cell;
    const float o[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
    for (int q = 0; q < 4; q++)
        if (cell + q < ncells) g[q] = unscale(o[q], scale[cell + q].y);
}

// One D of the low octant with anything to do.
struct DItem {
    int K = 0, nblk = 0;
    std::vector<std::array<int16_t, 9>> prod;  // by shell |n|: four pairs of rows (-1: none), their count
    uint32_t self = 0;                         // axes on which D is its own mirror
    std::vector<int> blk_n;                    // entries per block
    std::vector<uint32_t> off;                 // P row per entry, ascending within a block
    std::vector<float4> w;
    std::vector<std::pair<int, int>> targets;  // (output row 8 o + e, C row), by output row
};

template <typename T>
int upload(T **dst, const std::vector<T> &src)
{
    GD_CUDA(cudaMalloc(dst, sizeof(T) * std::max<size_t>(src.size(), 1)));
    if (!src.empty()) GD_CUDA(cudaMemcpy(*dst, src.data(), sizeof(T) * src.size(), cudaMemcpyHostToDevice));
    return GD_OK;
}

// The kernel instance of a tile width and slot count: the smallest NSLOT that
// holds them (64 registers of outputs per thread at most, of 128).
using OrbitKernel = void (*)(const OrbitArgs);
OrbitKernel orbit_kernel(int cpt, int need, int *nslot)
{
    struct Inst {
        int cpt, nslot;
        OrbitKernel k;
    };
    static const Inst inst[] = {{8, 8, orbit_gain_kernel<8, 8>},   {8, 16, orbit_gain_kernel<8, 16>},
                                {8, 24, orbit_gain_kernel<8, 24>}, {8, 32, orbit_gain_kernel<8, 32>},
                                {4, 48, orbit_gain_kernel<4, 48>}, {4, 56, orbit_gain_kernel<4, 56>},
                                {4, 64, orbit_gain_kernel<4, 64>}};
    for (const Inst &i : inst)
        if (i.cpt == cpt && i.nslot >= need) {
            *nslot = i.nslot;
            return i.k;
        }
    return nullptr;
}

}  // namespace

void orbit_free(Context &c)
{
    OrbitGain *g = c.orbit;
    if (!g) return;
    cudaFree(g->row_node);
    cudaFree(g->stream);
    cudaFree(g->start);
    cudaFree(g->bx);
    cudaFree(g->err);
    cudaFree(g->bounds);
    delete g;
    c.orbit = nullptr;
}

// Bounds in steps of the walk's parts, of about equal work.  A part costs a large
// batch some 5 us (start of its CTA, its sums stored and added) and a single cell
// waits for the longest one, so their number goes with the root of the work, up to a
// wave of CTAs.  Measured with 38, 76, 114 and 152 parts: 20^3, one cell 625, 325,
// 225, 176 us, 4096 cells 68.3, 69.2, 70.5, 71.4 ms (152 now 70.6); 16^3, one cell
// 148, 90, 70, 58 us, 1024 cells 4.11, 4.29, 4.45, 4.64 ms; 12^3, one cell 51, 38,
// 36, 31 us, 1501 cells 1.44, 1.58, 1.73, 1.75 ms.
static void orbit_parts(const OrbitGain &g, double cost, std::vector<int> &bounds)
{
    const std::vector<double> &pre = g.cost_prefix;
    const int n = (int)g.cuts.size() - 1;
    const int nparts = std::min(n, std::max(1, (int)(kOParts * std::min(1.0, std::sqrt(cost / 7e6)))));
    bounds.assign(1, 0);
    for (int k = 1, at = 0; k < nparts; k++) {
        const double want = pre[n] * k / nparts;
        int b = (int)(std::lower_bound(pre.begin(), pre.end(), want) - pre.begin());
        if (b > 0 && want - pre[b - 1] < pre[b] - want) b--;
        at = std::min(n, std::max(at, b));
        bounds.push_back(g.cuts[at]);
    }
    bounds.push_back(g.nsteps);
}

// Tables of the orbit kernel; leaves c.orbit null (the pair kernel of
// gd_gain.cu then serves the grid) when the lattice has no reflection symmetry
// or its rows do not fit a CTA's registers and shared memory.
int orbit_build(Context &c)
{
    const Dims &d = c.d;
    // rows 8 o + e; every axis has even n_a and the sphere is centred in the
    // box, so each low-octant node has its seven mirrors
    std::vector<int> row_of(d.nxyz, -1), row_node;
    int norb = 0;
    // orbits in blocks of 2 x 2 x 2: the four slots a warp gathers side by side
    // are then mostly of one block, with much the same number of targets in a D
    std::vector<int> low;
    for (int m = 0; m < d.n_pnt; m++)
        if (c.ui[m] < d.hx && c.vi[m] < d.hy && c.wi[m] < d.hz) low.push_back(m);
    auto block_key = [&](int m) {
        const int x = c.ui[m], y = c.vi[m], z = c.wi[m];
        return (((x >> 1) * 32 + (y >> 1)) * 32 + (z >> 1)) * 8 + (x & 1) * 4 + (y & 1) * 2 + (z & 1);
    };
    std::stable_sort(low.begin(), low.end(), [&](int p, int q) { return block_key(p) < block_key(q); });
    for (int m : low) {
        for (int e = 0; e < 8; e++) {
            const int x = e & 1 ? d.nx - 1 - c.ui[m] : c.ui[m], y = e & 2 ? d.ny - 1 - c.vi[m] : c.vi[m],
                      z = e & 4 ? d.nz - 1 - c.wi[m] : c.wi[m];
            const int b = (x * d.ny + y) * d.nz + z;
            if (c.cmap[b] < 0) return GD_OK;
            row_of[b] = 8 * norb + e;
            row_node.push_back(c.cmap[b]);
        }
        norb++;
    }
    if (8 * norb != d.n_pnt) return GD_OK;

    // tile width: eight cells where their outputs, f and some rows fit, else four;
    // seen before any table is built (they grow with the seventh power of n)
    int max_smem = 0;
    GD_CUDA(cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, c.device));
    const int slots = (norb + kOWarps * kOSlots - 1) / (kOWarps * kOSlots) * kOSlots;
    auto rows_of = [&](int w) { return (max_smem - (int)kOF - (d.n_pnt + 8) * w * 4) / (32 * w) - 1; };  // P and C rows
    auto c_rows = [](int rows) { return rows * 2 / 5 / kORows * kORows; };
    int nslot = 0;
    bool fits = false;
    for (int w : {8, 4}) fits = fits || (orbit_kernel(w, slots, &nslot) && rows_of(w) - c_rows(rows_of(w)) >= 64);
    if (!fits) return GD_OK;

    // group of every g and the groups' |g|^2
    std::vector<int> gid(d.nxyz, -1);
    std::vector<double> g2(c.n_groups, 0.0);
    for (int p = 0; p < 8; p++)
        for (int k = c.class_grp_off[p]; k < c.class_grp_off[p + 1]; k++)
            for (int t = c.h_grp_mem_off[k]; t < c.h_grp_mem_off[k + 1]; t++) {
                const uint32_t m = c.h_grp_members[t];
                const int x = 2 * (int)(m & 31) + (p & 1), y = 2 * (int)((m >> 6) & 31) + ((p >> 1) & 1),
                          z = 2 * (int)((m >> 12) & 31) + (p >> 2);
                gid[(x * d.ny + y) * d.nz + z] = k;
                g2[k] = (double)(d.du * x) * (d.du * x) + (double)(d.dv * y) * (d.dv * y) +
                        (double)(d.dw * z) * (d.dw * z);
            }
    const uint32_t unit = (uint32_t)c.gain_cb * 4u;

    // every D: its products, blocks and targets (threads take D round-robin)
    std::vector<DItem> items(d.nxyz);
    auto build_items = [&](int t0, int nt) {
        std::vector<int> prow(d.nclass, -1), cls, crow(c.n_groups, -1), want;
        std::vector<std::array<float, kORows>> w4(d.nclass);
        std::vector<int> touched;
        std::vector<char> mark(d.nclass, 0);
        std::vector<double> n2;
        std::vector<int> by;
        for (int Did = t0; Did < d.nxyz; Did += nt) {
            const int D[3] = {Did / d.nyz, (Did / d.nz) % d.ny, Did % d.nz};
            DItem &it = items[Did];
            it.self = (D[0] == d.nx - 1 ? 1u : 0u) | (D[1] == d.ny - 1 ? 2u : 0u) | (D[2] == d.nz - 1 ? 4u : 0u);
            cls.clear();
            want.clear();
            n2.clear();
            for (int x2 = 0; x2 <= D[0] >> 1; x2++)
                for (int y2 = 0; y2 <= D[1] >> 1; y2++)
                    for (int z2 = 0; z2 <= D[2] >> 1; z2++) {
                        const int n[3] = {2 * x2 + (D[0] & 1), 2 * y2 + (D[1] & 1), 2 * z2 + (D[2] & 1)};
                        int at[8];
                        for (int s = 0; s < 8; s++) {
                            const int x = (s & 1 ? D[0] + n[0] : D[0] - n[0]) >> 1, y = (s & 2 ? D[1] + n[1] : D[1] - n[1]) >> 1,
                                      z = (s & 4 ? D[2] + n[2] : D[2] - n[2]) >> 1;
                            at[s] = row_of[(x * d.ny + y) * d.nz + z];
                        }
                        // the four sign patterns l / l1: (+++), (+--), (++-), (+-+)
                        static const int pat[4] = {7, 1, 3, 5};
                        std::array<int16_t, 9> pw;
                        pw.fill(-1);
                        int have = 0;
                        for (int q = 0; q < 4; q++) {
                            const int t1 = at[pat[q]], t2 = at[7 - pat[q]];
                            if (t1 < 0 || t2 < 0) continue;
                            pw[2 * have] = (int16_t)t1;
                            pw[2 * have++ + 1] = (int16_t)t2;
                        }
                        pw[8] = (int16_t)have;
                        const int k = (x2 * d.hy + y2) * d.hz + z2;
                        if (have) {
                            it.K++;
                            cls.push_back(k);
                            n2.push_back((double)(d.du * n[0]) * (d.du * n[0]) + (double)(d.dv * n[1]) * (d.dv * n[1]) +
                                         (double)(d.dw * n[2]) * (d.dw * n[2]));
                            it.prod.push_back(pw);
                        }
                        const int grp = gid[(n[0] * d.ny + n[1]) * d.nz + n[2]];
                        for (int s = 0; s < 8; s++) {
                            if ((!(s & 1) && n[0] == 0) || (!(s & 2) && n[1] == 0) || (!(s & 4) && n[2] == 0)) continue;
                            if (at[s] < 0) continue;
                            it.targets.emplace_back(at[s], grp);
                            if (crow[grp] < 0) {
                                crow[grp] = 0;
                                want.push_back(grp);
                            }
                        }
                    }
            if (it.K && !want.empty()) {
                by.resize(it.K);
                for (int k = 0; k < it.K; k++) by[k] = k;
                std::stable_sort(by.begin(), by.end(), [&](int x, int y) { return n2[x] < n2[y]; });
                std::vector<std::array<int16_t, 9>> sorted(it.K);
                for (int k = 0; k < it.K; k++) {
                    sorted[k] = it.prod[by[k]];
                    prow[cls[by[k]]] = k;
                }
                it.prod.swap(sorted);
                std::sort(want.begin(), want.end(), [&](int x, int y) { return g2[x] != g2[y] ? g2[x] < g2[y] : x < y; });
                for (size_t k = 0; k < want.size(); k++) crow[want[k]] = (int)k;
                it.nblk = ((int)want.size() + kORows - 1) / kORows;
                for (int b = 0; b < it.nblk; b++) {
                    touched.clear();
                    for (int q = 0; q < kORows && b * kORows + q < (int)want.size(); q++) {
                        const int grp = want[b * kORows + q];
                        for (int e = c.h_grp_row_off[grp]; e < c.h_grp_row_off[grp + 1]; e++) {
                            const WEntry we = c.h_grp_rows[e];
                            if (we.w == 0.0f) continue;  // row padding
                            const int pr = prow[we.off / unit];
                            if (pr < 0) continue;
                            if (!mark[pr]) {
                                mark[pr] = 1;
                                touched.push_back(pr);
                                w4[pr].fill(0.f);
                            }
                            w4[pr][q] = we.w;
                        }
                    }
                    std::sort(touched.begin(), touched.end());
                    for (int pr : touched) {
                        mark[pr] = 0;
                        it.off.push_back((uint32_t)pr);
                        it.w.push_back(make_float4(w4[pr][0], w4[pr][1], w4[pr][2], w4[pr][3]));
                    }
                    it.blk_n.push_back((int)touched.size());
                }
                for (auto &t : it.targets) t.second = crow[t.second];
                std::sort(it.targets.begin(), it.targets.end());
            }
            for (int k : cls) prow[k] = -1;
            for (int g : want) crow[g] = -1;
            if (!it.nblk) it = DItem();
        }
    };
    const int nt = std::max(1, std::min(8, (int)std::thread::hardware_concurrency()));
    if (!run_workers(nt, [&](int t) { build_items(t, nt); }))
        return set_error(GD_ERR_OUT_OF_MEMORY, "host memory for the gain tables");
    int mmax = 0;
    int64_t ktotal = 0;
    double flop = 0.0;  // of a cell: a D stands for its distinct reflections
    for (const DItem &it : items) {
        int64_t ops = (int64_t)it.targets.size();
        for (const auto &pw : it.prod) ops += 2 * pw[8] - 1;
        for (const float4 &v : it.w) ops += 2 * ((v.x != 0.f) + (v.y != 0.f) + (v.z != 0.f) + (v.w != 0.f));
        if (it.nblk) flop += (double)ops * (8 >> __builtin_popcount(it.self));
        ktotal += it.K;
        mmax = std::max(mmax, it.nblk * kORows);
    }
    if (!ktotal || !mmax) return GD_OK;

    auto orbit_of = [](int w, int j) { return (j / kOSlots * kOWarps + w) * kOSlots + j % kOSlots; };
    int cpt = 0, pcap = 0, mcap = 0;
    for (int w : {8, 4}) {
        if (!orbit_kernel(w, slots, &nslot)) continue;
        const int rows = rows_of(w);
        mcap = std::max(mmax, c_rows(rows));
        pcap = rows - mcap;
        if (pcap >= 64) {
            cpt = w;
            break;
        }
    }
    if (!cpt) return GD_OK;
    // a small lattice still gets ~96 steps, so that few cells spread over the SMs
    const int kstep = std::min(pcap, std::max(32, (int)(ktotal / 96)));
    const uint32_t row_bytes = 32u * (uint32_t)cpt;

    std::unique_ptr<OrbitGain> og(new OrbitGain);
    og->cuts.push_back(0);
    og->cost_prefix.push_back(0.0);
    double cost = 0.0;
    // shared-memory offsets, held in the tables
    const uint32_t f_row = 4u * (uint32_t)cpt, p_at = kOF + ((uint32_t)d.n_pnt + 8u) * f_row, c_at = p_at + (uint32_t)pcap * row_bytes;
    const uint32_t zero_at = c_at + (uint32_t)mcap * row_bytes, zero_f = kOF + (uint32_t)d.n_pnt * f_row;
    std::vector<std::vector<uint4>> ws(kOWarps);  // the warps' streams
    std::vector<std::vector<int>> start(kOWarps);
    auto pad_chunk = [](std::vector<uint4> &v) {
        while (v.size() % (kOChunk / 16)) v.push_back(make_uint4(0, 0, 0, 0));
    };
    auto need = [&](std::vector<uint4> &v, uint32_t bytes) {  // a record does not cross a chunk's end
        const uint32_t used = (uint32_t)(v.size() % (kOChunk / 16)) * 16u;
        if (used && kOChunk - used < bytes) pad_chunk(v);
    };
    std::vector<std::vector<uint16_t>> tl(norb);  // per orbit: C row << 3 | octant
    // a step: rows [k0, k1) of each of its D, all of their C rows; the target
    // lists in tl (empty before a D's last part)
    struct Part {
        int item, k0, k1;
    };
    auto emit = [&](const std::vector<Part> &parts, bool last) {
        struct Blk {
            int n, item, b, e0, crow, k0, kbase;
            bool cont;
        };
        std::vector<Blk> bl;
        struct Row {
            const std::array<int16_t, 9> *pairs;
            uint32_t self;
            int at;  // its P row
        };
        std::vector<Row> prod;
        int mrow = 0;
        size_t targets = 0;
        for (const auto &t : tl) targets += t.size();
        for (const Part &pt : parts) {
            const DItem &it = items[pt.item];
            const int kbase = (int)prod.size();
            for (int k = pt.k0; k < pt.k1; k++) prod.push_back(Row{&it.prod[k], it.self, 0});
            int e0 = 0;
            for (int b = 0; b < it.nblk; e0 += it.blk_n[b++]) {
                const auto lo = it.off.begin() + e0, hi = lo + it.blk_n[b];
                const int f0 = (int)(std::lower_bound(lo, hi, (uint32_t)pt.k0) - lo),
                          f1 = (int)(std::lower_bound(lo, hi, (uint32_t)pt.k1) - lo);
                // a block starts in the first part that has entries of it, or
                // in the first part when no part has (its C rows are zero)
                if (f0 == f1 && !(pt.k0 == 0 && it.blk_n[b] == 0)) continue;
                bl.push_back(Blk{f1 - f0, pt.item, b, e0 + f0, mrow + b * kORows, pt.k0, kbase, f0 > 0});
            }
            mrow += it.nblk * kORows;
        }
        // P rows: those of three or four pairs first
        int na = 0, nb = 0;
        for (Row &rw : prod)
            if ((*rw.pairs)[8] > 2) rw.at = na++;
        for (Row &rw : prod)
            if ((*rw.pairs)[8] <= 2) rw.at = na + nb++;
        std::vector<const Row *> by_row(prod.size());
        for (const Row &rw : prod) by_row[rw.at] = &rw;
        // the blocks go to the warps largest first, each to the least loaded
        std::stable_sort(bl.begin(), bl.end(), [](const Blk &x, const Blk &y) { return x.n > y.n; });
        std::vector<std::vector<const Blk *>> mine(kOWarps);
        std::vector<int> load(kOWarps, 0);
        for (const Blk &b : bl) {
            const int w = (int)(std::min_element(load.begin(), load.end()) - load.begin());
            load[w] += b.n + 6;
            mine[w].push_back(&b);
        }
        for (int w = 0; w < kOWarps; w++) {
            std::vector<uint4> &v = ws[w];
            need(v, 16);
            start[w].push_back((int)v.size());
            const size_t h = v.size();
            v.push_back(make_uint4(0, 0, 0, 0));
            uint4 hd = make_uint4(0, 0, (uint32_t)na, (uint32_t)mine[w].size());
            for (int half = 0; half < 2; half++) {
                uint32_t &count = half ? hd.y : hd.x;
                for (int k = (half ? na : 0) + w; k < (half ? na + nb : na); k += kOWarps, count++) {
                    uint32_t off[8];
                    for (int q = 0; q < 8; q++) {
                        const int t = (*by_row[k]->pairs)[q];
                        off[q] = t < 0 ? zero_f : kOF + (uint32_t)t * f_row;
                    }
                    off[0] |= by_row[k]->self;
                    need(v, half ? 16 : 32);
                    v.push_back(make_uint4(off[0], off[1], off[2], off[3]));
                    if (!half) v.push_back(make_uint4(off[4], off[5], off[6], off[7]));
                }
            }
            for (const Blk *b : mine[w]) {
                const DItem &it = items[b->item];
                const int quads = (b->n + 3) / 4;
                need(v, 16);
                v.push_back(make_uint4((uint32_t)quads, c_at + (uint32_t)b->crow * row_bytes, b->cont ? 1u : 0u, 0));
                for (int q = 0; q < quads; q++) {
                    uint32_t off[4];
                    float4 wt[4];
                    for (int z = 0; z < 4; z++) {
                        // padding repeats a row of the block with weight 0
                        const int e = 4 * q + z, e1 = std::min(e, b->n - 1);
                        off[z] = p_at + (uint32_t)prod[it.off[b->e0 + e1] - b->k0 + b->kbase].at * row_bytes;
                        wt[z] = e < b->n ? it.w[b->e0 + e] : make_float4(0.f, 0.f, 0.f, 0.f);
                    }
                    need(v, kOQuad);
                    v.push_back(make_uint4(off[0], off[1], off[2], off[3]));
                    for (int z = 0; z < 4; z++) {
                        uint4 u;
                        std::memcpy(&u, &wt[z], 16);
                        v.push_back(u);
                    }
                }
            }
            std::vector<uint8_t> counts((nslot / kOSlots + 15) / 16 * 16, 0);
            for (int j = 0; j < nslot; j++)
                if (const int o = orbit_of(w, j); o < norb)
                    counts[j / kOSlots] = std::max(counts[j / kOSlots], (uint8_t)((tl[o].size() + 1) / 2));
            if (*std::max_element(counts.begin(), counts.end())) {
                hd.w |= 0x80000000u;
                need(v, (uint32_t)counts.size());
                v.resize(v.size() + counts.size() / 16);
                std::memcpy(&v[v.size() - counts.size() / 16], counts.data(), counts.size());
                for (int g = 0; g < nslot / kOSlots; g++) {
                    need(v, 32u * counts[g]);
                    for (size_t q = 0; q < counts[g]; q++) {
                        uint32_t off[2 * kOSlots];
                        for (int z = 0; z < 2 * kOSlots; z++) {
                            const int o = orbit_of(w, g * kOSlots + z / 2);
                            const size_t t = 2 * q + z % 2;
                            off[z] = o < norb && t < tl[o].size() ? c_at + (uint32_t)(tl[o][t] >> 3) * row_bytes + (tl[o][t] & 7u) * f_row
                                                                  : zero_at;
                        }
                        v.push_back(make_uint4(off[0], off[1], off[2], off[3]));
                        v.push_back(make_uint4(off[4], off[5], off[6], off[7]));
                    }
                }
            }
            v[h] = hd;
        }
        // instructions of the busiest warp: the kernel is bound by issue
        const double most = (double)*std::max_element(load.begin(), load.end());
        cost += 400.0 + 3.1 * (double)prod.size() + 15.0 * most + 0.34 * (double)targets;
        og->nsteps++;
        if (last) {
            og->cuts.push_back(og->nsteps);
            og->cost_prefix.push_back(cost);
        }
        for (auto &t : tl) t.clear();
    };
    std::vector<Part> cur;
    int krow = 0, mrow = 0;
    auto close = [&]() {
        if (!cur.empty()) emit(cur, true);
        cur.clear();
        krow = mrow = 0;
    };
    auto add_targets = [&](const DItem &it) {
        for (const auto &t : it.targets) tl[t.first >> 3].push_back((uint16_t)((mrow + t.second) << 3 | (t.first & 7)));
        bool fits = true;
        for (const auto &t : it.targets) fits = fits && (int)tl[t.first >> 3].size() <= 2 * kOGroup;
        if (!fits)
            for (const auto &t : it.targets) tl[t.first >> 3].pop_back();
        return fits;
    };
    // D past the P rows run in parts of their own; the others, largest first,
    // are packed into steps with the largest that still fit, so that a step's
    // barriers and per-slot work are paid for as much work as its rows hold
    std::vector<int> rest;
    for (int Did = 0; Did < d.nxyz; Did++) {
        const DItem &it = items[Did];
        if (!it.nblk) continue;
        if (it.K <= kstep) {
            rest.push_back(Did);
            continue;
        }
        const int parts = (it.K + kstep - 1) / kstep;
        for (int p = 0; p < parts; p++) {
            if (p == parts - 1 && !add_targets(it)) {
                return GD_OK;
            }
            emit({Part{Did, (int)((int64_t)it.K * p / parts), (int)((int64_t)it.K * (p + 1) / parts)}}, p == parts - 1);
        }
    }
    std::stable_sort(rest.begin(), rest.end(), [&](int x, int y) { return items[x].K > items[y].K; });
    while (!rest.empty()) {
        std::vector<int> left;
        for (int Did : rest) {
            const DItem &it = items[Did];
            if (krow + it.K <= kstep && mrow + it.nblk * kORows <= mcap && add_targets(it)) {
                krow += it.K;
                mrow += it.nblk * kORows;
                cur.push_back(Part{Did, 0, it.K});
            } else {
                left.push_back(Did);
            }
        }
        if (cur.empty()) {  // a single D that does not fit
            return GD_OK;
        }
        close();
        rest.swap(left);
    }
    og->cpt = cpt;
    og->flop = flop;
    og->nslot = nslot;
    og->norb = norb;
    og->pcap = pcap;
    og->mcap = mcap;
    og->p_at = p_at;
    og->zero_at = zero_at;
    og->smem = (size_t)zero_at + row_bytes;
    // one buffer: warp after warp, each followed by the chunks that its last
    // steps copy ahead
    std::vector<uint4> stream;
    std::vector<int> st((size_t)og->nsteps * kOWarps);
    size_t total = 0;
    for (const auto &v : ws) total += v.size() + 5 * (kOChunk / 16);
    if (total * 16 >= (size_t)1 << 32) {  // positions are 32-bit
        return GD_OK;
    }
    stream.reserve(total);
    for (int w = 0; w < kOWarps; w++) {
        const int base = (int)stream.size();
        for (int k = 0; k < og->nsteps; k++) st[(size_t)k * kOWarps + w] = base + start[w][k];
        pad_chunk(ws[w]);
        stream.insert(stream.end(), ws[w].begin(), ws[w].end());
        stream.resize(stream.size() + 4 * (kOChunk / 16), make_uint4(0, 0, 0, 0));
        std::vector<uint4>().swap(ws[w]);
    }
    og->stream_bytes = stream.size() * 16;
    OrbitGain *built = c.orbit = og.release();  // freed with the context from here on
    int rc = upload(&built->row_node, row_node);
    if (!rc) rc = upload(&built->stream, stream);
    std::vector<int> bounds, first;
    orbit_parts(*built, cost, bounds);
    for (int k = 0; k + 1 < (int)bounds.size(); k++)
        for (int w = 0; w < kOWarps; w++) first.push_back(st[(size_t)std::min(bounds[k], built->nsteps - 1) * kOWarps + w]);
    built->nparts = (int)bounds.size() - 1;
    if (!rc) rc = upload(&built->bounds, bounds);
    if (!rc) rc = upload(&built->start, first);
    if (!rc) rc = upload(&built->err, std::vector<int>(1, 0));
    if (!rc) rc = orbit_loss_build(c);
    return rc;  // the caller destroys the context on failure
}

// bytes of packed f, of the parts' sums (one part writes the gain itself) and of the
// cells' scales
size_t orbit_bytes(const Context &c, int ncells)
{
    const OrbitGain &g = *c.orbit;
    return (size_t)((ncells + g.cpt - 1) / g.cpt * g.cpt) *
           (c.d.n_pnt * sizeof(float) * (g.nparts > 1 ? 1 + g.nparts : 1) + sizeof(float2));
}

// Cells of a launch for a batch of ncells in at most `room` bytes (a tile at
// least): equal slices of whole tiles.
int orbit_slice(const Context &c, int ncells, size_t room)
{
    const int cpt = c.orbit->cpt, tiles = (ncells + cpt - 1) / cpt;
    const int fit = (int)std::min<size_t>(std::max<size_t>(1, room / orbit_bytes(c, cpt)), tiles), slices = (tiles + fit - 1) / fit;
    return (tiles + slices - 1) / slices * cpt;
}

// buf holds orbit_bytes.  A cell whose f is so large or small that products would
// leave FP32's range is scaled by a power of two (orbit_scale_kernel), and a cell with
// a non-finite f gets NaN for all its outputs; other cells' bits are as without.
// (The contraction multiplies products by the zero weights of its blocks' other rows:
// an infinite one would spread.)
int launch_orbit(Context &c, const float *f, int ncells, int ld, float *gain, void *buf, cudaStream_t st)
{
    OrbitGain &g = *c.orbit;
    const Dims &d = c.d;
    const int tiles = (ncells + g.cpt - 1) / g.cpt, cells_pad = tiles * g.cpt;
    if ((int64_t)d.n_pnt * cells_pad >= ((int64_t)1 << 31))
        return set_error(GD_ERR_UNSUPPORTED, "FP32 gain: n_pnt * cells must stay below 2^31");
    float *ft = static_cast<float *>(buf);
    const int nparts = g.nparts;
    float *part = nparts > 1 ? ft + (size_t)cells_pad * d.n_pnt : nullptr;
    float2 *scale = reinterpret_cast<float2 *>(ft + (size_t)cells_pad * d.n_pnt * (nparts > 1 ? 1 + nparts : 1));
    const int sx = cells_pad <= 4 * c.sm_count ? 4 : 32;
    orbit_scale_kernel<<<(cells_pad + sx - 1) / sx, dim3(sx, 1024 / sx), 0, st>>>(f, ld, ncells, d.n_pnt, scale, cells_pad);
    GD_CUDA(cudaGetLastError());
    orbit_pack_kernel<<<dim3((cells_pad + 31) / 32, d.n_pnt / 8), dim3(32, 8), 0, st>>>(
        f, ld, ncells, d.n_pnt, g.cpt, g.row_node, scale, ft, cells_pad);
    GD_CUDA(cudaGetLastError());
    const OrbitArgs a{ft,    reinterpret_cast<const unsigned char *>(g.stream),
                      g.start, g.bounds, g.row_node, part, gain, scale, g.err, g.norb, d.n_pnt, ncells, ld,
                      g.p_at, g.zero_at, g.stall_next};
    g.stall_next = 0;  // fires once
    int nslot = 0;
    OrbitKernel kern = orbit_kernel(g.cpt, g.nslot, &nslot);
    GD_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)g.smem));
    kern<<<dim3(tiles, nparts), kOThreads, g.smem, st>>>(a);
    GD_CUDA(cudaGetLastError());
    if (part) {
        orbit_reduce_kernel<<<dim3(tiles, (d.n_pnt * (g.cpt / 4) + 31) / 32), dim3(32, 8), 0, st>>>(
            reinterpret_cast<const float4 *>(part), nparts, d.n_pnt, g.cpt, ncells, ld, g.row_node, scale, gain);
        GD_CUDA(cudaGetLastError());
    }
    return GD_OK;
}

// The tensor-core gain paths whose gain this kernel computes: it is the faster
// one, with a smaller error against FP64, on all but the smallest lattices.
// Measured against the BF16x3 matrices (ms of gain; R = 4.8, 4096 cells unless said):
// 12^3 3.82 / 5.21 (one cell 0.060 / 0.057), 16^3 (1024 cells) 4.3 / 9.2, 20^3 (1024)
// 17.8 / 50.7, 24^3 (512) 36 / 107, 10^3 (R = 5.2, 624 nodes) 2.13 / 2.58, 8^3 whole box
// (512 nodes) 1.26 / 1.37; 10^3 (480 nodes) 1.53 / 1.35 and 8^3 (208 nodes) 0.61 / 0.34,
// where the matrices stay.  Against pair_tc_kernel it wins wherever it exists: 4^3 0.06
// / 0.50, 8^3 0.61 / 5.6, 24^3 (512 cells) 36 / 168.
bool orbit_serves(const Context &c, int path)
{
    return c.orbit && (path == GD_GAIN_PAIR_TC || (path == GD_GAIN_CMATRIX_BF16X3 && c.d.n_pnt >= kOMatrixNodes));
}

int run_orbit(Context &c, const float *f, int ncells, int ld, float *gain, cudaStream_t st)
{
    // slices of cells: a cell's sums are the same in any batch
    const int slice = orbit_slice(c, ncells, kOScratch);
    int rc = ensure_scratch(c, orbit_bytes(c, slice));
    for (int at = 0; at < ncells && !rc; at += slice)
        rc = launch_orbit(c, f + at, std::min(slice, ncells - at), ld, gain + at, c.scratch.ptr, st);
    return rc;
}

// Launches of run_orbit for a batch.
int orbit_launches(const Context &c, int ncells)
{
    const int slice = orbit_slice(c, ncells, kOScratch);
    return (c.orbit->nparts > 1 ? 4 : 3) * ((ncells + slice - 1) / slice);
}

int orbit_take_timeout(Context &c, cudaStream_t st, bool *timed_out)
{
    int flag = 0;
    GD_CUDA(cudaMemcpyAsync(&flag, c.orbit->err, sizeof(int), cudaMemcpyDeviceToHost, st));
    GD_CUDA(cudaStreamSynchronize(st));
    *timed_out = flag != 0;
    if (flag) {
        GD_CUDA(cudaMemsetAsync(c.orbit->err, 0, sizeof(int), st));
        GD_CUDA(cudaStreamSynchronize(st));
    }
    return GD_OK;
}

}  // namespace gd
