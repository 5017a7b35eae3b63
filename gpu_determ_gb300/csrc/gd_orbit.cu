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
//  - The outputs stay in registers for a whole chunk of the walk: warp w owns
//    the orbits w, w + 16, ..., and reads each C row once per target.  No output
//    is read back or written in between, and no two warps share one, so every
//    sum has a fixed order and results are bitwise reproducible.
//
// A CTA takes one tile of CPT cells and one chunk of the steps.  f of the tile,
// the P rows and the C rows of a step sit in shared memory.  A step is as many D
// as fit these rows, or a part of one D's offsets (by shell |n|, its C rows then
// accumulate over the parts).  Contraction works on blocks of four rows of
// neighbouring |g|, whose shells overlap: one P row is read for four rows (1.2
// times the terms, a third of the shared-memory reads).  What a warp has to do
// is one linear stream of 512-byte chunks (products, contraction entries,
// targets, step by step), copied ahead into a ring of shared memory with
// cp.async, so that no table read waits for L2.
//
// Bound: shared-memory and L1 wavefronts (products, contraction and outputs
// all read one row per operation).  It replaces gain_pair_kernel (gd_gain.cu)
// on every lattice whose rows fit: 12^3 (R = 4.8), 1501 cells 20.3 -> 2.1 ms;
// 16^3 (whole box), 256 cells 22.6 -> 5.8 ms; 20^3 (R = 4.8), one cell 10.5 ->
// 0.30 ms; its error against FP64 is half as large (two-level sums: targets of
// a step, then steps).
#include "gd_internal.h"

#include <algorithm>
#include <array>
#include <cmath>
#include <cstring>
#include <thread>

namespace gd {
namespace {

constexpr int kOWarps = 16;
constexpr int kOThreads = 32 * kOWarps;
constexpr int kORows = 4;            // rows of a contraction block
constexpr int kOChunk = 512;         // bytes of a stream chunk: one 16-byte copy per lane
constexpr int kORing = 4 * kOChunk;  // a warp's ring
constexpr int kOQuads = 6;           // contraction quads (80 bytes) per chunk
constexpr int kOProd = 31;           // products per warp and step (one chunk, after its header)
constexpr uint32_t kNoPair = 0xffff7fffu;

struct OrbitArgs {
    const float *ft;      // [tile][row][CPT]
    const uint4 *stream;  // per warp: the chunks of every step
    const int *start;     // [step][warp] first chunk
    const int *bounds;    // [chunks + 1] step bounds
    const int *row_node;
    float *part;          // [chunk][row][cells_pad], or null: write gain
    float *gain;
    int norb, ns, cells_pad, ncells, ld;
    int pcap, mcap;
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
};
template <>
struct Vec<4> {
    using T = float;
    static __device__ __forceinline__ T zero() { return 0.f; }
    static __device__ __forceinline__ T mac(T a, T b, T c) { return __fmaf_rn(a, b, c); }
    static __device__ __forceinline__ T add(T a, T b) { return __fadd_rn(a, b); }
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
__device__ __forceinline__ uint2 lds<uint2>(uint32_t addr)
{
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr));
    return v;
}
template <>
__device__ __forceinline__ uint4 lds<uint4>(uint32_t addr)
{
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
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
    constexpr uint32_t kRow = 32 * sizeof(T);      // bytes of a P or C row
    constexpr int kShift = CPT == 8 ? 5 : 4;       // (row << 3 | e) -> bytes: e selects CPT cells
    extern __shared__ __align__(1024) unsigned char smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t lb = lane * (uint32_t)sizeof(T);  // r * (CPT cells) + cell, in bytes
    const int r = lane >> 2;
    // rings, f, P and C
    const uint32_t ring = (uint32_t)__cvta_generic_to_shared(smem) + warp * kORing;
    const uint32_t F = (uint32_t)__cvta_generic_to_shared(smem) + kOWarps * kORing;
    const uint32_t P = F + (uint32_t)a.ns * CPT * 4, C = P + (uint32_t)a.pcap * kRow;

    const int s0 = a.bounds[blockIdx.y], s1 = a.bounds[blockIdx.y + 1];
    if (s0 < s1) {
        // the ring: chunk c sits at (c % 4) chunks; three chunks are in flight
        const uint4 *src = a.stream + (size_t)__ldg(a.start + s0 * kOWarps + warp) * (kOChunk / 16) + lane;
        uint32_t head = 0;  // bytes consumed so far
        auto fetch = [&](uint32_t at) {
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(ring + (at & (kORing - 1)) + lane * 16), "l"(src)
                         : "memory");
            asm volatile("cp.async.commit_group;" ::: "memory");
            src += kOChunk / 16;
        };
        for (int k = 0; k < 3; k++) fetch(k * kOChunk);
        // the next chunk has landed: its address; the chunk before it is done with
        auto next = [&]() -> uint32_t {
            __syncwarp();
            fetch(head + 3 * kOChunk);
            asm volatile("cp.async.wait_group 3;" ::: "memory");
            __syncwarp();
            const uint32_t at = ring + (head & (kORing - 1));
            head += kOChunk;
            return at;
        };
        const float4 *ft = reinterpret_cast<const float4 *>(a.ft + (size_t)blockIdx.x * a.ns * CPT);
        for (int i = threadIdx.x; i < a.ns * CPT / 4; i += kOThreads) {
            const float4 v = __ldg(ft + i);
            asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(F + i * 16), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
                         : "memory");
        }
        if (warp == 0) sts(C + a.mcap * kRow + lb, V::zero());  // padding targets read this row
        T acc[NSLOT];
#pragma unroll
        for (int j = 0; j < NSLOT; j++) acc[j] = V::zero();
        __syncthreads();

        // C rows of a step into this warp's outputs: per slot a count of quads,
        // then 16-bit entries row << 3 | e; the list may wrap around the ring
        auto gather = [&](int nchunks) {
            if (nchunks == 0) return;
            uint32_t pos = next() - ring;
            if (nchunks == 2) {  // the second chunk too, the first still in use
                asm volatile("cp.async.wait_group 2;" ::: "memory");
                __syncwarp();
            }
            uint32_t cpos = pos;
            pos += NSLOT;
#pragma unroll
            for (int j4 = 0; j4 < NSLOT; j4 += 8, cpos += 8) {
                const uint2 cw2 = lds<uint2>(ring + cpos);
#pragma unroll
                for (int jj = 0; jj < 8; jj++) {
                    const uint32_t cw = jj < 4 ? cw2.x : cw2.y;
                    const int n = (cw >> (8 * (jj & 3))) & 255;
                    T s = V::zero();
#pragma unroll 1
                    for (int q = 0; q < n; q++, pos += 8) {
                        const uint2 v = lds<uint2>(ring + (pos & (kORing - 1)));
                        constexpr uint32_t m = 0xffffu << kShift;
                        const T c0 = lds<T>(C + (((v.x << kShift) & m) ^ lb)), c1 = lds<T>(C + (((v.x >> (16 - kShift)) & m) ^ lb));
                        const T c2 = lds<T>(C + (((v.y << kShift) & m) ^ lb)), c3 = lds<T>(C + (((v.y >> (16 - kShift)) & m) ^ lb));
                        s = V::add(s, V::add(V::add(c0, c1), V::add(c2, c3)));
                    }
                    acc[j4 + jj] = V::add(acc[j4 + jj], s);
                }
            }
            if (nchunks == 2) {
                __syncwarp();
                fetch(head + 3 * kOChunk);
                head += kOChunk;
            }
        };

        int tgt_chunks = 0;
        for (int st = s0; st < s1; st++) {
            gather(tgt_chunks);
            // products: this warp's rows warp, warp + 16, ...
            uint32_t at = next();
            const uint4 hd = lds<uint4>(at);  // products, contraction quads, target chunks
            uint32_t prow = P + warp * kRow + lb;
#pragma unroll 1
            for (uint32_t k = 0; k < hd.x; k++, prow += kOWarps * kRow) {
                at += 16;
                const uint4 d = lds<uint4>(at);
                const uint32_t w[4] = {d.x, d.y, d.z, d.w};
                T x[4], y[4];
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    x[q] = y[q] = V::zero();
                    if ((int)w[q] >= 0) {
                        constexpr uint32_t m = 0x7fffu << kShift;
                        x[q] = lds<T>(F + (((w[q] << kShift) & m) ^ lb));
                        y[q] = lds<T>(F + (((w[q] >> (16 - kShift)) & m) ^ lb));
                    }
                }
                T p = V::mac(x[0], y[0], V::mac(x[1], y[1], V::zero()));
                p = V::add(p, V::mac(x[2], y[2], V::mac(x[3], y[3], V::zero())));
                // a reflection of an axis on which D is its own mirror repeats D
                const uint32_t self = ((w[0] >> 15) & 1u) | ((w[1] >> 14) & 2u) | ((w[2] >> 13) & 4u);
                if (self & (uint32_t)r) p = V::zero();
                sts(prow, p);
            }
            __syncthreads();
            // contraction: per quad four entries {P offset; the block's four weights};
            // bit 0 of the first offset: last quad of its block, bit 1: the block's
            // sums continue those of an earlier part; the C row in the second's top bits
            T c0 = V::zero(), c1 = V::zero(), c2 = V::zero(), c3 = V::zero();
            for (uint32_t left = hd.y; left > 0;) {
                uint32_t e = next();
                const uint32_t n = min(left, (uint32_t)kOQuads);
                left -= n;
#pragma unroll 1
                for (uint32_t q = 0; q < n; q++, e += 80) {
                    const uint4 o = lds<uint4>(e);
                    const float4 w0 = lds<float4>(e + 16), w1 = lds<float4>(e + 32), w2 = lds<float4>(e + 48),
                                 w3 = lds<float4>(e + 64);
                    const T p0 = lds<T>(P + (o.x & ~3u) + lb), p1 = lds<T>(P + (o.y & 0x3ffffu) + lb);
                    const T p2 = lds<T>(P + o.z + lb), p3 = lds<T>(P + o.w + lb);
                    const uint32_t cr = C + (o.y >> 18) * kRow + lb;
                    if (o.x & 2u) {
                        c0 = lds<T>(cr);
                        c1 = lds<T>(cr + kRow);
                        c2 = lds<T>(cr + 2 * kRow);
                        c3 = lds<T>(cr + 3 * kRow);
                    }
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
                    if (o.x & 1u) {
                        sts(cr, c0);
                        sts(cr + kRow, c1);
                        sts(cr + 2 * kRow, c2);
                        sts(cr + 3 * kRow, c3);
                        c0 = c1 = c2 = c3 = V::zero();
                    }
                }
            }
            tgt_chunks = (int)hd.z;
            __syncthreads();
        }
        gather(tgt_chunks);
        asm volatile("cp.async.wait_group 0;" ::: "memory");  // the copies ahead of the last chunk
        // lane (r, cells): output row 8 o + r
        const int cell = blockIdx.x * CPT + (lane & 3) * (CPT / 4);
#pragma unroll
        for (int j = 0; j < NSLOT; j++) {
            const int o = warp + j * kOWarps;
            if (o >= a.norb) continue;
            const int row = 8 * o + r;
            if (a.part) {
                *reinterpret_cast<T *>(a.part + ((size_t)blockIdx.y * a.ns + row) * a.cells_pad + cell) = acc[j];
            } else {
                float *g = a.gain + (size_t)__ldg(a.row_node + row) * a.ld + cell;
                const float *v = reinterpret_cast<const float *>(&acc[j]);
#pragma unroll
                for (int q = 0; q < CPT / 4; q++)
                    if (cell + q < a.ncells) g[q] = v[q];
            }
        }
    } else if (a.part) {  // an empty chunk (more chunks than work): zero partial sums
        for (int t = threadIdx.x; t < a.ns * CPT; t += kOThreads)
            a.part[((size_t)blockIdx.y * a.ns + t / CPT) * a.cells_pad + blockIdx.x * CPT + t % CPT] = 0.f;
    }
}

// ft[tile][row][CPT] from f[node][cell]: the packed rows the product loads
// read; cells past ncells are zero.  Block = 32 cells x 8 rows.
__global__ void orbit_pack_kernel(const float *__restrict__ f, int ld, int ncells, int ns, int cpt,
                                  const int *__restrict__ row_node, float *__restrict__ ft, int cells_pad)
{
    const int cell = blockIdx.x * 32 + threadIdx.x, row = blockIdx.y * 8 + threadIdx.y;
    if (row >= ns || cell >= cells_pad) return;
    const float v = cell < ncells ? f[(size_t)__ldg(row_node + row) * ld + cell] : 0.f;
    ft[((size_t)(cell / cpt) * ns + row) * cpt + cell % cpt] = v;
}

// gain[node][cell] = sum over the chunks: each of the block's eight y rows adds
// a contiguous eighth of the chunks in order, and the eight are added in order.
__global__ void orbit_reduce_kernel(const float *__restrict__ part, int nchunks, int ns, int cells_pad, int ncells,
                                    int ld, const int *__restrict__ row_node, float *__restrict__ gain)
{
    __shared__ float red[8][32];
    const int x = threadIdx.x, y = threadIdx.y;
    const int o = blockIdx.x * 32 + x;
    const int total = ns * ncells;
    const int row = o < total ? o / ncells : 0, cell = o < total ? o - row * ncells : 0;
    const int k0 = nchunks * y / 8, k1 = nchunks * (y + 1) / 8;
    const float *p = part + (size_t)row * cells_pad + cell;
    const size_t step = (size_t)ns * cells_pad;
    float s = 0.f;
#pragma unroll 4
    for (int k = k0; k < k1; k++) s += __ldg(p + (size_t)k * step);
    red[y][x] = s;
    __syncthreads();
    if (y == 0 && o < total) {
        for (int k = 1; k < 8; k++) s += red[k][x];
        gain[(size_t)__ldg(row_node + row) * ld + cell] = s;
    }
}

// One D of the low octant with anything to do.
struct DItem {
    int K = 0, nblk = 0;
    std::vector<uint4> prod;                   // by shell |n|
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
    for (auto &kv : g->bounds_dev) cudaFree(kv.second);
    delete g;
    c.orbit = nullptr;
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
    for (int m = 0; m < d.n_pnt; m++) {
        if (c.ui[m] >= d.hx || c.vi[m] >= d.hy || c.wi[m] >= d.hz) continue;
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
            const uint32_t self = (D[0] == d.nx - 1 ? 1u : 0u) | (D[1] == d.ny - 1 ? 2u : 0u) | (D[2] == d.nz - 1 ? 4u : 0u);
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
                        uint32_t pw[4], have = 0;
                        int np = 0;
                        for (int q = 0; q < 4; q++) {
                            const int t1 = at[pat[q]], t2 = at[7 - pat[q]];
                            if (t1 >= 0 && t2 >= 0) pw[np++] = (uint32_t)t1 | (uint32_t)t2 << 16;
                        }
                        have = np;
                        while (np < 4) pw[np++] = kNoPair;
                        const int k = (x2 * d.hy + y2) * d.hz + z2;
                        if (have) {
                            for (int q = 0; q < 3; q++)
                                if ((self >> q) & 1u) pw[q] |= 0x8000u;
                            it.K++;
                            cls.push_back(k);
                            n2.push_back((double)(d.du * n[0]) * (d.du * n[0]) + (double)(d.dv * n[1]) * (d.dv * n[1]) +
                                         (double)(d.dw * n[2]) * (d.dw * n[2]));
                            it.prod.push_back(make_uint4(pw[0], pw[1], pw[2], pw[3]));
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
                std::vector<uint4> sorted(it.K);
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
    {
        const int nt = std::max(1, std::min(8, (int)std::thread::hardware_concurrency()));
        std::vector<std::thread> th;
        for (int t = 1; t < nt; t++) th.emplace_back(build_items, t, nt);
        build_items(0, nt);
        for (auto &t : th) t.join();
    }
    int mmax = 0;
    int64_t ktotal = 0;
    for (const DItem &it : items) {
        ktotal += it.K;
        mmax = std::max(mmax, it.nblk * kORows);
    }
    if (!ktotal || !mmax) return GD_OK;

    // tile width: eight cells where their outputs and rows fit, else four
    int max_smem = 0;
    GD_CUDA(cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, c.device));
    const int slots = (norb + kOWarps - 1) / kOWarps;
    int cpt = 0, nslot = 0, pcap = 0, mcap = 0;
    for (int w : {8, 4}) {
        if (!orbit_kernel(w, slots, &nslot)) continue;
        const int rows = (max_smem - kOWarps * kORing - d.n_pnt * w * 4) / (32 * w) - 1;  // P and C rows
        mcap = std::min(8184, std::max(mmax, rows * 2 / 5 / kORows * kORows));
        pcap = std::min(kOWarps * kOProd, rows - mcap);
        if (pcap >= 64) {
            cpt = w;
            break;
        }
    }
    if (!cpt) return GD_OK;
    // a small lattice still gets ~96 steps, so that few cells spread over the SMs
    const int kstep = std::min(pcap, std::max(32, (int)(ktotal / 96)));
    const uint32_t row_bytes = 32u * (uint32_t)cpt;

    OrbitGain *og = new OrbitGain;
    og->cuts.push_back(0);
    og->cost_prefix.push_back(0.0);
    double cost = 0.0;
    std::vector<std::vector<uint4>> ws(kOWarps);  // the warps' streams
    std::vector<std::vector<int>> start(kOWarps);
    auto pad_chunk = [](std::vector<uint4> &v) {
        while (v.size() % (kOChunk / 16)) v.push_back(make_uint4(0, 0, 0, 0));
    };
    std::vector<std::vector<uint16_t>> tl(norb);
    const int max_quads = (2 * kOChunk - nslot) / 8;
    auto list_quads = [&](int warp) {
        int q = 0;
        for (int o = warp; o < norb; o += kOWarps) q += ((int)tl[o].size() + 3) / 4;
        return q;
    };
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
        std::vector<const uint4 *> prod;
        int mrow = 0;
        double entries = 0.0, targets = 0.0;
        for (const Part &pt : parts) {
            const DItem &it = items[pt.item];
            const int kbase = (int)prod.size();
            for (int k = pt.k0; k < pt.k1; k++) prod.push_back(&it.prod[k]);
            int e0 = 0;
            for (int b = 0; b < it.nblk; e0 += it.blk_n[b++]) {
                const auto lo = it.off.begin() + e0, hi = lo + it.blk_n[b];
                const int f0 = (int)(std::lower_bound(lo, hi, (uint32_t)pt.k0) - lo),
                          f1 = (int)(std::lower_bound(lo, hi, (uint32_t)pt.k1) - lo);
                // a block starts in the first part that has entries of it, or
                // in the first part when no part has (its C rows are zero)
                if (f0 == f1 && !(pt.k0 == 0 && it.blk_n[b] == 0)) continue;
                bl.push_back(Blk{f1 - f0, pt.item, b, e0 + f0, mrow + b * kORows, pt.k0, kbase, f0 > 0});
                entries += f1 - f0;
            }
            mrow += it.nblk * kORows;
        }
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
            start[w].push_back((int)(v.size() / (kOChunk / 16)));
            const size_t h = v.size();
            v.push_back(make_uint4(0, 0, 0, 0));
            uint32_t np = 0, nq = 0;
            for (size_t k = w; k < prod.size(); k += kOWarps, np++) v.push_back(*prod[k]);
            pad_chunk(v);
            for (const Blk *b : mine[w]) {
                const DItem &it = items[b->item];
                const int quads = std::max(1, (b->n + 3) / 4);
                for (int q = 0; q < quads; q++, nq++) {
                    if (nq && nq % kOQuads == 0) pad_chunk(v);
                    uint32_t off[4];
                    float4 wt[4];
                    for (int z = 0; z < 4; z++) {
                        const int e = 4 * q + z;
                        // padding repeats a row of the block with weight 0
                        const int row = b->n ? (int)it.off[b->e0 + std::min(e, b->n - 1)] - b->k0 : 0;
                        off[z] = (uint32_t)(row + b->kbase) * row_bytes;
                        wt[z] = e < b->n ? it.w[b->e0 + e] : make_float4(0.f, 0.f, 0.f, 0.f);
                    }
                    off[0] |= (q == quads - 1 ? 1u : 0u) | (q == 0 && b->cont ? 2u : 0u);
                    off[1] |= (uint32_t)b->crow << 18;
                    v.push_back(make_uint4(off[0], off[1], off[2], off[3]));
                    for (int z = 0; z < 4; z++) {
                        uint4 u;
                        std::memcpy(&u, &wt[z], 16);
                        v.push_back(u);
                    }
                }
            }
            pad_chunk(v);
            uint32_t tc = 0;
            std::vector<uint8_t> list(nslot, 0);
            for (int j = 0, o = w; o < norb; j++, o += kOWarps) {
                list[j] = (uint8_t)((tl[o].size() + 3) / 4);
                targets += (double)tl[o].size();
                for (size_t t = 0; t < (size_t)list[j] * 4; t++) {
                    const uint16_t e = t < tl[o].size() ? tl[o][t] : (uint16_t)(mcap << 3);  // the zero row
                    list.push_back((uint8_t)(e & 255));
                    list.push_back((uint8_t)(e >> 8));
                }
            }
            if ((int)list.size() > nslot) {
                list.resize((list.size() + 15) / 16 * 16, 0);
                const size_t at = v.size();
                v.resize(at + list.size() / 16);
                std::memcpy(&v[at], list.data(), list.size());
                pad_chunk(v);
                tc = (uint32_t)((v.size() - at) / (kOChunk / 16));
            }
            v[h] = make_uint4(np, nq, tc, 0);
        }
        cost += 600.0 + 15.0 * (double)prod.size() + 3.5 * entries + 8.0 * (double)bl.size() + 2.3 * targets;
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
        for (int w = 0; fits && w < kOWarps; w++) fits = list_quads(w) <= max_quads;
        for (const auto &t : it.targets) fits = fits && tl[t.first >> 3].size() <= 1020;
        if (!fits)
            for (const auto &t : it.targets) tl[t.first >> 3].pop_back();
        return fits;
    };
    for (int Did = 0; Did < d.nxyz; Did++) {
        const DItem &it = items[Did];
        if (!it.nblk) continue;
        if (it.K > kstep) {  // parts of its own
            close();
            const int parts = (it.K + kstep - 1) / kstep;
            for (int p = 0; p < parts; p++) {
                if (p == parts - 1 && !add_targets(it)) {
                    delete og;
                    return GD_OK;
                }
                emit({Part{Did, (int)((int64_t)it.K * p / parts), (int)((int64_t)it.K * (p + 1) / parts)}}, p == parts - 1);
            }
            continue;
        }
        for (int pass = 0; pass < 2; pass++) {
            if (krow + it.K <= kstep && mrow + it.nblk * kORows <= mcap && add_targets(it)) {
                krow += it.K;
                mrow += it.nblk * kORows;
                cur.push_back(Part{Did, 0, it.K});
                break;
            }
            if (cur.empty()) {  // a single D that does not fit
                delete og;
                return GD_OK;
            }
            close();
        }
    }
    close();
    og->cpt = cpt;
    og->nslot = nslot;
    og->norb = norb;
    og->pcap = pcap;
    og->mcap = mcap;
    og->smem = (size_t)kOWarps * kORing + (size_t)d.n_pnt * cpt * 4 + (size_t)(pcap + mcap + 1) * row_bytes;
    // one buffer: warp after warp, each followed by the chunks that the last
    // steps fetch ahead
    std::vector<uint4> stream;
    std::vector<int> st((size_t)og->nsteps * kOWarps);
    for (int w = 0; w < kOWarps; w++) {
        const int base = (int)(stream.size() / (kOChunk / 16));
        for (int k = 0; k < og->nsteps; k++) st[(size_t)k * kOWarps + w] = base + start[w][k];
        stream.insert(stream.end(), ws[w].begin(), ws[w].end());
        stream.resize(stream.size() + 4 * (kOChunk / 16), make_uint4(0, 0, 0, 0));
        std::vector<uint4>().swap(ws[w]);
    }
    c.orbit = og;
    int rc = upload(&og->row_node, row_node);
    if (!rc) rc = upload(&og->stream, stream);
    if (!rc) rc = upload(&og->start, st);
    if (!rc) rc = fold_loss_build(c);
    return rc;  // the caller destroys the context on failure
}

// Chunks of the steps for a batch: at least gain_waves CTAs per SM (a CTA
// fills an SM), and of the next few counts the one whose last wave is fullest.
int orbit_chunks(const Context &c, int ncells)
{
    const OrbitGain &g = *c.orbit;
    const int tiles = (ncells + g.cpt - 1) / g.cpt, sms = std::max(1, c.sm_count);
    const int most = (int)g.cuts.size() - 1;
    const int lo = std::min(most, std::max(1, (std::max(1, c.gain_waves) * sms + tiles - 1) / tiles));
    int best = lo;
    double best_fill = 0.0;
    for (int k = lo; k <= std::min(most, lo + 8); k++) {
        const int64_t ctas = (int64_t)tiles * k;
        const double fill = (double)ctas / (double)((ctas + sms - 1) / sms * sms) - 0.002 * (k - lo);
        if (fill > best_fill + 1e-9) {
            best_fill = fill;
            best = k;
        }
    }
    return best;
}

size_t orbit_pack_bytes(const Context &c, int ncells)
{
    const int cpt = c.orbit->cpt;
    return (size_t)((ncells + cpt - 1) / cpt * cpt) * c.d.n_pnt * sizeof(float);
}

// partial sums of nchunks chunks (one chunk writes the gain itself)
size_t orbit_part_bytes(const Context &c, int ncells, int nchunks)
{
    return nchunks > 1 ? orbit_pack_bytes(c, ncells) * (size_t)nchunks : 0;
}

void orbit_chunk_bounds(const Context &c, int nchunks, int *bounds)
{
    const OrbitGain &g = *c.orbit;
    const std::vector<double> &pre = g.cost_prefix;
    const int n = (int)g.cuts.size() - 1;
    int at = 0;
    bounds[0] = 0;
    for (int k = 1; k < nchunks; k++) {
        const double want = pre[n] * k / nchunks;
        int b = (int)(std::lower_bound(pre.begin(), pre.end(), want) - pre.begin());
        if (b > 0 && want - pre[b - 1] < pre[b] - want) b--;
        at = std::min(n, std::max(at, b));
        bounds[k] = g.cuts[at];
    }
    bounds[nchunks] = g.nsteps;
}

int launch_orbit(Context &c, const float *f, int ncells, int ld, float *gain, void *buf, int nchunks,
                 const int *d_bounds, cudaStream_t st)
{
    OrbitGain &g = *c.orbit;
    const Dims &d = c.d;
    const int tiles = (ncells + g.cpt - 1) / g.cpt, cells_pad = tiles * g.cpt;
    if ((int64_t)d.n_pnt * std::max(ld, cells_pad) >= ((int64_t)1 << 31))
        return set_error(GD_ERR_UNSUPPORTED, "pair gain: n_pnt * ld must stay below 2^31");
    float *ft = static_cast<float *>(buf);
    float *part = nchunks > 1 ? ft + (size_t)cells_pad * d.n_pnt : nullptr;
    orbit_pack_kernel<<<dim3((cells_pad + 31) / 32, d.n_pnt / 8), dim3(32, 8), 0, st>>>(
        f, ld, ncells, d.n_pnt, g.cpt, g.row_node, ft, cells_pad);
    GD_CUDA(cudaGetLastError());
    const OrbitArgs a{ft,     g.stream, g.start,   d_bounds, g.row_node, part,  gain,
                      g.norb, d.n_pnt,  cells_pad, ncells,   ld,         g.pcap, g.mcap};
    int nslot = 0;
    OrbitKernel kern = orbit_kernel(g.cpt, g.nslot, &nslot);
    GD_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)g.smem));
    kern<<<dim3(tiles, nchunks), kOThreads, g.smem, st>>>(a);
    GD_CUDA(cudaGetLastError());
    if (part) {
        const int64_t outs = (int64_t)d.n_pnt * ncells;
        orbit_reduce_kernel<<<(unsigned)((outs + 31) / 32), dim3(32, 8), 0, st>>>(part, nchunks, d.n_pnt, cells_pad, ncells,
                                                                                 ld, g.row_node, gain);
        GD_CUDA(cudaGetLastError());
    }
    return GD_OK;
}

int run_orbit(Context &c, const float *f, int ncells, int ld, float *gain, cudaStream_t st)
{
    OrbitGain &g = *c.orbit;
    const int nchunks = orbit_chunks(c, ncells);
    auto it = g.bounds_dev.find(nchunks);
    if (it == g.bounds_dev.end()) {
        std::vector<int> b(nchunks + 1);
        orbit_chunk_bounds(c, nchunks, b.data());
        int *dev = nullptr;
        GD_CUDA(cudaMalloc(&dev, sizeof(int) * (nchunks + 1)));
        cudaError_t e = cudaMemcpy(dev, b.data(), sizeof(int) * (nchunks + 1), cudaMemcpyHostToDevice);
        if (e != cudaSuccess) {
            cudaFree(dev);
            return cuda_error(e, "gain chunk bounds");
        }
        it = g.bounds_dev.emplace(nchunks, dev).first;
    }
    int rc = ensure_scratch(c, orbit_pack_bytes(c, ncells) + orbit_part_bytes(c, ncells, nchunks));
    if (rc) return rc;
    return launch_orbit(c, f, ncells, ld, gain, c.scratch.ptr, nchunks, it->second, st);
}

}  // namespace gd
