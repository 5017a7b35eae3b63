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
// A CTA takes one tile of CPT cells and one chunk of the steps; a step is as
// many D as fit the P and C buffers, so that the two barriers of a step are
// paid for ~1e4 cycles of work.  Contraction works on blocks of four rows of
// neighbouring |g|, whose shells overlap: one P row is read for four rows
// (1.2 times the terms, a third of the shared-memory reads).
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
constexpr int kORows = 4;              // rows of a contraction block
constexpr int kOStage = 1024;          // bytes of a warp's staged target list
constexpr uint32_t kNoPair = 0xffffffffu;

struct OrbitArgs {
    const float *ft;       // [tile][row][CPT]
    const uint4 *prod;     // per P row up to four pairs t1 | t2 << 16 (kNoPair: none); bit 15 of the
                           // low half of word a: axis a of D is its own mirror
    const int4 *steps;     // {first product, products, 0, 0}
    const int4 *work;      // [step][warp] {first block, end block, first quad of the target list, quads}
    const int4 *blocks;    // {first entry, entry quads, C byte offset, 0}
    const uint4 *ent_off;  // P byte offsets of four entries
    const float4 *ent_w;   // the four rows' weights of one entry
    const uint2 *targets;  // per (step, warp): a count per slot (bytes, in quads), then 16-bit entries row << 3 | e
    const int *bounds;     // [chunks + 1] step bounds
    const int *row_node;
    float *part;           // [chunk][row][cells_pad], or null: write gain
    float *gain;
    int norb, ns, cells_pad, ncells, ld;
    int kcap, mcap;
};

template <int CPT>
struct Vec;
template <>
struct Vec<8> {
    using T = float2;
    static __device__ __forceinline__ T zero() { return make_float2(0.f, 0.f); }
    static __device__ __forceinline__ T fma(T a, T b, T c) { return make_float2(__fmaf_rn(a.x, b.x, c.x), __fmaf_rn(a.y, b.y, c.y)); }
    static __device__ __forceinline__ T fma(float w, T b, T c) { return make_float2(__fmaf_rn(w, b.x, c.x), __fmaf_rn(w, b.y, c.y)); }
    static __device__ __forceinline__ T add(T a, T b) { return make_float2(a.x + b.x, a.y + b.y); }
};
template <>
struct Vec<4> {
    using T = float;
    static __device__ __forceinline__ T zero() { return 0.f; }
    static __device__ __forceinline__ T fma(T a, T b, T c) { return __fmaf_rn(a, b, c); }
    static __device__ __forceinline__ T add(T a, T b) { return a + b; }
};

template <int CPT, int NSLOT>
__global__ void __launch_bounds__(kOThreads, 1) orbit_gain_kernel(const __grid_constant__ OrbitArgs a)
{
    using V = Vec<CPT>;
    using T = typename V::T;
    constexpr uint32_t kRow = 32 * sizeof(T);        // bytes of a P or C row
    constexpr int kEntryShift = CPT == 8 ? 5 : 4;    // (row << 3 | e) -> bytes: e selects CPT cells
    extern __shared__ __align__(1024) unsigned char smem[];
    unsigned char *P = smem;
    unsigned char *C = smem + (size_t)a.kcap * kRow;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned char *stage = C + (size_t)(a.mcap + 1) * kRow + warp * kOStage;
    const uint32_t lb = lane * (uint32_t)sizeof(T);  // r * (CPT cells) + cell, in bytes
    const int r = lane >> 2;
    const unsigned char *ft = reinterpret_cast<const unsigned char *>(a.ft + (size_t)blockIdx.x * a.ns * CPT);
    T acc[NSLOT];
#pragma unroll
    for (int j = 0; j < NSLOT; j++) acc[j] = V::zero();
    if (warp == 0) *reinterpret_cast<T *>(C + (size_t)a.mcap * kRow + lb) = V::zero();  // padding targets read this row

    const int s0 = a.bounds[blockIdx.y], s1 = a.bounds[blockIdx.y + 1];
    // targets of the step whose list is staged: C rows into this warp's outputs
    auto gather = [&]() {
        const unsigned char *pos = stage + NSLOT;
#pragma unroll
        for (int j4 = 0; j4 < NSLOT; j4 += 4) {
            const uint32_t cw = *reinterpret_cast<const uint32_t *>(stage + j4);
            if (cw == 0) continue;
#pragma unroll
            for (int jj = 0; jj < 4; jj++) {
                const int n = (cw >> (8 * jj)) & 255;
                T s = V::zero();
#pragma unroll 1
                for (int q = 0; q < n; q++, pos += 8) {
                    const uint2 v = *reinterpret_cast<const uint2 *>(pos);
                    constexpr uint32_t m = 0xffffu << kEntryShift;
                    const uint32_t o0 = ((v.x << kEntryShift) & m) ^ lb, o1 = ((v.x >> (16 - kEntryShift)) & m) ^ lb;
                    const uint32_t o2 = ((v.y << kEntryShift) & m) ^ lb, o3 = ((v.y >> (16 - kEntryShift)) & m) ^ lb;
                    const T c0 = *reinterpret_cast<const T *>(C + o0), c1 = *reinterpret_cast<const T *>(C + o1);
                    const T c2 = *reinterpret_cast<const T *>(C + o2), c3 = *reinterpret_cast<const T *>(C + o3);
                    s = V::add(s, V::add(V::add(c0, c1), V::add(c2, c3)));
                }
                acc[j4 + jj] = V::add(acc[j4 + jj], s);
            }
        }
    };

    for (int st = s0; st < s1; st++) {
        if (st > s0) gather();
        // products
        const int4 hd = __ldg(a.steps + st);
        for (int k = warp; k < hd.y; k += kOWarps) {
            const uint4 d = __ldg(a.prod + hd.x + k);
            const uint32_t w[4] = {d.x, d.y, d.z, d.w};
            T x[4], y[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                x[q] = y[q] = V::zero();
                if ((int)w[q] >= 0) {
                    constexpr uint32_t m = 0x7fffu << kEntryShift;
                    const uint32_t o1 = ((w[q] << kEntryShift) & m) ^ lb;
                    const uint32_t o2 = ((w[q] >> (16 - kEntryShift)) & m) ^ lb;
                    x[q] = __ldg(reinterpret_cast<const T *>(ft + o1));
                    y[q] = __ldg(reinterpret_cast<const T *>(ft + o2));
                }
            }
            T p = V::fma(x[0], y[0], V::fma(x[1], y[1], V::zero()));
            p = V::add(p, V::fma(x[2], y[2], V::fma(x[3], y[3], V::zero())));
            // a reflection of an axis on which D is its own mirror repeats D
            const uint32_t self = ((w[0] >> 15) & 1u) | ((w[1] >> 14) & 2u) | ((w[2] >> 13) & 4u);
            if (self & (uint32_t)r) p = V::zero();
            *reinterpret_cast<T *>(P + (size_t)k * kRow + lb) = p;
        }
        __syncthreads();
        // contraction
        const int4 wk = __ldg(a.work + st * kOWarps + warp);
        for (int i = lane; i < wk.w; i += 32)
            reinterpret_cast<uint2 *>(stage)[i] = __ldg(a.targets + wk.z + i);
        for (int b = wk.x; b < wk.y; b++) {
            const int4 h = __ldg(a.blocks + b);
            T c0 = V::zero(), c1 = V::zero(), c2 = V::zero(), c3 = V::zero();
            const uint4 *po = a.ent_off + (h.x >> 2);
            const float4 *pw = a.ent_w + h.x;
#pragma unroll 2
            for (int g = 0; g < h.y; g++, po++, pw += 4) {
                const uint4 o = __ldg(po);
                const float4 w0 = __ldg(pw), w1 = __ldg(pw + 1), w2 = __ldg(pw + 2), w3 = __ldg(pw + 3);
                const T p0 = *reinterpret_cast<const T *>(P + o.x + lb), p1 = *reinterpret_cast<const T *>(P + o.y + lb);
                const T p2 = *reinterpret_cast<const T *>(P + o.z + lb), p3 = *reinterpret_cast<const T *>(P + o.w + lb);
#define GD_MAC(wv, pv)           \
    c0 = V::fma((wv).x, pv, c0); \
    c1 = V::fma((wv).y, pv, c1); \
    c2 = V::fma((wv).z, pv, c2); \
    c3 = V::fma((wv).w, pv, c3)
                GD_MAC(w0, p0);
                GD_MAC(w1, p1);
                GD_MAC(w2, p2);
                GD_MAC(w3, p3);
#undef GD_MAC
            }
            unsigned char *cr = C + h.z + lb;
            *reinterpret_cast<T *>(cr) = c0;
            *reinterpret_cast<T *>(cr + kRow) = c1;
            *reinterpret_cast<T *>(cr + 2 * kRow) = c2;
            *reinterpret_cast<T *>(cr + 3 * kRow) = c3;
        }
        __syncthreads();
    }
    if (s1 > s0) gather();
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
    std::vector<uint4> prod;
    std::vector<int> blk_n;                    // entries per block, padded to four
    std::vector<uint32_t> off;                 // P row per entry
    std::vector<float4> w;
    std::vector<std::pair<int, int>> targets;  // (output row 8 o + e, C row), by output row
};

}  // namespace

struct OrbitGain {
    int cpt = 8, nslot = 0, norb = 0, kcap = 0, mcap = 0, nsteps = 0;
    size_t smem = 0;
    std::vector<double> cost_prefix;  // [nsteps + 1]
    int *row_node = nullptr;
    uint4 *prod = nullptr;
    int4 *steps = nullptr, *work = nullptr, *blocks = nullptr;
    uint4 *ent_off = nullptr;
    float4 *ent_w = nullptr;
    uint2 *targets = nullptr;
    std::map<int, int *> bounds_dev;
};

void orbit_free(Context &c)
{
    OrbitGain *g = c.orbit;
    if (!g) return;
    cudaFree(g->row_node);
    cudaFree(g->prod);
    cudaFree(g->steps);
    cudaFree(g->work);
    cudaFree(g->blocks);
    cudaFree(g->ent_off);
    cudaFree(g->ent_w);
    cudaFree(g->targets);
    for (auto &kv : g->bounds_dev) cudaFree(kv.second);
    delete g;
    c.orbit = nullptr;
}

namespace {

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
                                {4, 48, orbit_gain_kernel<4, 48>}, {4, 64, orbit_gain_kernel<4, 64>}};
    for (const Inst &i : inst)
        if (i.cpt == cpt && i.nslot >= need) {
            *nslot = i.nslot;
            return i.k;
        }
    return nullptr;
}

}  // namespace

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
        for (int Did = t0; Did < d.nxyz; Did += nt) {
            const int D[3] = {Did / d.nyz, (Did / d.nz) % d.ny, Did % d.nz};
            DItem &it = items[Did];
            const uint32_t self = (D[0] == d.nx - 1 ? 1u : 0u) | (D[1] == d.ny - 1 ? 2u : 0u) | (D[2] == d.nz - 1 ? 4u : 0u);
            cls.clear();
            want.clear();
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
                        while (np < 4) pw[np++] = kNoPair & ~0x8000u;
                        const int k = (x2 * d.hy + y2) * d.hz + z2;
                        if (have) {
                            for (int q = 0; q < 3; q++)
                                if ((self >> q) & 1u) pw[q] |= 0x8000u;
                            prow[k] = it.K++;
                            cls.push_back(k);
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
                    int n = (int)touched.size();
                    for (; n & 3; n++) {  // padding repeats a row of the block with weight 0
                        it.off.push_back((uint32_t)touched[0]);
                        it.w.push_back(make_float4(0.f, 0.f, 0.f, 0.f));
                    }
                    it.blk_n.push_back(n);
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
    int kmax = 0, mmax = 0;
    for (const DItem &it : items) {
        kmax = std::max(kmax, it.K);
        mmax = std::max(mmax, it.nblk * kORows);
    }
    if (!kmax || !mmax) return GD_OK;

    // tile width: eight cells where their outputs and rows fit, else four
    int max_smem = 0;
    GD_CUDA(cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, c.device));
    const int slots = (norb + kOWarps - 1) / kOWarps;
    int cpt = 0, nslot = 0, cap = 0;
    for (int w : {8, 4}) {
        if (!orbit_kernel(w, slots, &nslot)) continue;
        cap = (max_smem - kOWarps * kOStage) / (32 * 4 * (w / 4)) - 1;  // P and C rows
        if (cap >= kmax + mmax) {
            cpt = w;
            break;
        }
    }
    if (!cpt) return GD_OK;
    const int mcap = std::min({8188, std::max(mmax, cap * 3 / 10 / kORows * kORows), (cap - kmax) / kORows * kORows});
    const int kcap = cap - mcap;
    // a small lattice still gets ~96 steps, so that few cells spread over the SMs
    int64_t ktotal = 0;
    for (const DItem &it : items) ktotal += it.K;
    const int kstep = std::min(kcap, std::max<int>(kmax, (int)(ktotal / 96)));
    const uint32_t row_bytes = 32u * 4u * (uint32_t)(cpt / 4);

    // steps: consecutive D while their rows and target lists fit
    std::vector<uint4> prod;
    std::vector<int4> steps, work, blocks;
    std::vector<uint32_t> ent_off;
    std::vector<float4> ent_w;
    std::vector<uint2> targets;
    OrbitGain *og = new OrbitGain;
    og->cost_prefix.push_back(0.0);
    const int max_quads = (kOStage - nslot) / 8;
    std::vector<int> cur;
    std::vector<std::vector<uint16_t>> tl(norb);
    auto list_quads = [&](int warp) {
        int q = 0;
        for (int o = warp; o < norb; o += kOWarps) q += ((int)tl[o].size() + 3) / 4;
        return q;
    };
    auto close_step = [&]() {
        // the blocks go to the warps largest first, each to the least loaded
        struct Blk {
            int cost, item, b, e0, row;
        };
        std::vector<Blk> bl;
        int krow = 0, mrow = 0;
        const int p0 = (int)prod.size();
        std::vector<int> kbase(cur.size());
        double cost = 0.0;
        for (size_t i = 0; i < cur.size(); i++) {
            const DItem &it = items[cur[i]];
            kbase[i] = krow;
            prod.insert(prod.end(), it.prod.begin(), it.prod.end());
            int e0 = 0;
            for (int b = 0; b < it.nblk; b++) {
                bl.push_back(Blk{it.blk_n[b] * 3 + 30, (int)i, b, e0, mrow + b * kORows});
                e0 += it.blk_n[b];
            }
            cost += 9.0 * it.K + 4.0 * e0 + 2.5 * (double)it.targets.size();
            krow += it.K;
            mrow += it.nblk * kORows;
        }
        std::stable_sort(bl.begin(), bl.end(), [](const Blk &x, const Blk &y) { return x.cost > y.cost; });
        std::vector<std::vector<const Blk *>> mine(kOWarps);
        std::vector<int> load(kOWarps, 0);
        for (const Blk &b : bl) {
            const int w = (int)(std::min_element(load.begin(), load.end()) - load.begin());
            load[w] += b.cost;
            mine[w].push_back(&b);
        }
        steps.push_back(make_int4(p0, krow, 0, 0));
        for (int w = 0; w < kOWarps; w++) {
            const int b0 = (int)blocks.size(), q0 = (int)targets.size();
            for (const Blk *b : mine[w]) {
                const DItem &it = items[cur[b->item]];
                const int n = it.blk_n[b->b];
                blocks.push_back(make_int4((int)ent_w.size(), n / 4, (int)((uint32_t)b->row * row_bytes), 0));
                for (int e = 0; e < n; e++) {
                    ent_off.push_back((it.off[b->e0 + e] + (uint32_t)kbase[b->item]) * row_bytes);
                    ent_w.push_back(it.w[b->e0 + e]);
                }
            }
            std::vector<uint8_t> cnt(nslot, 0);
            std::vector<uint16_t> ent;
            for (int j = 0, o = w; o < norb; j++, o += kOWarps) {
                cnt[j] = (uint8_t)((tl[o].size() + 3) / 4);
                ent.insert(ent.end(), tl[o].begin(), tl[o].end());
                while (ent.size() & 3) ent.push_back((uint16_t)(mcap << 3));  // the zero row
            }
            const size_t quads = (size_t)nslot / 8 + ent.size() / 4;
            targets.resize(q0 + quads);
            std::memcpy(&targets[q0], cnt.data(), nslot);
            if (!ent.empty()) std::memcpy(&targets[q0 + nslot / 8], ent.data(), ent.size() * 2);
            work.push_back(make_int4(b0, (int)blocks.size(), q0, (int)quads));
        }
        og->cost_prefix.push_back(og->cost_prefix.back() + cost);
        for (auto &t : tl) t.clear();
        cur.clear();
    };
    int krow = 0, mrow = 0;
    for (int Did = 0; Did < d.nxyz; Did++) {
        const DItem &it = items[Did];
        if (!it.nblk) continue;
        for (int pass = 0; pass < 2; pass++) {
            bool fits = krow + it.K <= kstep && mrow + it.nblk * kORows <= mcap;
            if (fits) {
                for (const auto &t : it.targets) tl[t.first >> 3].push_back((uint16_t)((mrow + t.second) << 3 | (t.first & 7)));
                for (int w = 0; fits && w < kOWarps; w++) fits = list_quads(w) <= max_quads;
                for (const auto &t : it.targets) fits = fits && tl[t.first >> 3].size() <= 1020;
                if (!fits)
                    for (const auto &t : it.targets) tl[t.first >> 3].pop_back();
            }
            if (fits) {
                krow += it.K;
                mrow += it.nblk * kORows;
                cur.push_back(Did);
                break;
            }
            if (cur.empty()) {  // a single D that does not fit
                delete og;
                return GD_OK;
            }
            close_step();
            krow = mrow = 0;
        }
    }
    if (!cur.empty()) close_step();
    og->cpt = cpt;
    og->nslot = nslot;
    og->norb = norb;
    og->kcap = kcap;
    og->mcap = mcap;
    og->nsteps = (int)steps.size();
    og->smem = (size_t)(kcap + mcap + 1) * row_bytes + kOWarps * kOStage;
    std::vector<uint4> off4(ent_off.size() / 4);
    if (!off4.empty()) std::memcpy(off4.data(), ent_off.data(), ent_off.size() * 4);
    c.orbit = og;
    int rc = upload(&og->row_node, row_node);
    if (!rc) rc = upload(&og->prod, prod);
    if (!rc) rc = upload(&og->steps, steps);
    if (!rc) rc = upload(&og->work, work);
    if (!rc) rc = upload(&og->blocks, blocks);
    if (!rc) rc = upload(&og->ent_off, off4);
    if (!rc) rc = upload(&og->ent_w, ent_w);
    if (!rc) rc = upload(&og->targets, targets);
    return rc;  // the caller destroys the context on failure
}

// Chunks of the steps for a batch: at least gain_waves CTAs per SM (a CTA
// fills an SM), and of the next few counts the one whose last wave is fullest.
int orbit_chunks(const Context &c, int ncells)
{
    const OrbitGain &g = *c.orbit;
    const int tiles = (ncells + g.cpt - 1) / g.cpt, sms = std::max(1, c.sm_count);
    const int lo = std::min(g.nsteps, std::max(1, (std::max(1, c.gain_waves) * sms + tiles - 1) / tiles));
    int best = lo;
    double best_fill = 0.0;
    for (int k = lo; k <= std::min(g.nsteps, lo + 8); k++) {
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
    const std::vector<double> &pre = c.orbit->cost_prefix;
    const int n = c.orbit->nsteps;
    bounds[0] = 0;
    for (int k = 1; k < nchunks; k++) {
        const double want = pre[n] * k / nchunks;
        int b = (int)(std::lower_bound(pre.begin(), pre.end(), want) - pre.begin());
        if (b > 0 && want - pre[b - 1] < pre[b] - want) b--;
        bounds[k] = std::min(n, std::max(bounds[k - 1], b));
    }
    bounds[nchunks] = n;
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
    const OrbitArgs a{ft,        g.prod,     g.steps, g.work, g.blocks, g.ent_off, g.ent_w, g.targets, d_bounds,
                      g.row_node, part,      gain,    g.norb, d.n_pnt,  cells_pad, ncells,  ld,        g.kcap, g.mcap};
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
