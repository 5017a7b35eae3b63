// gd_project.cu -- FP64 conservation projection, relaxation step, moments and
// the correction basis (sm_103a).
//
// Projection (intended semantics of collision_integral.cu:217-526, one 5x5
// system per cell): with phi = (1, xi_x, xi_y, xi_z, xi^2),
//   A_kl = sum_i f_i nu_i phi_k phi_l,  B_k = sum_i (I_i - f_i nu_i) phi_k,
//   A X = B,  nu'_i = nu_i (1 + X.phi_i),  Q_i = I_i - f_i nu'_i,
// after which sum_i Q_i phi_k = 0 (mass, momentum, energy) up to FP64 rounding.
// The nodes of one (x, y) form a line along z, and the sums over a line need only
// powers of z: 11 FP64 accumulators per node (z^0..z^4 of f nu, z^0..z^2 of I - f nu
// and of f) that enter the 25 sums once per line, 18 FP64 operations per node and
// cell instead of 46; the second pass likewise takes two fused operations for 1 +
// X.phi instead of five.  The lines fall into 8 to 64 classes (project_classes): a
// class is summed line after line, the classes' sums are added as a tree.  That order
// is the lattice's alone, so a cell's results have the same bits in any batch,
// whichever way the work is split: a warp takes LC cells times 32 / LC classes, or,
// for few cells, lines of one cell (LC = 1), and a cluster of CTAs shares the lines
// of its cells.
// Bound: the FP64 pipe (its rate is 1/64 of the FP32 rate and a hardware float to
// double conversion takes a slot of it, so to_double does that in integers).
// 20^3: 4096 cells 1.54 -> 0.84 ms, 256 cells 1.6 -> 0.095, one cell 1.6 -> 0.046
// (with the splits free to change the order of the sums: 0.84, 0.092 and 0.057).
#include "gd_internal.h"
#include "gd_tc.cuh"

#include <algorithm>
#include <cfloat>

namespace gd {
namespace {

constexpr int kWarps = 8;
constexpr int kSums = 25;  // 5 B, 15 A (upper triangle), 5 moments
constexpr size_t kProjSmem = (size_t)(kWarps + 1) * kSums * 32 * sizeof(double);  // the warps' sums, the CTA's

struct ProjArgs {
    Dims d;
    const float *f, *nu, *gain;
    int ld, ncells;
    int nlines, classes;    // lines l, l + classes, ... are summed in order, the classes' sums as a tree
    const int4 *lines;      // {first node, end node, z index of the first, 0}
    const double2 *line_xy;
    const double2 *zpow;    // (z, z^2), (z^3, z^4) per z index
    float *nu_corr;
    double *q;
    double *x;
    int update;  // 1: write f_out = f + dt Q
    float dt;
    float *f_out;
    double *m5;
    unsigned int *status;  // [0] flags (1 non-finite sums, 2 singular system), [1] first cell
};

// Gaussian elimination with partial pivoting on a symmetric 5x5 system, all
// indices static (rows swapped by selection).  Singular (false): what is left of a
// column is nowhere above the rounding of the sums it came from, 2^-50 of the root of
// the row's and the column's diagonal entries.  A cell with all its mass on one node
// leaves at most 2.7e-16 there (all nodes of 8^3 to 20^3; an exact zero for two thirds
// of them), a Maxwellian of half the lattice's step in width 1e-6.
__device__ __forceinline__ bool solve5(double A[5][5], double b[5], double x[5])
{
    double rs[5], cs[5];  // the rows' and the columns' scales
#pragma unroll
    for (int k = 0; k < 5; k++) rs[k] = cs[k] = fabs(A[k][k]);
#pragma unroll
    for (int k = 0; k < 5; k++) {
        int piv = k;
        double best = fabs(A[k][k]);
#pragma unroll
        for (int r = k + 1; r < 5; r++)
            if (fabs(A[r][k]) > best) {
                best = fabs(A[r][k]);
                piv = r;
            }
        bool any = false;
#pragma unroll
        for (int r = k; r < 5; r++) any = any || A[r][k] * A[r][k] > 0x1p-100 * rs[r] * cs[k];
        if (!(best > 0.0) || !any) return false;
#pragma unroll
        for (int r = k + 1; r < 5; r++) {
            const bool p = piv == r;
            const double su = rs[k], sv = rs[r];
            rs[k] = p ? sv : su;
            rs[r] = p ? su : sv;
#pragma unroll
            for (int t = k; t < 5; t++) {
                const double u = A[k][t], v = A[r][t];
                A[k][t] = p ? v : u;
                A[r][t] = p ? u : v;
            }
            const double u = b[k], v = b[r];
            b[k] = p ? v : u;
            b[r] = p ? u : v;
        }
#pragma unroll
        for (int r = k + 1; r < 5; r++) {
            const double m = A[r][k] / A[k][k];
#pragma unroll
            for (int t = k; t < 5; t++) A[r][t] -= m * A[k][t];
            b[r] -= m * b[k];
        }
    }
#pragma unroll
    for (int k = 4; k >= 0; k--) {
        double s = b[k];
#pragma unroll
        for (int t = k + 1; t < 5; t++) s -= A[k][t] * x[t];
        x[k] = s / A[k][k];
    }
    return true;
}

// A double in another CTA's shared memory (same offset), rank `rank`.
__device__ __forceinline__ double peer_load(const double *p, uint32_t rank)
{
    double v;
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(tc::mapa_cluster(tc::smem_u32(p), rank)) : "memory");
    return v;
}

// (double)v, by moving the bits where v is a normal number.
__device__ __forceinline__ double to_double(float v)
{
    const uint32_t u = __float_as_uint(v);
    if (((u >> 23) & 255u) - 1u < 254u)
        return __hiloint2double((int)((u & 0x80000000u) | (((u & 0x7fffffffu) >> 3) + 0x38000000u)), (int)(u << 29));
    return (double)v;
}

// What the 25 sums need of a line: powers of z.
struct LineSums {
    double S0, S1, S2, S3, S4, R0, R1, R2, M0, M1, M2;
};
constexpr int kLineSums = 11;

template <bool M5>
__device__ __forceinline__ LineSums sum_line(const ProjArgs &a, int4 ln, int cell)
{
    LineSums v = {};
    const double2 *zp = a.zpow + 2 * ln.z;
    size_t o = (size_t)ln.x * a.ld + cell;
#pragma unroll 4
    for (int i = ln.x; i < ln.y; i++, zp += 2, o += a.ld) {
        const double fv = to_double(a.f[o]), nv = to_double(a.nu[o]), gv = to_double(a.gain[o]);
        const double z = zp[0].x, z2 = zp[0].y;
        const double fn = fv * nv, r = gv - fn;
        v.R0 = __dadd_rn(v.R0, r);
        v.R1 = __fma_rn(r, z, v.R1);
        v.R2 = __fma_rn(r, z2, v.R2);
        v.S0 = __dadd_rn(v.S0, fn);
        v.S1 = __fma_rn(fn, z, v.S1);
        v.S2 = __fma_rn(fn, z2, v.S2);
        v.S3 = __fma_rn(fn, zp[1].x, v.S3);
        v.S4 = __fma_rn(fn, zp[1].y, v.S4);
        if (M5) {
            v.M0 = __dadd_rn(v.M0, fv);
            v.M1 = __fma_rn(fv, z, v.M1);
            v.M2 = __fma_rn(fv, z2, v.M2);
        }
    }
    return v;
}

// A line's part of the sums.  Every operation is spelled out: wherever a line is
// added the bits are the same.
template <bool M5>
__device__ __forceinline__ void add_line(double *s, const LineSums &v, double2 xy)
{
    const double x = xy.x, y = xy.y, rho = __fma_rn(x, x, __dmul_rn(y, y));
    const double E0 = __fma_rn(rho, v.S0, v.S2), E1 = __fma_rn(rho, v.S1, v.S3),
                 E2 = __fma_rn(rho, __dadd_rn(E0, v.S2), v.S4), xS = __dmul_rn(x, v.S0), yS = __dmul_rn(y, v.S0);
    s[0] = __dadd_rn(s[0], v.R0);
    s[1] = __fma_rn(x, v.R0, s[1]);
    s[2] = __fma_rn(y, v.R0, s[2]);
    s[3] = __dadd_rn(s[3], v.R1);
    s[4] = __dadd_rn(s[4], __fma_rn(rho, v.R0, v.R2));
    s[5] = __dadd_rn(s[5], v.S0);
    s[6] = __dadd_rn(s[6], xS);
    s[7] = __dadd_rn(s[7], yS);
    s[8] = __dadd_rn(s[8], v.S1);
    s[9] = __dadd_rn(s[9], E0);
    s[10] = __fma_rn(x, xS, s[10]);
    s[11] = __fma_rn(x, yS, s[11]);
    s[12] = __fma_rn(x, v.S1, s[12]);
    s[13] = __fma_rn(x, E0, s[13]);
    s[14] = __fma_rn(y, yS, s[14]);
    s[15] = __fma_rn(y, v.S1, s[15]);
    s[16] = __fma_rn(y, E0, s[16]);
    s[17] = __dadd_rn(s[17], v.S2);
    s[18] = __dadd_rn(s[18], E1);
    s[19] = __dadd_rn(s[19], E2);
    if (M5) {
        s[20] = __dadd_rn(s[20], v.M0);
        s[21] = __fma_rn(x, v.M0, s[21]);
        s[22] = __fma_rn(y, v.M0, s[22]);
        s[23] = __dadd_rn(s[23], v.M1);
        s[24] = __dadd_rn(s[24], __fma_rn(rho, v.M0, v.M2));
    }
}

// Sum of n = 1, 2, 4 or 8 values, neighbours first.
template <typename F>
__device__ __forceinline__ double tree8(int n, F value)
{
    double v[8];
#pragma unroll
    for (int k = 0; k < 8; k++) v[k] = k < n ? value(k) : 0.;
#pragma unroll
    for (int w = 1; w < 8; w *= 2)
#pragma unroll
        for (int k = 0; k < 8; k += 2 * w)
            if (w < n) v[k] += v[k + w];
    return v[0];
}

template <bool M5, int LC>
__global__ void __launch_bounds__(kWarps * 32, LC == 1 ? 3 : 2) project_kernel(const __grid_constant__ ProjArgs a, int cs)
{
    extern __shared__ __align__(16) double red[];  // [kWarps][kSums][32], then the CTA's sums [kSums][32]
    __shared__ double xs[5][32];
    double *mine = red + kWarps * kSums * 32;
    constexpr int NS = M5 ? kSums : kSums - 5;  // without the moments
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int rank = (int)blockIdx.x % cs;
    constexpr int G = 32 / LC;  // lines side by side in a warp
    const int col = lane % LC;
    const int cell = (int)blockIdx.x / cs * LC + col;
    const bool live = cell < a.ncells;
    // this thread's lines: a class of them, or where one cell has a CTA to itself
    // (LC = 1) every line its own thread; CTA r then takes the classes c % cs == r
    const int first = LC == 1 ? rank + (int)threadIdx.x * cs : (rank * kWarps + warp) * G + lane / LC;
    const int step = LC == 1 ? (int)blockDim.x * cs : a.classes;
    double s[kSums];
#pragma unroll
    for (int k = 0; k < NS; k++) s[k] = 0.;
    if (LC == 1) {
        double *ls = red;  // [line of the CTA][kLineSums]
        for (int l = first; l < a.nlines; l += step)
            *reinterpret_cast<LineSums *>(ls + (size_t)(l / cs) * kLineSums) = sum_line<M5>(a, __ldg(a.lines + l), cell);
        __syncthreads();
        const int c = rank + (int)threadIdx.x * cs;
        if (c < a.classes)
            for (int l = c; l < a.nlines; l += a.classes)
                add_line<M5>(s, *reinterpret_cast<const LineSums *>(ls + (size_t)(l / cs) * kLineSums), __ldg(a.line_xy + l));
        __syncthreads();
        double *cl = red;  // [class of the CTA][kSums]
        if (c < a.classes)
#pragma unroll
            for (int k = 0; k < NS; k++) cl[(size_t)(c / cs) * kSums + k] = s[k];
        if (cs > 1) tc::cluster_sync();
        else __syncthreads();
        // the classes' sums, neighbours first: a warp per sum
        if (rank == 0)
            for (int k = warp; k < NS; k += kWarps) {
                double v[2];
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int q = lane + 32 * h;
                    v[h] = q >= a.classes ? 0. : cs > 1 ? peer_load(cl + (size_t)(q / cs) * kSums + k, (uint32_t)(q % cs))
                                                        : cl[(size_t)q * kSums + k];
#pragma unroll
                    for (int w = 1; w < 32; w *= 2) {
                        const double u = __shfl_xor_sync(0xffffffffu, v[h], w);
                        if (w < a.classes) v[h] += u;
                    }
                }
                mine[k * 32 + lane] = __shfl_sync(0xffffffffu, a.classes > 32 ? v[0] + v[1] : v[0], 0);
            }
        if (rank == 0) __syncthreads();
    } else {
        if (live)
            for (int l = first; l < a.nlines; l += step)
                add_line<M5>(s, sum_line<M5>(a, __ldg(a.lines + l), cell), __ldg(a.line_xy + l));
        // the classes' sums, neighbours first: over the lane groups, the warps and the CTAs
#pragma unroll
        for (int k = 0; k < NS; k++) {
#pragma unroll
            for (int w = LC; w < 32; w *= 2) s[k] += __shfl_xor_sync(0xffffffffu, s[k], w);
            red[((size_t)warp * kSums + k) * 32 + lane] = s[k];
        }
        __syncthreads();
        for (int t = threadIdx.x; t < NS * 32; t += kWarps * 32)
            mine[t] = tree8(kWarps, [&](int w) { return red[(size_t)w * kSums * 32 + t]; });
        if (cs > 1) tc::cluster_sync();
        else __syncthreads();
        if (rank == 0 && cs > 1) {
            for (int t = threadIdx.x; t < NS * 32; t += kWarps * 32)
                red[t] = tree8(cs, [&](int k) { return k == 0 ? mine[t] : peer_load(mine + t, (uint32_t)k); });
            __syncthreads();
        }
    }
    if (rank == 0) {
        if (warp == 0) {
            const double *all = LC != 1 && cs > 1 ? red : mine;
            double tot[kSums] = {};
#pragma unroll
            for (int k = 0; k < NS; k++) tot[k] = all[k * 32 + lane];
            double A[5][5], B[5], X[5];
            int t = 5;
#pragma unroll
            for (int k = 0; k < 5; k++) B[k] = tot[k];
#pragma unroll
            for (int k = 0; k < 5; k++)
#pragma unroll
                for (int l = k; l < 5; l++) {
                    A[k][l] = tot[t];
                    A[l][k] = tot[t];
                    t++;
                }
            bool finite = true;
#pragma unroll
            for (int k = 0; k < NS; k++) finite = finite && isfinite(tot[k]);
            const bool solved = finite && solve5(A, B, X);
            if (!solved) {
#pragma unroll
                for (int k = 0; k < 5; k++) X[k] = 0.;
                // recorded for gd_ctx_check: the flags OR together, the smallest
                // failing cell wins, so the record does not depend on scheduling
                bool record = live && lane < LC && a.status;
                if (record && finite) {
                    // an empty cell has nothing to correct (its mass is not among the
                    // sums: it would cost every cell a sixteenth of the pipe's time)
                    double mass = 0.;
                    for (int i = 0; i < a.d.n_pnt; i++) mass += to_double(a.f[(size_t)i * a.ld + cell]);
                    record = mass != 0.;
                }
                if (record) {
                    atomicOr(a.status, finite ? 2u : 1u);
                    atomicMin(a.status + 1, (unsigned int)cell);
                }
            }
#pragma unroll
            for (int k = 0; k < 5; k++) xs[k][lane] = X[k];
            if (live && lane < LC) {
                if (a.x)
#pragma unroll
                    for (int k = 0; k < 5; k++) a.x[(size_t)cell * 5 + k] = X[k];
                if (M5 && a.m5)
#pragma unroll
                    for (int k = 0; k < 5; k++) a.m5[(size_t)cell * 5 + k] = tot[20 + k] * (double)a.d.d3v;
            }
        }
    }
    double X[5];
    if (cs > 1) {
        tc::cluster_sync();
#pragma unroll
        for (int k = 0; k < 5; k++) X[k] = peer_load(&xs[k][lane], 0);
        // rank 0's shared memory stays until every CTA has read it
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    } else {
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 5; k++) X[k] = xs[k][lane];
    }
    if (live) {
        for (int l = first; l < a.nlines; l += step) {
            const int4 ln = __ldg(a.lines + l);
            const double2 xy = __ldg(a.line_xy + l);
            const double rho = __fma_rn(xy.x, xy.x, __dmul_rn(xy.y, xy.y));
            const double c0 = __fma_rn(X[4], rho, __fma_rn(X[2], xy.y, __fma_rn(X[1], xy.x, __dadd_rn(1., X[0]))));
            const double2 *zp = a.zpow + 2 * ln.z;
            size_t o = (size_t)ln.x * a.ld + cell;
#pragma unroll 4
            for (int i = ln.x; i < ln.y; i++, zp += 2, o += a.ld) {
                const double fv = to_double(a.f[o]), nv = to_double(a.nu[o]), gv = to_double(a.gain[o]);
                const double nc = __dmul_rn(nv, __fma_rn(X[4], zp->y, __fma_rn(X[3], zp->x, c0)));
                const double qv = __fma_rn(-fv, nc, gv);
                if (a.nu_corr) a.nu_corr[o] = (float)nc;
                if (a.q) a.q[o] = qv;
                if (a.update) a.f_out[o] = (float)__fma_rn((double)a.dt, qv, fv);
            }
        }
    }
    if (cs > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Per-block maximum of nu' (non-negative); a second launch with one block
// reduces the block maxima.  Block b takes the rows b, b + gridDim.x, ..., its
// threads the cells of each row (32-bit indices, four loads in flight per
// thread).  The maximum does not depend on the order.
__global__ void max_kernel(const float *__restrict__ v, int n_pnt, int ncells, int ld,
                           float *__restrict__ out)
{
    __shared__ float sm[256];
    float m0 = 0.f, m1 = 0.f, m2 = 0.f, m3 = 0.f;
    const int step = blockDim.x;
    for (int node = blockIdx.x; node < n_pnt; node += gridDim.x) {
        const float *row = v + (size_t)node * ld;
        int c = threadIdx.x;
        for (; c + 3 * step < ncells; c += 4 * step) {
            m0 = fmaxf(m0, __ldg(row + c));
            m1 = fmaxf(m1, __ldg(row + c + step));
            m2 = fmaxf(m2, __ldg(row + c + 2 * step));
            m3 = fmaxf(m3, __ldg(row + c + 3 * step));
        }
        for (; c < ncells; c += step) m0 = fmaxf(m0, __ldg(row + c));
    }
    sm[threadIdx.x] = fmaxf(fmaxf(m0, m1), fmaxf(m2, m3));
    __syncthreads();
    for (int s = 128; s > 0; s >>= 1) {
        if (threadIdx.x < s) sm[threadIdx.x] = fmaxf(sm[threadIdx.x], sm[threadIdx.x + s]);
        __syncthreads();
    }
    if (threadIdx.x == 0) out[blockIdx.x] = sm[0];
}

// dt = courant / max nu' (get_delta_t, collision_integral.cu:776-807: the
// minimum of courant/nu over all nodes and cells equals courant over the
// largest nu after rounding, since division is monotone), or a fixed dt.
__global__ void dt_kernel(const float *__restrict__ blockmax, int nb, int mode, float param,
                          float *__restrict__ dt_out, float *__restrict__ time_dev,
                          float *__restrict__ dt_user)
{
    if (blockIdx.x != 0 || threadIdx.x >= 32) return;
    float dt = param;
    if (mode == GD_DT_COURANT) {
        // one warp: lanes take strided block maxima, then a shuffle maximum
        float m = 0.f;
        for (int k = threadIdx.x; k < nb; k += 32) m = fmaxf(m, blockmax[k]);
        for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        dt = m > 0.f ? param / m : 1.0e10f;
    }
    if (threadIdx.x != 0) return;
    *dt_out = dt;
    if (dt_user) *dt_user = dt;
    if (time_dev) *time_dev += dt;
}

// f <- f + dt (I - f nu')  (evolve_f, collision_integral.cu:809-833), in FP64.
// Block b takes the rows b, b + gridDim.x, ..., its threads the cells of each
// row (32-bit indices).
__global__ void relax_kernel(float *__restrict__ f, const float *__restrict__ nu,
                             const float *__restrict__ gain, const double *__restrict__ q, int n_pnt,
                             int ncells, int ld, const float *__restrict__ dt_dev)
{
    const double dt = *dt_dev;
    for (int node = blockIdx.x; node < n_pnt; node += gridDim.x) {
        const size_t r = (size_t)node * ld;
        for (int c = threadIdx.x; c < ncells; c += blockDim.x) {
            const size_t o = r + c;
            const double fv = f[o];
            const double qv = q ? q[o] : (double)gain[o] - fv * (double)nu[o];
            f[o] = (float)(fv + dt * qv);
        }
    }
}

__global__ void __launch_bounds__(kWarps * 32) moments_kernel(Dims d, const float *__restrict__ f,
                                                              int ld, int ncells,
                                                              const double *__restrict__ phi,
                                                              double *__restrict__ m5)
{
    __shared__ double red[kWarps][5][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int cell = blockIdx.x * 32 + lane;
    const bool live = cell < ncells;
    const int n = d.n_pnt;
    double s[5] = {0., 0., 0., 0., 0.};
    if (live)
        for (int i = warp; i < n; i += kWarps) {
            const double fv = f[(size_t)i * ld + cell];
            s[0] += fv;
#pragma unroll
            for (int k = 1; k < 5; k++) s[k] += fv * phi[k * n + i];
        }
#pragma unroll
    for (int k = 0; k < 5; k++) red[warp][k][lane] = s[k];
    __syncthreads();
    if (warp == 0 && live)
        for (int k = 0; k < 5; k++) {
            double v = 0.;
            for (int w = 0; w < kWarps; w++) v += red[w][k][lane];
            m5[(size_t)cell * 5 + k] = v * (double)d.d3v;
        }
}

// The 14 basis rows of fill_correction_array (velocity.cu:17-50) over the box,
// in float as the reference forms them.
__global__ void basis_kernel(Dims d, const float *__restrict__ u, const float *__restrict__ v,
                             const float *__restrict__ w, float *__restrict__ out)
{
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= d.nxyz) return;
    const int k = idx % d.nz, j = (idx / d.nz) % d.ny, i = idx / d.nyz;
    const float xx = u[i], xy = v[j], xz = w[k];
    float x2 = xx * xx;
    x2 = x2 + xy * xy;
    x2 = x2 + xz * xz;
    const float vals[14] = {xx, xy, xz, x2, xx * xx, xx * xy, xx * xz, xx * x2,
                            xy * xy, xy * xz, xy * x2, xz * xz, xz * x2, x2 * x2};
#pragma unroll
    for (int r = 0; r < 14; r++) out[(size_t)r * d.nxyz + idx] = vals[r];
}

}  // namespace

// Classes of lines (8 to 64): about four lines in each.
int project_classes(const Context &c)
{
    int n = 8;
    while (n < 64 && n * 4 < c.nlines) n *= 2;
    return n;
}

// Cells per warp (32, 16 or 8: a class of lines per thread; 1: a line per thread) and
// CTAs per group of cells, by the FP64 pipe's time in instructions of a warp (about
// ten in a us).  A class per thread: so many lines each (15 per node and 40 per
// line), then 20 sums over lanes, warps and CTAs (about 125); an SM works off its
// CTAs one after the other; clusters of four and eight find room in fewer SMs (their
// GPC's); one CTA per SM waits for its loads when they come from HBM.  A line per
// thread: three CTAs wait for their loads side by side.  Measured, us (cells per
// warp, CTAs), 20^3: one cell (1, 2) 46, (1, 1) 59, (32, 8) 125; 256 cells (1, 1) 95,
// (32, 8) 127; 512 (16, 4) 132, (1, 1) 182, (32, 8) 220; 1024 (32, 8) 237, (16, 4)
// 241; 4096 (32, 8) 841, (16, 4) 881, (8, 2) 911; 8^3: 400 cells (1, 1) 35, (32, 2)
// 46; 512 (1, 1) 61, (32, 2) 46.
struct ProjSplit {
    int lc, cs;
};
ProjSplit project_split(const Context &c, int ncells)
{
    const int sms = std::max(1, c.sm_count), classes = project_classes(c);
    const double line = 15.0 * c.d.n_pnt / c.nlines + 40.0;
    const bool hbm = (int64_t)c.d.n_pnt * ncells > ((int64_t)100 << 20) / 24;
    ProjSplit best{0, 0};
    double least = 0.0;
    for (int lc : {32, 16, 8, 1})
        for (int cs = 1; cs <= 8; cs *= 2) {
            const int64_t ctas = ((int64_t)ncells + lc - 1) / lc * cs;
            double cost = 0.0;
            if (lc == 1) {
                // the sums of a CTA's lines in shared memory
                if (cs > 2 || (c.nlines + cs - 1) / cs * kLineSums > kWarps * kSums * 32) continue;
                cost = 240.0 * (double)((ctas + 3 * sms - 1) / (3 * sms)) +
                       (double)((ctas + sms - 1) / sms) * (c.nlines * line / (cs * kWarps * 32) + 50.0);
                if (hbm) cost *= 1.2;  // a sector for each value
            } else {
                if (cs * kWarps * (32 / lc) != classes) continue;
                const int room = cs == 8 ? sms * 3 / 4 : cs == 4 ? sms * 11 / 12 : sms;
                const int many = cs >= 4 ? std::max(1, sms * 14 / 15) : sms;
                const int64_t turns = ctas <= room ? 1 : std::max<int64_t>(2, (ctas + many - 1) / many);
                cost = (double)turns * ((c.nlines + classes - 1) / classes * line + 125.0);
                if (turns == 1 && hbm) cost *= 1.15;
                cost *= lc == 8 ? 1.15 : lc == 16 ? 1.04 : 1.0;  // rows of 32 and 64 bytes
            }
            if (least == 0.0 || cost < least * (1.0 - 1e-9)) {
                least = cost;
                best = ProjSplit{lc, cs};
            }
        }
    return best;
}

int run_project(Context &c, const float *f, const float *nu, const float *gain, int ncells, int ld,
                float *nu_corr, double *q, double *x, int fixed_dt_mode, float dt, float *f_out,
                double *m5, cudaStream_t st)
{
    const ProjArgs a{c.d,   f, nu, gain, ld, ncells, c.nlines, project_classes(c), c.d_lines, c.d_line_xy, c.d_zpow, nu_corr,
                     q,     x, fixed_dt_mode ? 1 : 0, dt, f_out, m5,     c.d_status};
    const ProjSplit split = project_split(c, ncells);
    const int lc = split.lc, cs = split.cs, blocks = (ncells + lc - 1) / lc;
    auto kern = lc == 32 ? (m5 ? project_kernel<true, 32> : project_kernel<false, 32>)
                : lc == 16 ? (m5 ? project_kernel<true, 16> : project_kernel<false, 16>)
                : lc == 8 ? (m5 ? project_kernel<true, 8> : project_kernel<false, 8>)
                          : (m5 ? project_kernel<true, 1> : project_kernel<false, 1>);
    GD_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kProjSmem));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(blocks * cs));
    cfg.blockDim = dim3(kWarps * 32);
    cfg.dynamicSmemBytes = kProjSmem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)cs;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    GD_CUDA(cudaLaunchKernelEx(&cfg, kern, a, cs));
    GD_CUDA(cudaGetLastError());
    return GD_OK;
}

int run_relax_q(Context &c, float *f, const float *nu_corr, const float *gain, const double *q,
                int ncells, int ld, int mode, float param, float *time_dev, float *dt_dev,
                cudaStream_t st)
{
    // blocks of the maximum: a few per SM, within the reduction buffer
    const int nb = std::max(1, std::min(std::min(4 * c.sm_count, kReduceFloats - 1), c.d.n_pnt));
    float *blockmax = c.d_reduce;        // [nb]
    float *dt_scalar = c.d_reduce + nb;  // [1]
    if (mode == GD_DT_COURANT) {
        max_kernel<<<nb, 256, 0, st>>>(nu_corr, c.d.n_pnt, ncells, ld, blockmax);
        GD_CUDA(cudaGetLastError());
    }
    dt_kernel<<<1, 32, 0, st>>>(blockmax, nb, mode, param, dt_scalar, time_dev, dt_dev);
    GD_CUDA(cudaGetLastError());
    const int blocks = std::min(c.d.n_pnt, c.sm_count * 16);
    relax_kernel<<<std::max(blocks, 1), 256, 0, st>>>(f, nu_corr, gain, q, c.d.n_pnt, ncells, ld, dt_scalar);
    GD_CUDA(cudaGetLastError());
    return GD_OK;
}

int run_relax(Context &c, float *f, const float *nu_corr, const float *gain, int ncells, int ld,
              int mode, float param, float *time_dev, float *dt_dev, cudaStream_t st)
{
    return run_relax_q(c, f, nu_corr, gain, nullptr, ncells, ld, mode, param, time_dev, dt_dev, st);
}

int run_moments(Context &c, const float *f, int ncells, int ld, double *m5, cudaStream_t st)
{
    moments_kernel<<<(ncells + 31) / 32, kWarps * 32, 0, st>>>(c.d, f, ld, ncells, c.d_phi, m5);
    GD_CUDA(cudaGetLastError());
    return GD_OK;
}

int run_basis(Context &c, float *basis, cudaStream_t st)
{
    float *du = nullptr;
    const size_t n = c.u.size() + c.v.size() + c.w.size();
    GD_CUDA(cudaMallocAsync(&du, sizeof(float) * n, st));
    cudaError_t e = cudaMemcpyAsync(du, c.u.data(), sizeof(float) * c.u.size(), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(du + c.u.size(), c.v.data(), sizeof(float) * c.v.size(), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(du + c.u.size() + c.v.size(), c.w.data(), sizeof(float) * c.w.size(),
                            cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) {
        basis_kernel<<<(c.d.nxyz + 255) / 256, 256, 0, st>>>(c.d, du, du + c.u.size(),
                                                             du + c.u.size() + c.v.size(), basis);
        e = cudaGetLastError();
    }
    cudaError_t e2 = cudaFreeAsync(du, st);
    if (e != cudaSuccess) return cuda_error(e, "correction basis");
    if (e2 != cudaSuccess) return cuda_error(e2, "correction basis free");
    return GD_OK;
}

}  // namespace gd
