// gd_loss.cu -- loss frequency nu_i = sum_j b(|i - j|) f_j (sm_103a).
//
// Reference: evolve_direct_colisions, collision_integral.cu:32-72 (full-box
// partner loop; f is zero outside the sphere so only in-sphere partners
// contribute).  The reference sums all partners in one FP32 chain; both
// kernels here sum short chains and add them with compensated (Kahan)
// summation, which keeps the frequency within a few FP32 ulp of the FP64 sum
// (one chain over the ~3600 partners of a 20^3 grid drifts to ~2e-6): the loss
// multiplies f in Q = I - f nu, where near equilibrium I and f nu agree to
// 1e-3, so its rounding shows up a thousandfold in Q.
//
// folded_loss_kernel serves the lattices with orbit rows (gd_orbit.cu): b is
// invariant under the lattice's reflections, so with nodes (o, e) (orbit,
// octant) and the eight characters s(x, e) = (-1)^popcount(x & e) of the group,
//   nu(o, e) = 1/8 sum_x s(x, e) sum_o' B_x[o][o'] f_x[o'],
//   f_x[o'] = sum_e s(x, e) f(o', e),  B_x[o][o'] = sum_e s(x, e) b((o, 0), (o', e)):
// eight products of an eighth of the size each way, an eighth of the work.
// loss_kernel (lane = cell, kRows outputs per warp, b and the node coordinates
// in shared memory) serves the other lattices.  20^3: 4096 cells 22.1 -> 0.64 ms,
// one cell 0.89 -> 0.029 ms;
// the folded sums are the closer ones to FP64 (3.2e-8 against 4.2e-8 relative
// L2 at 20^3), since their chains are sixteen long and unfolded in FP64.
#include "gd_internal.h"

#include <algorithm>

namespace gd {
namespace {

constexpr int kRows = 8;
constexpr int kWarps = 8;
constexpr int kBlock = 64;  // partners per partial chain

__global__ void __launch_bounds__(kWarps * 32) loss_kernel(Dims d, const float *__restrict__ f, int ld,
                                                           int ncells, const float *__restrict__ b,
                                                           const uint32_t *__restrict__ nodes,
                                                           float *__restrict__ nu)
{
    extern __shared__ __align__(16) unsigned char smem[];
    float *bs = reinterpret_cast<float *>(smem);
    uint32_t *ns = reinterpret_cast<uint32_t *>(smem + (((size_t)d.nxyz * 4 + 15) & ~(size_t)15));
    for (int t = threadIdx.x; t < d.nxyz; t += blockDim.x) bs[t] = b[t];
    for (int t = threadIdx.x; t < d.n_pnt; t += blockDim.x) ns[t] = nodes[t];
    __syncthreads();

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int cell = blockIdx.x * 32 + lane;
    const bool live = cell < ncells;
    const float *fcol = f + (live ? cell : 0);
    const int row0 = (blockIdx.y * kWarps + warp) * kRows;
    if (row0 >= d.n_pnt) return;
    int ox[kRows], oy[kRows], oz[kRows];
#pragma unroll
    for (int r = 0; r < kRows; r++) {
        const int node = min(row0 + r, d.n_pnt - 1);
        const uint32_t p = ns[node];
        ox[r] = p & 1023;
        oy[r] = (p >> 10) & 1023;
        oz[r] = p >> 20;
    }
    float acc[kRows], comp[kRows];
#pragma unroll
    for (int r = 0; r < kRows; r++) acc[r] = comp[r] = 0.f;
    for (int j0 = 0; j0 < d.n_pnt; j0 += kBlock) {
        float part[kRows];
#pragma unroll
        for (int r = 0; r < kRows; r++) part[r] = 0.f;
        const int j1 = min(j0 + kBlock, d.n_pnt);
        for (int j = j0; j < j1; j++) {
            const uint32_t p = ns[j];
            const int jx = p & 1023, jy = (p >> 10) & 1023, jz = p >> 20;
            const float fj = live ? __ldg(fcol + (size_t)j * ld) : 0.f;
#pragma unroll
            for (int r = 0; r < kRows; r++) {
                const int idx = abs(ox[r] - jx) * d.nyz + abs(oy[r] - jy) * d.nz + abs(oz[r] - jz);
                part[r] = __fmaf_rn(bs[idx], fj, part[r]);
            }
        }
#pragma unroll
        for (int r = 0; r < kRows; r++) {
            const float y = __fsub_rn(part[r], comp[r]);
            const float t = __fadd_rn(acc[r], y);
            comp[r] = __fsub_rn(__fsub_rn(t, acc[r]), y);
            acc[r] = t;
        }
    }
    if (!live) return;
#pragma unroll
    for (int r = 0; r < kRows; r++)
        if (row0 + r < d.n_pnt) nu[(size_t)(row0 + r) * ld + cell] = acc[r];
}

// Folded loss: CTA = TO orbits x TC cells, warp x = character x; a thread holds
// 4 orbits x TC / 4 cells.  Per sixteen orbits o' the CTA folds f of its cells
// into shared memory (one thread per (o', cell): eight loads, 24 additions) and
// copies the B_x tiles with cp.async, both for the next sixteen while the
// current ones are multiplied.  Bound by FP32 issue (the products and a quarter
// as much for the compensated sums).
constexpr int kFo = 32;  // orbits per CTA
constexpr int kFk = 16;  // orbits o' per step: the length of a partial chain

template <int TC>
constexpr size_t folded_smem()
{
    const size_t stages = 2 * 8 * kFk * (kFo + TC) * sizeof(float), out = 8 * kFo * TC * sizeof(double);
    return stages > out ? stages : out;
}

template <int TC>
__global__ void __launch_bounds__(256, 2) folded_loss_kernel(const float *__restrict__ f, int ld, int ncells, int norb, int opad,
                                                          const int *__restrict__ row_node,
                                                          const float *__restrict__ bx,  // [8][o'][opad]
                                                          float *__restrict__ nu)
{
    constexpr int NC = TC / 4;                        // cells per thread
    constexpr int kItems = (kFk * TC + 255) / 256;    // (o', cell) folds per thread
    extern __shared__ __align__(16) unsigned char smem[];
    float *Bs = reinterpret_cast<float *>(smem);      // [2][8][kFk][kFo]
    float *Fs = Bs + 2 * 8 * kFk * kFo;               // [2][8][kFk][TC]
    const int tid = threadIdx.x, x = tid >> 5, lane = tid & 31;
    const int o0 = blockIdx.y * kFo, c0 = blockIdx.x * TC;
    const int to = (lane >> 2) * 4, tc = (lane & 3) * NC;
    const int steps = (norb + kFk - 1) / kFk;

    float raw[kItems][8];
    auto load_f = [&](int k0) {
#pragma unroll
        for (int q = 0; q < kItems; q++) {
            const int it = tid + q * 256, k = k0 + it / TC, c = c0 + it % TC;
            const bool live = it < kFk * TC && k < norb && c < ncells;
#pragma unroll
            for (int e = 0; e < 8; e++) raw[q][e] = live ? __ldg(f + (size_t)__ldg(row_node + 8 * k + e) * ld + c) : 0.f;
        }
    };
    auto store_f = [&](int buf) {
#pragma unroll
        for (int q = 0; q < kItems; q++) {
            const int it = tid + q * 256;
            if (it >= kFk * TC) continue;
            float *v = raw[q];
#pragma unroll
            for (int b = 1; b < 8; b <<= 1)
#pragma unroll
                for (int e = 0; e < 8; e++)
                    if (!(e & b)) {
                        const float lo = v[e], hi = v[e | b];
                        v[e] = lo + hi;
                        v[e | b] = lo - hi;
                    }
#pragma unroll
            for (int e = 0; e < 8; e++) Fs[((size_t)(buf * 8 + e) * kFk + it / TC) * TC + it % TC] = v[e];
        }
    };
    auto load_b = [&](int k0, int buf) {
        // 8 kFk rows of kFo floats, 16 bytes per copy; opad and o0 are multiples of kFo
        for (int t = tid; t < 8 * kFk * (kFo / 4); t += 256) {
            const int row = t / (kFo / 4), q = t % (kFo / 4) * 4, k = min(k0 + row % kFk, norb - 1);
            const float *src = bx + ((size_t)(row / kFk) * norb + k) * opad + o0 + q;
            const uint32_t dst = (uint32_t)__cvta_generic_to_shared(Bs + ((size_t)buf * 8 * kFk + row) * kFo + q);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    float acc[4][NC], comp[4][NC];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < NC; j++) acc[i][j] = comp[i][j] = 0.f;
    load_b(0, 0);
    load_f(0);
    store_f(0);
    for (int s = 0; s < steps; s++) {
        const int buf = s & 1;
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();  // step s is in shared memory, step s - 1 has been read
        if (s + 1 < steps) {
            load_b((s + 1) * kFk, buf ^ 1);
            load_f((s + 1) * kFk);  // rows past the last orbit read as zero
        }
        const float *B = Bs + (size_t)(buf * 8 + x) * kFk * kFo + to, *F = Fs + (size_t)(buf * 8 + x) * kFk * TC + tc;
        float part[4][NC];
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < NC; j++) part[i][j] = 0.f;
#pragma unroll
        for (int k = 0; k < kFk; k++) {
            const float4 b = *reinterpret_cast<const float4 *>(B + k * kFo);
            const float bv[4] = {b.x, b.y, b.z, b.w};
            float fv[NC];
#pragma unroll
            for (int j = 0; j < NC; j++) fv[j] = F[k * TC + j];
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < NC; j++) part[i][j] = __fmaf_rn(bv[i], fv[j], part[i][j]);
        }
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < NC; j++) {
                const float y = __fsub_rn(part[i][j], comp[i][j]), t = __fadd_rn(acc[i][j], y);
                comp[i][j] = __fsub_rn(__fsub_rn(t, acc[i][j]), y);
                acc[i][j] = t;
            }
        if (s + 1 < steps) store_f(buf ^ 1);
    }
    __syncthreads();
    double *out = reinterpret_cast<double *>(smem);  // [8][kFo][TC]
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < NC; j++)
            out[((size_t)x * kFo + to + i) * TC + tc + j] = (double)acc[i][j] - (double)comp[i][j];
    __syncthreads();
    for (int t = tid; t < kFo * TC; t += 256) {
        const int o = o0 + t / TC, c = c0 + t % TC;
        if (o >= norb || c >= ncells) continue;
        double v[8];
#pragma unroll
        for (int e = 0; e < 8; e++) v[e] = out[(size_t)e * kFo * TC + t];
#pragma unroll
        for (int b = 1; b < 8; b <<= 1)
#pragma unroll
            for (int e = 0; e < 8; e++)
                if (!(e & b)) {
                    const double lo = v[e], hi = v[e | b];
                    v[e] = lo + hi;
                    v[e | b] = lo - hi;
                }
#pragma unroll
        for (int e = 0; e < 8; e++) nu[(size_t)__ldg(row_node + 8 * o + e) * ld + c] = (float)(0.125 * v[e]);
    }
}

// B_x[o'][o] for the eight characters, columns past norb zero.
__global__ void fold_b_kernel(Dims d, int norb, int opad, const int *__restrict__ row_node,
                              const uint32_t *__restrict__ nodes, const float *__restrict__ b, float *__restrict__ bx)
{
    const int64_t total = (int64_t)norb * opad;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
        const int k = (int)(t / opad), o = (int)(t % opad);
        double v[8];
        for (int e = 0; e < 8; e++) {
            v[e] = 0.0;
            if (o >= norb) continue;
            const uint32_t p = nodes[row_node[8 * o]], q = nodes[row_node[8 * k + e]];
            const int dx = abs((int)(p & 1023) - (int)(q & 1023)), dy = abs((int)((p >> 10) & 1023) - (int)((q >> 10) & 1023)),
                      dz = abs((int)(p >> 20) - (int)(q >> 20));
            v[e] = (double)b[dx * d.nyz + dy * d.nz + dz];
        }
        for (int w = 1; w < 8; w <<= 1)
            for (int e = 0; e < 8; e++)
                if (!(e & w)) {
                    const double lo = v[e], hi = v[e | w];
                    v[e] = lo + hi;
                    v[e | w] = lo - hi;
                }
        for (int e = 0; e < 8; e++) bx[(size_t)e * total + t] = (float)v[e];
    }
}

template <int TC>
int launch_folded_loss(Context &c, const float *f, int ncells, int ld, float *nu, cudaStream_t st)
{
    const OrbitGain &g = *c.orbit;
    const size_t smem = folded_smem<TC>();
    GD_CUDA(cudaFuncSetAttribute(folded_loss_kernel<TC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const dim3 grid((ncells + TC - 1) / TC, (g.norb + kFo - 1) / kFo);
    folded_loss_kernel<TC><<<grid, 256, smem, st>>>(f, ld, ncells, g.norb, g.opad, g.row_node, g.bx, nu);
    GD_CUDA(cudaGetLastError());
    return GD_OK;
}

}  // namespace

// The folded loss matrices of a context with orbit rows.
int fold_loss_build(Context &c)
{
    OrbitGain &g = *c.orbit;
    g.opad = (g.norb + kFo - 1) / kFo * kFo;
    GD_CUDA(cudaMalloc(&g.bx, (size_t)8 * g.norb * g.opad * sizeof(float)));
    const int64_t n = (int64_t)g.norb * g.opad;
    fold_b_kernel<<<(unsigned)std::min<int64_t>((n + 255) / 256, (int64_t)c.sm_count * 32), 256>>>(
        c.d, g.norb, g.opad, g.row_node, c.d_nodes, c.d_b, g.bx);
    GD_CUDA(cudaGetLastError());
    return GD_OK;
}

int run_loss(Context &c, const float *f, int ncells, int ld, float *nu, cudaStream_t st)
{
    // 32 cells per CTA, eight where wider tiles would leave most SMs idle
    if (c.orbit) {
        const int wide = (ncells + 31) / 32 * ((c.orbit->norb + kFo - 1) / kFo);
        return wide >= c.sm_count ? launch_folded_loss<32>(c, f, ncells, ld, nu, st)
                                  : launch_folded_loss<8>(c, f, ncells, ld, nu, st);
    }
    const Dims &d = c.d;
    const size_t smem = (((size_t)d.nxyz * 4 + 15) & ~(size_t)15) + (size_t)d.n_pnt * 4;
    GD_CUDA(cudaFuncSetAttribute(loss_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    dim3 grid((ncells + 31) / 32, (d.n_pnt + kWarps * kRows - 1) / (kWarps * kRows));
    loss_kernel<<<grid, kWarps * 32, smem, st>>>(d, f, ld, ncells, c.d_b, c.d_nodes, nu);
    GD_CUDA(cudaGetLastError());
    return GD_OK;
}

}  // namespace gd
