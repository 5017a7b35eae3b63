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
// orbit_loss_kernel serves the lattices with orbit rows (gd_orbit.cu): b is
// invariant under the lattice's reflections, so with nodes (o, e) (orbit, octant)
//   nu(o, e) = sum_o' sum_x b_x[o][o'] f(o', e ^ x),  b_x[o][o'] = b((o, 0), (o', x)):
// eight values of b and eight of f make 64 products, and b of a pair of orbits is
// read from a table of an eighth of the size, without indexing it by node
// differences.  Every term is the product b f of its own partner: the sum is as close
// for a node whose frequency is small beside its mirrors' as for any other, exactly
// zero where only the node itself is filled, and never negative.  (With f and b
// folded by the group's characters the products are an eighth, 0.64 ms instead of
// 2.46 at 20^3 / 4096 cells, but the differences of mirrors that they end in leave an
// error of the largest mirror's size: 1e-6 of a small frequency, and negative ones.)
// loss_kernel (lane = cell, kRows outputs per warp, b and the node coordinates
// in shared memory) serves the other lattices.  20^3: 4096 cells 22.1 -> 2.46 ms,
// one cell 0.89 -> 0.016 ms.
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

// CTA = 4 TO orbits x 8 cells.  The partner orbits o' are shared out to the eight
// warps in contiguous eighths; a thread holds TO orbits of a cell.  A warp takes kPk
// orbits o' per step: their f and b are copied to its own shared memory by cp.async,
// for the next step while the current ones are multiplied.  The 8 kPk products of a
// step are a chain; the chains, then the warps' sums, are added with compensation,
// all in an order that is the lattice's alone, so a cell's bits are the same in any
// batch.  Bound by instruction issue (85 % of the slots; two thirds are the products
// and compensated sums).  16 orbits x 8 cells 2.46 ms (20^3, 4096 cells), 8 x 16 2.77,
// 8 x 8 2.56, 16 x 16 2.52; pairs of FP32 operations in one instruction: no change.
constexpr int kPk = 4;
constexpr int kLossCells = 8;

template <int TO>
constexpr uint32_t loss_stage()  // floats of a warp's stage: f [kPk][2][cell][4], b [kPk][2][4 TO][4]
{
    return kPk * 8 * (kLossCells + 4 * TO);
}
template <int TO>
constexpr size_t loss_smem()
{
    const size_t stages = (size_t)8 * 2 * loss_stage<TO>() * sizeof(float), out = (size_t)8 * 32 * TO * 8 * sizeof(float2);
    return stages > out ? stages : out;
}

// s - c is the sum of x into s - c (Kahan).
__device__ __forceinline__ void add_comp(float &s, float &c, float x)
{
    const float y = __fsub_rn(x, c), t = __fadd_rn(s, y);
    c = __fsub_rn(__fsub_rn(t, s), y);
    s = t;
}

template <int TO>
__global__ void __launch_bounds__(256, 2) orbit_loss_kernel(const float *__restrict__ f, int ld, int ncells, int norb, int opad,
                                                            const int *__restrict__ row_node,
                                                            const float4 *__restrict__ bx,  // [o'][2][opad]
                                                            float *__restrict__ nu)
{
    constexpr int NO = 4 * TO, NC = kLossCells;
    extern __shared__ __align__(16) unsigned char smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int o0 = blockIdx.y * NO, c0 = blockIdx.x * NC;
    const int to = lane >> 3, tc = lane & 7;  // orbits to + 4 i, cell tc
    const int k0 = norb * warp / 8, k1 = norb * (warp + 1) / 8;
    float *stage = reinterpret_cast<float *>(smem) + (size_t)warp * 2 * loss_stage<TO>();
    const uint32_t at = (uint32_t)__cvta_generic_to_shared(stage);

    // lane: cell lane % NC of the tile, every 32 / NC-th row (o', e)
    constexpr int kRowsPer = 32 / NC;
    const int cell = c0 + lane % NC, row = lane / NC;
    const bool live = cell < ncells;
    const float *fc = f + (live ? cell : 0);
    const uint32_t fdst = at + (row / 4 * NC * 4 + lane % NC * 4 + row % 4) * 4;
    const float4 *bc = bx + o0 + lane % NO;  // row lane / NO, and so on
    auto load = [&](int k, int buf) {
        const uint32_t fs = fdst + buf * loss_stage<TO>() * 4, bs = at + (buf * loss_stage<TO>() + kPk * 8 * NC) * 4 + lane * 16;
        const int node = __ldg(row_node + min(8 * k + lane, 8 * norb - 1));  // of (o', e) = lane
#pragma unroll
        for (int i = 0; i < kPk * 8 / kRowsPer; i++) {
            const int m = __shfl_sync(0xffffffffu, node, i * kRowsPer + row);
            const int size = live && k + i * kRowsPer / 8 < k1 ? 4 : 0;  // rows past the warp's: zeros
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(fs + (i * kRowsPer / 4 * NC * 4 + i * kRowsPer % 4) * 4),
                         "l"(fc + (int64_t)m * ld), "r"(size)
                         : "memory");
        }
#pragma unroll
        for (int i = 0; i < (kPk * 2 * NO + 31) / 32; i++)
            if (kPk * 2 * NO % 32 == 0 || i * 32 + lane < kPk * 2 * NO)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(bs + i * 512),
                             "l"(bc + (int64_t)min(2 * k + i * (32 / NO) + lane / NO, 2 * norb - 1) * opad)
                             : "memory");
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    float acc[TO][8], comp[TO][8];
#pragma unroll
    for (int i = 0; i < TO; i++)
#pragma unroll
        for (int e = 0; e < 8; e++) acc[i][e] = comp[i][e] = 0.f;
    if (k0 < k1) load(k0, 0);
    for (int k = k0, buf = 0; k < k1; k += kPk, buf ^= 1) {
        if (k + kPk < k1) {
            load(k + kPk, buf ^ 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncwarp();
        const float4 *F = reinterpret_cast<const float4 *>(stage + buf * loss_stage<TO>()), *B = F + kPk * 2 * NC;
        float part[TO][8];
#pragma unroll
        for (int i = 0; i < TO; i++)
#pragma unroll
            for (int e = 0; e < 8; e++) part[i][e] = 0.f;
#pragma unroll 1
        for (int q = 0; q < kPk; q++) {
            const float4 f0 = F[2 * q * kLossCells + tc], f1 = F[(2 * q + 1) * kLossCells + tc];
            const float fv[8] = {f0.x, f0.y, f0.z, f0.w, f1.x, f1.y, f1.z, f1.w};
#pragma unroll
            for (int i = 0; i < TO; i++) {
                const float4 b0 = B[2 * q * NO + to + 4 * i], b1 = B[(2 * q + 1) * NO + to + 4 * i];
                const float bv[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
                for (int x = 0; x < 8; x++)
#pragma unroll
                    for (int e = 0; e < 8; e++) part[i][e] = __fmaf_rn(bv[x], fv[e ^ x], part[i][e]);
            }
        }
#pragma unroll
        for (int i = 0; i < TO; i++)
#pragma unroll
            for (int e = 0; e < 8; e++) add_comp(acc[i][e], comp[i][e], part[i][e]);
        __syncwarp();  // the stage is read
    }
    __syncthreads();
    float2 *out = reinterpret_cast<float2 *>(smem);  // [warp][octant][orbit][cell]
#pragma unroll
    for (int i = 0; i < TO; i++)
#pragma unroll
        for (int e = 0; e < 8; e++)
                out[((warp * 8 + e) * NO + to + 4 * i) * NC + tc] = make_float2(acc[i][e], comp[i][e]);
    __syncthreads();
    for (int t = threadIdx.x; t < 8 * NO * NC; t += 256) {
        const int c = c0 + t % NC, o = o0 + t / NC % NO, e = t / (NC * NO);
        if (o >= norb || c >= ncells) continue;
        float s = 0.f, rest = 0.f;
#pragma unroll
        for (int w = 0; w < 8; w++) {
            const float2 v = out[w * 8 * NO * NC + t];
            add_comp(s, rest, v.x);
            rest += v.y;
        }
        nu[(size_t)__ldg(row_node + 8 * o + e) * ld + c] = __fsub_rn(s, rest);
    }
}

// b of orbits o' and o: [o'][half][o][4], x = 4 half + 0..3, columns past norb zero.
__global__ void orbit_b_kernel(Dims d, int norb, int opad, const int *__restrict__ row_node,
                               const uint32_t *__restrict__ nodes, const float *__restrict__ b, float4 *__restrict__ bx)
{
    const int64_t total = (int64_t)norb * 2 * opad;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
        const int k = (int)(t / (2 * opad)), h = (int)(t / opad) & 1, o = (int)(t % opad);
        float v[4] = {0.f, 0.f, 0.f, 0.f};
        for (int x = 0; x < 4 && o < norb; x++) {
            const uint32_t p = nodes[row_node[8 * o]], q = nodes[row_node[8 * k + 4 * h + x]];
            const int dx = abs((int)(p & 1023) - (int)(q & 1023)), dy = abs((int)((p >> 10) & 1023) - (int)((q >> 10) & 1023)),
                      dz = abs((int)(p >> 20) - (int)(q >> 20));
            v[x] = b[dx * d.nyz + dy * d.nz + dz];
        }
        bx[t] = make_float4(v[0], v[1], v[2], v[3]);
    }
}

constexpr int kLossPad = 16;  // orbits of the wider tile

template <int TO>
int launch_orbit_loss(Context &c, const float *f, int ncells, int ld, float *nu, cudaStream_t st)
{
    const OrbitGain &g = *c.orbit;
    const size_t smem = loss_smem<TO>();
    GD_CUDA(cudaFuncSetAttribute(orbit_loss_kernel<TO>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const dim3 grid((ncells + kLossCells - 1) / kLossCells, (g.norb + 4 * TO - 1) / (4 * TO));
    orbit_loss_kernel<TO><<<grid, 256, smem, st>>>(f, ld, ncells, g.norb, g.opad, g.row_node, g.bx, nu);
    GD_CUDA(cudaGetLastError());
    return GD_OK;
}

}  // namespace

// The table of b by orbits of a context with orbit rows.
int orbit_loss_build(Context &c)
{
    OrbitGain &g = *c.orbit;
    g.opad = (g.norb + kLossPad - 1) / kLossPad * kLossPad;
    const int64_t n = (int64_t)g.norb * 2 * g.opad;
    GD_CUDA(cudaMalloc(&g.bx, (size_t)n * sizeof(float4)));
    orbit_b_kernel<<<(unsigned)std::min<int64_t>((n + 255) / 256, (int64_t)c.sm_count * 32), 256>>>(
        c.d, g.norb, g.opad, g.row_node, c.d_nodes, c.d_b, g.bx);
    GD_CUDA(cudaGetLastError());
    return GD_OK;
}

int run_loss(Context &c, const float *f, int ncells, int ld, float *nu, cudaStream_t st)
{
    // 16 orbits per CTA, 4 where the wider tiles would not fill the chip twice
    if (c.orbit) {
        const int64_t wide = (int64_t)((ncells + kLossCells - 1) / kLossCells) * ((c.orbit->norb + 15) / 16);
        return wide >= 4 * c.sm_count ? launch_orbit_loss<4>(c, f, ncells, ld, nu, st)
                                      : launch_orbit_loss<1>(c, f, ncells, ld, nu, st);
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
