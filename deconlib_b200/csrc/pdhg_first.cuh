// PDHG with the identity or the gradient regulariser: the regulariser half of an
// iteration as three kernels, L x_bar, L^T y2 and L (x_new - x) formed on the
// fly.
//
// As separate operators an iteration stored and re-read x_bar, its gradient,
// the divergence, x_new - x and its gradient: 8 launches over 31 volumes'
// worth of traffic at one scalar load per step (119 us at 60x210x190, next to
// 110 us of convolutions; now 26 + 17 + 18 us).  Here a thread marches along z
// with its column's next value in a register; y and x neighbours come from L1.
// Bound by load latency: the volumes of such solves stay in L2.  The float
// operations are those of k_xbar, k_gradient_fwd / _adj, k_dual_reg, k_primal
// and k_diffsq_slot, which serve the other regularisers.
#pragma once

#include "solvers.cuh"
#include "stencil.cuh"

namespace dk {

constexpr int kFirstX = 64, kFirstY = 8, kFirstThreads = kFirstX * kFirstY;

struct FirstGeo {
    int nz, ny, nx, ntx, nty, zc;  // zc: planes per march
    int64_t ntiles, n;
};

// f(z, y, x, i) for every voxel, each thread marching along z; start() at the top
// of a column piece.
template <class Start, class Body>
__device__ __forceinline__ void first_walk(const FirstGeo& g, const Start& start, const Body& body) {
    const int tx = threadIdx.x % kFirstX, ty = threadIdx.x / kFirstX;
    const int64_t plane = (int64_t)g.ny * g.nx;
    for (int64_t tile = blockIdx.x; tile < g.ntiles; tile += gridDim.x) {
        const int bx = (int)(tile % g.ntx);
        const int64_t r = tile / g.ntx;
        const int x = bx * kFirstX + tx, y = (int)(r % g.nty) * kFirstY + ty;
        if (x >= g.nx || y >= g.ny) continue;
        const int z0 = (int)(r / g.nty) * g.zc, z1 = min(z0 + g.zc, g.nz);
        int64_t i = (int64_t)z0 * plane + (int64_t)y * g.nx + x;
        start(z0, i);
        // unrolled: the next planes' loads go out before this one's are used
#pragma unroll 4
        for (int z = z0; z < z1; ++z, i += plane) body(z, y, x, i);
    }
}

// y2 = proj(y2 + sigma L x_bar), x_bar = x + theta (x - x_prev).  KIND 0:
// identity (1 component), 1: gradient (r dz, dy, dx).
template <int KIND, int NORM>
__global__ void __launch_bounds__(kFirstThreads) k_first_dual(PdhgDev* s, float* y2, const float* __restrict__ xc,
                                                    const float* __restrict__ xp, FirstGeo g, float r, float alpha) {
    chain_enter();
    if (s->stop) return;
    constexpr int C = KIND == 0 ? 1 : 3;
    const float sg = (float)s->sigma, th = (float)s->theta;
    const int64_t n = g.n, plane = (int64_t)g.ny * g.nx;
    auto bar = [&](int64_t i) { return xbar_of(__ldg(xc + i), __ldg(xp + i), th); };
    float f = 0.f;
    first_walk(
        g, [&](int, int64_t i) { f = bar(i); },
        [&](int z, int y, int x, int64_t i) {
            float v[C];
            if constexpr (KIND == 0) {
                v[0] = dual_arg(y2[i], sg, bar(i));
            } else {
                const float fz = z + 1 < g.nz ? bar(i + plane) : f;
                const float fy = y + 1 < g.ny ? bar(i + g.nx) : f;
                const float fx = x + 1 < g.nx ? bar(i + 1) : f;
                v[0] = dual_arg(y2[i], sg, r * (fz - f));
                v[1] = dual_arg(y2[n + i], sg, fy - f);
                v[2] = dual_arg(y2[2 * n + i], sg, fx - f);
                f = fz;
            }
            if constexpr (NORM == 0) {
#pragma unroll
                for (int c = 0; c < C; ++c) y2[c * n + i] = fminf(fmaxf(v[c], -alpha), alpha);
            } else {
                float ss = 0.f;
#pragma unroll
                for (int c = 0; c < C; ++c) ss += v[c] * v[c];
                const float sc = fmaxf(sqrtf(ss + 1e-12f) / alpha, 1.f);
#pragma unroll
                for (int c = 0; c < C; ++c) y2[c * n + i] = v[c] / sc;
            }
        });
}

// d1_fwd_adj (linops_core_mlx.py:35-39) from the values before and at index i.
__device__ __forceinline__ float first_adj(float before, float here, int i, int n, float sc) {
    if (n == 1 || i == 0) return -(here * sc);
    if (i == n - 1) return before * sc;
    return before * sc - here * sc;
}

// x_new = max(0, x - tau (A^T y1 + L^T y2)) and its FP64 sums.
template <int KIND>
__global__ void __launch_bounds__(kFirstThreads) k_first_primal(PdhgDev* s, const float* __restrict__ xc,
                                                      const float* __restrict__ aty, const float* __restrict__ y2,
                                                      float* __restrict__ xn, FirstGeo g, float r, int s_dx2, int s_xc2,
                                                      int s_xn2) {
    chain_enter();
    if (s->stop) return;
    const float tau = (float)s->tau;
    const int64_t n = g.n, plane = (int64_t)g.ny * g.nx;
    double dx2 = 0.0, xc2 = 0.0, xn2 = 0.0;
    float gz = 0.f;  // the z component one plane before
    first_walk(
        g, [&](int z, int64_t i) { gz = KIND == 1 && z > 0 ? __ldg(y2 + i - plane) : 0.f; },
        [&](int z, int y, int x, int64_t i) {
            float lt;
            if constexpr (KIND == 0) {
                lt = __ldg(y2 + i);
            } else {
                const float hz = __ldg(y2 + i), hy = __ldg(y2 + n + i), hx = __ldg(y2 + 2 * n + i);
                const float gy = y > 0 ? __ldg(y2 + n + i - g.nx) : 0.f;
                const float gx = x > 0 ? __ldg(y2 + 2 * n + i - 1) : 0.f;
                lt = (first_adj(gz, hz, z, g.nz, r) + first_adj(gy, hy, y, g.ny, 1.f)) +
                     first_adj(gx, hx, x, g.nx, 1.f);
                gz = hz;
            }
            const float a = __ldg(xc + i);
            const float v = primal_of(a, tau, __fadd_rn(__ldg(aty + i), lt));
            xn[i] = v;
            const float d = v - a;
            dx2 += (double)d * d;
            xc2 += (double)a * a;
            xn2 += (double)v * v;
        });
    put_slot(s, s_dx2, dx2);
    put_slot(s, s_xc2, xc2);
    put_slot(s, s_xn2, xn2);
}

// ||L (x_new - x)||^2 and ||A x_new - A x||^2 over m elements.
template <int KIND>
__global__ void __launch_bounds__(kFirstThreads) k_first_dk(PdhgDev* s, const float* __restrict__ axn,
                                                  const float* __restrict__ axc, int64_t m,
                                                  const float* __restrict__ xn, const float* __restrict__ xc,
                                                  FirstGeo g, float r, int slot_a, int slot_l) {
    chain_enter();
    if (s->stop) return;
    double a2 = 0.0, l2 = 0.0;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
#pragma unroll 4
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += stride) {
        const double d = (double)__ldg(axn + i) - (double)__ldg(axc + i);
        a2 += d * d;
    }
    const int64_t plane = (int64_t)g.ny * g.nx;
    auto diff = [&](int64_t i) { return __ldg(xn + i) - __ldg(xc + i); };
    float f = 0.f;
    first_walk(
        g, [&](int, int64_t i) { f = diff(i); },
        [&](int z, int y, int x, int64_t i) {
            if constexpr (KIND == 0) {
                const double d = (double)diff(i);
                l2 += d * d;
            } else {
                const float fz = z + 1 < g.nz ? diff(i + plane) : f;
                const float fy = y + 1 < g.ny ? diff(i + g.nx) : f;
                const float fx = x + 1 < g.nx ? diff(i + 1) : f;
                const double a = (double)(r * (fz - f)), b = (double)(fy - f), c = (double)(fx - f);
                l2 += a * a;
                l2 += b * b;
                l2 += c * c;
                f = fz;
            }
        });
    put_slot(s, slot_a, a2);
    put_slot(s, slot_l, l2);
}

}  // namespace dk
