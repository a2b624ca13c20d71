// The forward Hessian stencils of PDHG (dual update, ||H dx||^2) with four
// adjacent x voxels per thread, for rows that are 16-byte aligned.
//
// A warp owns a row piece of 128 voxels and walks z; a CTA holds kWideRows rows
// and the two rows around them.  Everything along z and x stays in registers:
// a lane keeps its voxels of planes z - 1, z, z + 1, and x neighbours come by
// shuffle (the row piece's two outer neighbours are loaded by its first and
// last lane).  Only what the rows above and below need goes through shared
// memory, double-buffered, one barrier per plane.
//
// The one-voxel tile walks (pdhg_tiled.cuh) spend 12-20 instructions per voxel
// on addresses, staging and the halo window and are bound by instruction
// issue.  128x256x256: dual update 126 -> 101 us (470 MB, 4.65 TB/s), ||H dx||^2
// 42 -> 33 us; 64x128x128: 16.3 -> 11.6 and 9.1 -> 7.6 us.  The transpose
// (primal update) in the same form needs 130 registers and was slower than the
// tile walk (190 vs 90 us), and rows that are not aligned gained nothing
// consistently (voxels 32 apart: 29.3 vs 29.0 us at 60x150x210).  Float
// operations and their order are those of hess6_smem (pdhg_tiled.cuh): the values are
// the same bits.
#pragma once

#include "solvers.cuh"
#include "stencil.cuh"

namespace dk {

constexpr int kWideRows = 8;
constexpr int kWideThreads = 32 * (kWideRows + 2);

struct WideGeo {
    int nz, ny, nx, ntx, nty, zc;
    int64_t ntiles, n;  // n: voxels
};

constexpr int kWideX = 128;

// Four adjacent voxels of a row piece that starts at x0.
struct Quad {
    float v[4];
};
struct XLane {
    int lane, x0, nx;
    __device__ __forceinline__ int x() const { return x0 + 4 * lane; }
    __device__ __forceinline__ bool on() const { return x() < nx; }
    // the row's voxels, the last one repeated past its end
    __device__ __forceinline__ Quad load(const float* row) const {
        if (on()) {
            const float4 q = __ldg(reinterpret_cast<const float4*>(row + x()));
            return Quad{{q.x, q.y, q.z, q.w}};
        }
        const float e = __ldg(row + nx - 1);
        return Quad{{e, e, e, e}};
    }
    // the outer neighbour that the first and the last lane supply
    __device__ __forceinline__ bool outer() const { return lane == 0 || lane == 31; }
    __device__ __forceinline__ float load_outer(const float* row) const {
        return outer() ? __ldg(row + (lane == 0 ? max(x0 - 1, 0) : min(x0 + kWideX, nx - 1))) : 0.f;
    }
    __device__ __forceinline__ void put(float* s, const Quad& q) const {
        *reinterpret_cast<float4*>(s + 4 * lane) = make_float4(q.v[0], q.v[1], q.v[2], q.v[3]);
    }
    __device__ __forceinline__ Quad get(const float* s) const {
        const float4 q = *reinterpret_cast<const float4*>(s + 4 * lane);
        return Quad{{q.x, q.y, q.z, q.w}};
    }
    // x - 1 and x + 1 of every voxel; o: the value at this lane's outer neighbour
    __device__ __forceinline__ void sides(const Quad& q, float o, Quad& l, Quad& r) const {
        const float a = __shfl_up_sync(0xffffffffu, q.v[3], 1), b = __shfl_down_sync(0xffffffffu, q.v[0], 1);
        l = Quad{{lane == 0 ? o : a, q.v[0], q.v[1], q.v[2]}};
        r = Quad{{q.v[1], q.v[2], q.v[3], lane == 31 ? o : b}};
    }
};

// Row of this warp in a tile.
struct WideTile {
    int z0, z1, y;    // y: the row (may lie outside the volume in the outer rows)
    int64_t row;      // offset of the (clamped) row in a plane
    bool inside;      // an interior row of the volume
};
__device__ __forceinline__ WideTile wide_tile(const WideGeo& g, int64_t tile, XLane& xl) {
    const int wy = threadIdx.x >> 5;
    const int bx = (int)(tile % g.ntx);
    const int64_t r = tile / g.ntx;
    const int by = (int)(r % g.nty), bz = (int)(r / g.nty);
    WideTile t;
    xl.x0 = bx * kWideX;
    t.z0 = bz * g.zc;
    t.z1 = min(t.z0 + g.zc, g.nz);
    t.y = by * kWideRows - 1 + wy;
    t.row = (int64_t)min(max(t.y, 0), g.ny - 1) * g.nx;
    t.inside = wy >= 1 && wy <= kWideRows && t.y < g.ny;
    return t;
}

// H f at every voxel, f = val(a, b) of two fields.  early(i, xl) runs ahead of a
// plane's barrier, body(i, xl, h) after it: i is the offset of the row's x = 0
// in the volume, h[6] the weighted components.  AHEAD: planes that the field
// loads run ahead of their use (1 where the body's own operands take the
// registers, 2 where they are the only loads).
template <int AHEAD, class Val, class Early, class Body>
__device__ __forceinline__ void wide_hess(const WideGeo& g, const W6& w, const float* __restrict__ fa,
                                          const float* __restrict__ fb, const Val& val, const Early& early,
                                          const Body& body) {
    __shared__ __align__(16) float sf[2][kWideRows + 2][kWideX], sh[2][kWideRows + 2][kWideX];
    __shared__ float se[2][kWideRows + 2][2];  // f at the row piece's outer neighbours
    const int wy = threadIdx.x >> 5;
    XLane xl;
    xl.lane = threadIdx.x & 31;
    xl.nx = g.nx;
    const int64_t plane = (int64_t)g.ny * g.nx;
    struct Raw {
        Quad a, b;
        float oa, ob;
    };
    int buf = 0;
    for (int64_t tile = blockIdx.x; tile < g.ntiles; tile += gridDim.x) {
        const WideTile t = wide_tile(g, tile, xl);
        auto fetch = [&](int z) {
            const int64_t i = (int64_t)min(max(z, 0), g.nz - 1) * plane + t.row;
            return Raw{xl.load(fa + i), xl.load(fb + i), xl.load_outer(fa + i), xl.load_outer(fb + i)};
        };
        auto field = [&](const Raw& r, Quad& f, float& o) {
#pragma unroll
            for (int k = 0; k < 4; ++k) f.v[k] = val(r.a.v[k], r.b.v[k]);
            o = val(r.oa, r.ob);
        };
        Quad fm, fc;
        float om, oc;
        field(fetch(t.z0 - 1), fm, om);
        field(fetch(t.z0), fc, oc);
        Raw next[AHEAD];  // planes z + 1 ..
#pragma unroll
        for (int i = 0; i < AHEAD; ++i) next[i] = fetch(t.z0 + 1 + i);
        int64_t zo = (int64_t)t.z0 * plane + t.row;
        for (int z = t.z0; z < t.z1; ++z, zo += plane) {
            if (t.inside) early(zo, xl);
            Quad fp, hz;
            float op;
            field(next[0], fp, op);
#pragma unroll
            for (int i = 0; i + 1 < AHEAD; ++i) next[i] = next[i + 1];
            if (z + AHEAD < t.z1) next[AHEAD - 1] = fetch(z + AHEAD + 1);
#pragma unroll
            for (int k = 0; k < 4; ++k) hz.v[k] = (fp.v[k] - fm.v[k]) / 2.f;
            xl.put(sf[buf][wy], fc);
            xl.put(sh[buf][wy], hz);
            if (xl.outer()) se[buf][wy][xl.lane != 0] = oc;
            __syncthreads();
            if (t.inside) {
                Quad h[6], l, r, dy;
                Quad n = xl.get(sh[buf][wy - 1]), s = xl.get(sh[buf][wy + 1]);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    h[0].v[k] = d2v(fm.v[k], fc.v[k], fp.v[k]) * w.w[0];
                    h[3].v[k] = ((s.v[k] - n.v[k]) / 2.f) * w.w[3];
                }
                xl.sides(hz, (op - om) / 2.f, l, r);
#pragma unroll
                for (int k = 0; k < 4; ++k) h[4].v[k] = ((r.v[k] - l.v[k]) / 2.f) * w.w[4];
                xl.sides(fc, oc, l, r);
#pragma unroll
                for (int k = 0; k < 4; ++k) h[2].v[k] = d2v(l.v[k], fc.v[k], r.v[k]) * w.w[2];
                n = xl.get(sf[buf][wy - 1]);
                s = xl.get(sf[buf][wy + 1]);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    h[1].v[k] = d2v(n.v[k], fc.v[k], s.v[k]) * w.w[1];
                    dy.v[k] = (s.v[k] - n.v[k]) / 2.f;
                }
                const int side = xl.lane != 0;
                xl.sides(dy, (se[buf][wy + 1][side] - se[buf][wy - 1][side]) / 2.f, l, r);
#pragma unroll
                for (int k = 0; k < 4; ++k) h[5].v[k] = ((r.v[k] - l.v[k]) / 2.f) * w.w[5];
                body(zo, xl, h);
            }
            buf ^= 1;
            om = oc;
            oc = op;
            fm = fc;
            fc = fp;
        }
    }
}

// y2 = proj(y2 + sigma H x_bar), x_bar = x + theta (x - x_prev).
template <int NORM>
__global__ void __launch_bounds__(kWideThreads, 2) k_wide_dual(PdhgDev* s, float* y2, const float* __restrict__ xc,
                                                               const float* __restrict__ xp, WideGeo g, W6 w,
                                                               float alpha) {
    chain_enter();
    if (s->stop) return;
    const float sg = (float)s->sigma, th = (float)s->theta;
    const int64_t n = g.n;
    float4 y[6];
    wide_hess<1>(
        g, w, xc, xp, [&](float a, float b) { return xbar_of(a, b, th); },
        [&](int64_t i, const XLane& xl) {
            if (!xl.on()) return;
#pragma unroll
            for (int c = 0; c < 6; ++c) y[c] = *reinterpret_cast<const float4*>(y2 + c * n + i + xl.x());
        },
        [&](int64_t i, const XLane& xl, const Quad (&h)[6]) {
            if (!xl.on()) return;
            if constexpr (NORM == 0) {
#pragma unroll
                for (int c = 0; c < 6; ++c) {
                    float* v = reinterpret_cast<float*>(&y[c]);
#pragma unroll
                    for (int k = 0; k < 4; ++k) v[k] = fminf(fmaxf(dual_arg(v[k], sg, h[c].v[k]), -alpha), alpha);
                }
            } else {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    float ss = 0.f;
#pragma unroll
                    for (int c = 0; c < 6; ++c) {
                        float& v = reinterpret_cast<float*>(&y[c])[k];
                        v = dual_arg(v, sg, h[c].v[k]);
                        ss += v * v;
                    }
                    const float sc = fmaxf(sqrtf(ss + 1e-12f) / alpha, 1.f);
#pragma unroll
                    for (int c = 0; c < 6; ++c) reinterpret_cast<float*>(&y[c])[k] /= sc;
                }
            }
#pragma unroll
            for (int c = 0; c < 6; ++c) *reinterpret_cast<float4*>(y2 + c * n + i + xl.x()) = y[c];
        });
}

// ||H (x_new - x)||^2 and, over m elements, ||A x_new - A x||^2.
__global__ void __launch_bounds__(kWideThreads, 2) k_wide_dk(PdhgDev* s, const float* __restrict__ axn,
                                                             const float* __restrict__ axc, int64_t m,
                                                             const float* __restrict__ xn,
                                                             const float* __restrict__ xc, WideGeo g, W6 w, int slot_a,
                                                             int slot_l) {
    chain_enter();
    if (s->stop) return;
    double a2 = 0.0, l2 = 0.0;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x) {
        const double dd = (double)axn[i] - (double)axc[i];
        a2 += dd * dd;
    }
    wide_hess<2>(
        g, w, xn, xc, [](float a, float b) { return a - b; }, [](int64_t, const XLane&) {},
        [&](int64_t, const XLane& xl, const Quad (&h)[6]) {
            if (!xl.on()) return;
            // the six squares of one voxel in FP32, the sum over voxels in FP64
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                float v = 0.f;
#pragma unroll
                for (int c = 0; c < 6; ++c) v = fmaf(h[c].v[k], h[c].v[k], v);
                l2 += (double)v;
            }
        });
    put_slot(s, slot_a, a2);
    put_slot(s, slot_l, l2);
}

}  // namespace dk
