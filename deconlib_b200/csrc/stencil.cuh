// Hessian3D stencil arithmetic shared by the stand-alone operator kernels
// (ops.cu) and the fused PDHG kernels (solvers.cu), so both produce the same
// float32 values.  Neumann boundaries by index clamping, operation order as in
// deconlib's linops_core_mlx.py:25-80 and linops_mlx.py:224-259.
#pragma once

#include "common.cuh"

namespace dk {

__device__ __forceinline__ int64_t clampi(int64_t v, int64_t n) { return v < 0 ? 0 : (v >= n ? n - 1 : v); }

// d2 along one axis (linops_core_mlx.py:66-76): (f[i-1] - 2 f[i]) + f[i+1].
// The stencil arithmetic uses round-to-nearest intrinsics throughout: every
// product and sum is rounded as the reference's float32 array operations
// round it, and no multiply-add is contracted, so every kernel that inlines
// these functions (fused or not) produces the same bits.
__device__ __forceinline__ float d2v(float fm, float f0, float fp) {
    return __fadd_rn(__fsub_rn(fm, __fmul_rn(2.f, f0)), fp);
}
// w * v rounded (a weighted component value)
__device__ __forceinline__ float wmul(float v, float w) { return __fmul_rn(v, w); }
// The element-wise PDHG updates, each operation rounded as the reference's
// float32 arrays round it (pdhg_mlx.py:724, 733, 742, 841):
//   x_bar = x + theta (x - x_prev), dual argument y + sigma K x_bar,
//   x_new = max(0, x - tau g)
__device__ __forceinline__ float xbar_of(float x, float xp, float th) {
    return __fadd_rn(x, __fmul_rn(th, __fsub_rn(x, xp)));
}
__device__ __forceinline__ float dual_arg(float y, float sg, float kx) {
    return __fadd_rn(y, __fmul_rn(sg, kx));
}
__device__ __forceinline__ float primal_of(float x, float tau, float g) {
    return fmaxf(__fsub_rn(x, __fmul_rn(tau, g)), 0.f);
}

struct Dims {
    int64_t nz, ny, nx;
};

// Component weights [r^2, 1, 1, sqrt2 r, sqrt2 r, sqrt2] (linops_mlx.py:237-239;
// SQRT2 is a float32 device scalar there).
inline void hessian_weights(float r, float w[6]) {
    const float s2 = sqrtf(2.f);
    w[0] = (float)((double)r * (double)r);
    w[1] = 1.f;
    w[2] = 1.f;
    w[3] = r * s2;
    w[4] = r * s2;
    w[5] = s2;
}

struct W6 {
    float w[6];
};

// Hessian3D.adjoint of six stored components hw[c * n + i] on the tiled,
// staged walk of the fused PDHG kernels (solvers.cu).
int hess_adjoint_tiled(const float* hw, float* out, const Dims& d, const W6& w, cudaStream_t st);

}  // namespace dk
