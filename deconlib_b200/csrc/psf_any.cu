// Widefield PSF passes of any 7-smooth length on the runtime-radix engine.
#include <algorithm>

#include "psf_passes.cuh"

namespace dk {

// Pass 1: one CTA = T columns in use of one plane.
__global__ void __launch_bounds__(kDynThreads, 1) k_psf_cols_any(const __grid_constant__ PsfArgs a) {
    extern __shared__ float2 sm[];
    const int L = a.ax.L, T = a.T, tid = threadIdx.x;
    const int64_t o = blockIdx.x / a.ntiles;
    const int c0 = (int)(blockIdx.x - o * a.ntiles) * T;
    const int n = *a.nact;
    if (c0 >= n) return;
    const double zz = a.z[o];
    const int lg = 31 - __clz(T);
    for (int q = tid; q < L * T; q += blockDim.x) {
        const int j = q >> lg, t = q & (T - 1);
        float2 v = make_float2(0.f, 0.f);
        if (c0 + t < n) v = defocused(a, (int64_t)j * a.nx + a.act[c0 + t], zz);
        sm[phys(j, t, T)] = v;
    }
    __syncthreads();
    fft_lines<+1>(sm, T, tid % T, tid / T, a.ax);
    float2* dst = a.a + o * a.ny * a.nx + c0;
    for (int q = tid; q < L * T; q += blockDim.x) {
        const int j = q >> lg, t = q & (T - 1);
        if (c0 + t < n) dst[(int64_t)j * a.nx + t] = sm[phys(j, t, T)];
    }
}

// Pass 2: one CTA = T contiguous rows; inverse FFT along x, |.|^2 * scale.
__global__ void __launch_bounds__(kDynThreads, 1) k_psf_rows_any(const __grid_constant__ PsfArgs a) {
    extern __shared__ float2 sm[];
    const int L = a.ax.L, T = a.T, tid = threadIdx.x;
    const int64_t row0 = (int64_t)blockIdx.x * T;
    const int64_t left = a.nrows - row0;
    const int nr = left < T ? (int)left : T;
    const float2* src = a.a + row0 * L;
    for (int q = tid; q < T * L; q += blockDim.x) {
        const int t = fdiv(q, a.fd_L), j = q - t * L;
        const int p = a.pos[j];
        sm[phys(j, t, T)] = t < nr && p >= 0 ? src[(int64_t)t * L + p] : make_float2(0.f, 0.f);
    }
    __syncthreads();
    fft_lines<+1>(sm, T, tid % T, tid / T, a.ax);
    const float scale = psf_scale(a);
    float* dst = a.psf + row0 * L;
    for (int q = tid; q < nr * L; q += blockDim.x) {
        const int t = fdiv(q, a.fd_L), j = q - t * L;
        const float2 v = sm[phys(j, t, T)];
        dst[q] = (v.x * v.x + v.y * v.y) * scale;
    }
}

PsfKernel psf_any_kernel(const Axis& ax, bool cols) {
    const int T = fft_lines_per_cta(ax, 32);
    return PsfKernel{cols ? (void*)k_psf_cols_any : (void*)k_psf_rows_any, T,
                     std::max(64, (int)round_up((int64_t)T * ax.tpl, 32)), (size_t)T * ax.L * sizeof(float2)};
}

}  // namespace dk
