// The two FFT passes of the widefield PSF (psf.cu): the register kernels of the
// 5-smooth lengths up to 1024 and the runtime-radix ones of the others.
#pragma once

#include "codelets.cuh"
#include "conv_impl.cuh"

namespace dk {

struct PsfArgs {
    const float2* pupil;
    const double* kz;
    const double* z;       // this chunk's first plane
    float2* a;             // scratch [plane][y][place of the column], rows of nx
    float* psf;            // this chunk's first plane
    const int *act, *pos, *nact;  // columns in use, each column's place or -1, their number
    int nx, ny, ntiles, T;  // T: lines per CTA of the pass
    FastDiv fd_L;           // nx
    int64_t nrows;
    Axis ax;               // axis of the pass
    const double* energy;  // sum |P|^2 (normalize) or nullptr
    double norm_div;       // nz ny nx (normalize)
    float fixed_scale;     // 1 / (ny nx)^2 (no normalisation)
};
struct PsfKernel {
    void* fn = nullptr;
    int T = 0, nt = 0;
    size_t smem = 0;
};
PsfKernel psf_group_a(int L, bool cols);
PsfKernel psf_group_b(int L, bool cols);
PsfKernel psf_group_c(int L, bool cols);
PsfKernel psf_group_d(int L, bool cols);
PsfKernel psf_group_e(int L, bool cols);
PsfKernel psf_any_kernel(const Axis& ax, bool cols);

// Pupil value p with the defocus phase of one plane; a zero of the pupil stays
// zero whatever its (finite) phase.
__device__ __forceinline__ float2 defocused(const PsfArgs& a, int64_t p, double zz) {
    const float2 v = __ldg(a.pupil + p);
    const double turns = 2.0 * __ldg(a.kz + p) * zz;
    if (v.x == 0.f && v.y == 0.f && isfinite(turns)) return make_float2(0.f, 0.f);
    double sn, cs;
    sincospi(turns, &sn, &cs);
    return make_float2((float)((double)v.x * cs - (double)v.y * sn), (float)((double)v.x * sn + (double)v.y * cs));
}

__device__ __forceinline__ float psf_scale(const PsfArgs& a) {
    if (!a.energy) return a.fixed_scale;
    const double tot = a.norm_div * *a.energy;
    return tot > 0.0 ? (float)(1.0 / tot) : 1.f;
}

// ---- register kernels: L = R1 x R2 -------------------------------------------

template <int L>
struct PsfShape {
    static constexpr int R1 = small_radix(L), R2 = L / R1;
    static constexpr int TC = R2 < 18 ? 16 : 8;  // columns per CTA of pass 1
    static constexpr int NTC = TC * R2;
    static constexpr int step1 = R1 | 1;          // odd step between exchange rows
    static constexpr int TR = 16 * R2 <= 256 ? 16 : 8;  // rows per CTA of pass 2
    static constexpr int NTR = (TR * R2 + 31) / 32 * 32;
    static constexpr int pitch = R2 * step1;
};

// Pass 1: TC columns in use of one plane.  Thread (t, j): points j + r R2 of
// column t -> radix R1 -> exchange -> radix R2 -> points j + r R1.
template <int L>
__global__ void __launch_bounds__(PsfShape<L>::NTC) k_psf_cols(const __grid_constant__ PsfArgs a) {
    using H = PsfShape<L>;
    constexpr int R1 = H::R1, R2 = H::R2, T = H::TC;
    extern __shared__ float2 ex[];
    const int tid = threadIdx.x, t = tid % T, j = tid / T;
    const int o = blockIdx.x / a.ntiles, c0 = (blockIdx.x - o * a.ntiles) * T;
    const int n = *a.nact;
    if (c0 >= n) return;
    const bool ok = c0 + t < n;
    const int x = ok ? a.act[c0 + t] : 0;
    C1 v[R2];
    if (j < R2) {
        const double zz = a.z[o];
#pragma unroll
        for (int r = 0; r < R1; ++r)
            v[r] = ok ? as_c1(defocused(a, (int64_t)(j + r * R2) * a.nx + x, zz)) : C1{0.f, 0.f};
        dftn<R1, +1>(v);
#pragma unroll
        for (int r = 0; r < R1; ++r) ex[(j * H::step1 + r) * T + t] = as_f2(v[r]);
    }
    __syncthreads();
    if (j < R1) {
#pragma unroll
        for (int r = 0; r < R2; ++r) {
            v[r] = as_c1(ex[(j + r * H::step1) * T + t]);
            if (r > 0) v[r] = twist<true>(v[r], __ldg(&a.ax.tw[r * j]));
        }
        dftn<R2, +1>(v);
        if (ok) {
            float2* dst = a.a + ((int64_t)o * a.ny + j) * a.nx + c0 + t;
#pragma unroll
            for (int r = 0; r < R2; ++r) dst[(int64_t)(r * R1) * a.nx] = as_f2(v[r]);
        }
    }
}

// Pass 2: TR rows; inverse FFT along x, |.|^2 * scale.
template <int L>
__global__ void __launch_bounds__(PsfShape<L>::NTR) k_psf_rows(const __grid_constant__ PsfArgs a) {
    using H = PsfShape<L>;
    constexpr int R1 = H::R1, R2 = H::R2, T = H::TR;
    extern __shared__ float2 sm[];
    const int tid = threadIdx.x;
    const int64_t row0 = (int64_t)blockIdx.x * T;
    {
        const int l = tid / R2, j = tid - l * R2;
        if (l < T) {
            const bool ok = row0 + l < a.nrows;
            const float2* src = a.a + (row0 + l) * L;
            C1 v[R1];
#pragma unroll
            for (int r = 0; r < R1; ++r) {
                const int p = __ldg(a.pos + j + r * R2);
                v[r] = ok && p >= 0 ? as_c1(__ldg(src + p)) : C1{0.f, 0.f};
            }
            dftn<R1, +1>(v);
#pragma unroll
            for (int r = 0; r < R1; ++r) sm[l * H::pitch + j * H::step1 + r] = as_f2(v[r]);
        }
    }
    __syncthreads();
    const int l = tid / R1, j = tid - l * R1;
    if (l >= T || row0 + l >= a.nrows) return;
    C1 v[R2];
#pragma unroll
    for (int r = 0; r < R2; ++r) {
        v[r] = as_c1(sm[l * H::pitch + j + r * H::step1]);
        if (r > 0) v[r] = twist<true>(v[r], __ldg(&a.ax.tw[r * j]));
    }
    dftn<R2, +1>(v);
    const float scale = psf_scale(a);
    float* dst = a.psf + (row0 + l) * L + j;
#pragma unroll
    for (int r = 0; r < R2; ++r) dst[r * R1] = (v[r].re * v[r].re + v[r].im * v[r].im) * scale;
}

template <int L>
PsfKernel psf_kernel(bool cols) {
    using H = PsfShape<L>;
    return cols ? PsfKernel{(void*)k_psf_cols<L>, H::TC, H::NTC, (size_t)H::TC * H::pitch * sizeof(float2)}
                : PsfKernel{(void*)k_psf_rows<L>, H::TR, H::NTR, (size_t)H::TR * H::pitch * sizeof(float2)};
}

}  // namespace dk
