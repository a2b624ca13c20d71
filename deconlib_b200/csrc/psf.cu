// Widefield PSF synthesis on the device: PSF(z) = |IFFT2(P(kx, ky) e^{2 pi i kz z})|^2.
//
// Replaces the NumPy loop of deconlib's pupil_to_psf (psf/widefield.py:18-73)
// with two FFT passes per chunk of z planes (psf_passes.cuh):
//
//   pass 1: defocus P(ky, kx) e^{2 pi i kz z} on load (phase in FP64 with
//     sincospi; pupil and kz are re-read per plane from L2), inverse FFT along
//     y over tiles of columns, complex columns written to scratch;
//   pass 2: inverse FFT along x over rows, intensity |.|^2 times the final
//     scale, written straight into the PSF.
//
// A pupil is zero outside the aperture, a disc that covers 4 % of the plane
// and 23 % of its columns at the sampling of a 2x refined grid, and a zero
// column stays zero under the defocus: k_psf_support lists the columns that
// hold anything, pass 1 transforms those only (packed side by side in the
// scratch) and pass 2 takes the others as zeros.  128x256x256 at 0.0425 um,
// NA 1.4: passes 83 + 67 us without the list and on the shared-memory engine.
// The unit-sum normalisation needs no pass over the PSF: |e^{i phi}| = 1, so by
// Parseval every plane's unnormalised intensity sums to ny nx sum|P|^2, and
// the total is nz ny nx sum|P|^2, an FP64 reduction over the pupil alone.
// numpy's ifft2 divides by ny nx; without normalisation the PSF carries that
// factor squared.
#include <algorithm>
#include <cmath>
#include <map>
#include <mutex>
#include <vector>

#include "psf_passes.cuh"

namespace dk {

// Complex scratch per chunk of planes: at most this many voxels (256 MB), or
// one plane when a plane is larger.
constexpr int64_t kPsfChunkVoxels = int64_t(1) << 25;

// Per column x: flags[x] = 1 if the column of the pupil holds a non-zero (or
// its phase may not be finite: |kz| > 1e100), and the block's share of sum |P|^2
// in FP64.  32 columns per CTA; blockIdx.y: a part of the rows, with flags of its
// own (with all rows in one CTA, 64 CTAs of a 2048x2048 pupil read it alone).
__global__ void k_psf_support(const float2* __restrict__ pupil, const double* __restrict__ kz, int ny, int nx,
                              int* __restrict__ flags, double* __restrict__ partials) {
    __shared__ int any[32];
    if (threadIdx.y == 0) any[threadIdx.x] = 0;
    __syncthreads();
    const int x = blockIdx.x * 32 + threadIdx.x;
    double acc = 0.0;
    bool on = false;
    if (x < nx) {
#pragma unroll 4
        for (int y = blockIdx.y * blockDim.y + threadIdx.y; y < ny; y += gridDim.y * blockDim.y) {
            const int64_t p = (int64_t)y * nx + x;
            const float2 v = pupil[p];
            acc += (double)v.x * v.x + (double)v.y * v.y;
            on = on || !(v.x == 0.f && v.y == 0.f) || !(fabs(kz[p]) <= 1e100);
        }
    }
    if (on) any[threadIdx.x] = 1;
    // block_sum numbers threads by threadIdx.x: fold the rows first
    __shared__ double part[32][33];
    part[threadIdx.y][threadIdx.x] = acc;
    __syncthreads();
    if (threadIdx.y == 0) {
        if (x < nx) flags[(int64_t)blockIdx.y * nx + x] = any[threadIdx.x];
        double t = 0.0;
        for (int i = 0; i < 32; ++i) t += part[i][threadIdx.x];
        for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
        if (threadIdx.x == 0) partials[blockIdx.y * gridDim.x + blockIdx.x] = t;
    }
}

// One CTA: the columns in use as a list (act) and each column's place in it
// (pos, -1 for a zero column), and the energy.  Every column is in use when a
// z is not finite or huge.
__global__ void __launch_bounds__(1024) k_psf_scan(const int* __restrict__ flags, int nx, int nflags, const double* __restrict__ z,
                                                   int64_t nz, const double* __restrict__ partials, int nparts,
                                                   int* __restrict__ act, int* __restrict__ pos, int* __restrict__ nact,
                                                   double* __restrict__ energy) {
    __shared__ int warp_base[32];
    __shared__ int base, all;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    if (tid == 0) base = all = 0;
    __syncthreads();
    for (int64_t i = tid; i < nz; i += blockDim.x)
        if (!(fabs(z[i]) <= 1e100)) all = 1;
    __syncthreads();
    for (int x0 = 0; x0 < nx; x0 += blockDim.x) {
        const int x = x0 + tid;
        int f = all;
        if (x < nx)
            for (int i = 0; i < nflags; ++i) f |= flags[(int64_t)i * nx + x];
        const bool on = x < nx && f;
        const unsigned m = __ballot_sync(0xffffffffu, on);
        if (lane == 0) warp_base[w] = __popc(m);
        __syncthreads();
        if (tid == 0) {
            int t = base;
            for (int i = 0; i < (int)(blockDim.x >> 5); ++i) {
                const int c = warp_base[i];
                warp_base[i] = t;
                t += c;
            }
            base = t;
        }
        __syncthreads();
        const int at = warp_base[w] + __popc(m & ((1u << lane) - 1));
        if (x < nx) pos[x] = on ? at : -1;
        if (on) act[at] = x;
        __syncthreads();
    }
    if (tid == 0) *nact = base;
    if (w == 0) {
        double t = 0.0;
        for (int i = lane; i < nparts; i += 32) t += partials[i];
        for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
        if (lane == 0) *energy = t;
    }
}

static PsfKernel pick(const Axis& ax, bool cols) {
    for (auto group : {psf_group_a, psf_group_b, psf_group_c, psf_group_d, psf_group_e}) {
        const PsfKernel k = group(ax.L, cols);
        if (k.fn) return k;
    }
    return psf_any_kernel(ax, cols);
}

static int launch_args(void* fn, int64_t nblk, int nthr, size_t smem, cudaStream_t st, void* args) {
    DK_TRY(kernel_prepare(fn, smem, nthr, nullptr));
    if (nblk > 0x7fffffffLL) return fail(DECON_ERR_UNSUPPORTED, "decon_pupil_to_psf: grid too large");
    void* params[] = {args};
    DK_CUDA(cudaLaunchKernel(fn, dim3((unsigned)nblk), dim3(nthr), params, smem, st));
    count_launch();
    return DECON_OK;
}

}  // namespace dk

using namespace dk;

extern "C" int decon_pupil_to_psf(const float* pupil, const double* kz, const double* z, int64_t nz,
                                  int64_t ny, int64_t nx, int normalize, float* psf, void* stream) {
    if (nz < 1 || ny < 1 || nx < 1) return fail(DECON_ERR_VALUE, "decon_pupil_to_psf: empty shape");
    if (!pupil || !kz || !z || !psf) return fail(DECON_ERR_NULL, "decon_pupil_to_psf: null pointer");
    if (ny > kSmemElems || nx > kSmemElems)
        return fail(DECON_ERR_UNSUPPORTED, "decon_pupil_to_psf: planes larger than %d points per axis",
                    kSmemElems);
    Axis axx, axy;
    if (!plan_axis((int)nx, axx) || !plan_axis((int)ny, axy))
        return fail(DECON_ERR_UNSUPPORTED,
                    "decon_pupil_to_psf: pupil shape (%lld, %lld) must factor into 2, 3, 5 and 7",
                    (long long)ny, (long long)nx);
    const cudaStream_t st = as_stream(stream);
    const int64_t nyx = ny * nx;
    const int64_t chunk = std::max<int64_t>(1, std::min<int64_t>(nz, kPsfChunkVoxels / nyx));
    const float2 *twx = nullptr, *twy = nullptr;
    DK_TRY(twiddle_table((int)nx, &twx));
    DK_TRY(twiddle_table((int)ny, &twy));
    axx.tw = twx;
    axy.tw = twy;
    axx.tws = axy.tws = 1;
    cudaMemPool_t pool;
    DK_TRY(device_pool(&pool));
    // scratch: complex chunk, then energy, partials, and the column lists
    // two rows or more per thread of the support search, and no more than two CTAs per SM
    const int64_t gx = cdiv(nx, 32);
    const int gy = (int)std::max<int64_t>(1, std::min(cdiv(ny, 64), 2 * sm_count() / gx));
    const int nparts = (int)gx * gy;
    const size_t chunk_bytes = (size_t)round_up(chunk * nyx * (int64_t)sizeof(float2), 256);
    const size_t bytes = chunk_bytes + (1 + nparts) * sizeof(double) + ((gy + 2) * nx + 1) * sizeof(int);
    char* buf = nullptr;
    auto run = [&]() -> int {
        DK_CUDA(cudaMallocFromPoolAsync((void**)&buf, bytes, pool, st));
        PsfArgs a{};
        a.pupil = reinterpret_cast<const float2*>(pupil);
        a.kz = kz;
        a.a = reinterpret_cast<float2*>(buf);
        double* energy = reinterpret_cast<double*>(buf + chunk_bytes);
        double* partials = energy + 1;
        int* flags = reinterpret_cast<int*>(partials + nparts);
        int *act = flags + gy * nx, *pos = act + nx, *nact = pos + nx;
        k_psf_support<<<dim3((unsigned)gx, (unsigned)gy), dim3(32, 32), 0, st>>>(a.pupil, kz, (int)ny, (int)nx, flags, partials);
        DK_LAUNCHED();
        k_psf_scan<<<1, 1024, 0, st>>>(flags, (int)nx, gy, z, nz, partials, nparts, act, pos, nact, energy);
        DK_LAUNCHED();
        const double inv_n = 1.0 / ((double)nx * (double)ny);
        a.energy = normalize ? energy : nullptr;
        a.norm_div = (double)nz * (double)nyx;
        a.fixed_scale = (float)(inv_n * inv_n);
        a.act = act;
        a.pos = pos;
        a.nact = nact;
        a.nx = (int)nx;
        a.ny = (int)ny;
        a.fd_L = make_fastdiv(nx);
        const PsfKernel kc = pick(axy, true), kr = pick(axx, false);
        for (int64_t z0 = 0; z0 < nz; z0 += chunk) {
            const int64_t nzc = std::min(chunk, nz - z0);
            a.z = z + z0;
            a.psf = psf + z0 * nyx;
            a.nrows = nzc * ny;
            a.ax = axy;
            a.T = kc.T;
            a.ntiles = (int)cdiv(nx, kc.T);
            DK_TRY(launch_args(kc.fn, nzc * a.ntiles, kc.nt, kc.smem, st, &a));
            a.ax = axx;
            a.T = kr.T;
            DK_TRY(launch_args(kr.fn, cdiv(a.nrows, kr.T), kr.nt, kr.smem, st, &a));
        }
        return DECON_OK;
    };
    const int status = run();
    if (buf) cudaFreeAsync(buf, st);
    return status;
}
