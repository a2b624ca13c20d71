// Linear FFT convolution on the B200: pruned 3D R2C / C2R FFTs with the OTF
// product fused into the axial pass.
//
// Replaces deconlib's LinearFFTConvolver (deconvolution/linops_mlx.py:435-533)
// and FFTConvolver (:384-432).  With signal N = (Nz, Ny, Nx) zero-padded to
// the canvas F = (Fz, Fy, Fx), a convolution is five passes:
//
//   1. X R2C   N rows of x            -> S1[Nz][Ny][P]   (real FFT, length Fx)
//   2. Y FFT   S1, Ny non-zero points -> S2[Nz][Fy][P]
//   3. Z pass  S2 in place: FFT over Fz (Nz non-zero inputs), x OTF (or
//              conj(OTF) for the adjoint), inverse FFT, keep the first Nz
//   4. Y IFFT  S2 -> S1, keep the first Ny points
//   5. X C2R   S1 -> out, keep x < Nx, scale 1/(Fz Fy Fx), fused epilogue
//
// On a canvas of one plane passes 2 to 4 are one, in S1, and there is no S2.
//
// Zero padding never exists in memory (the loads return zeros) and only the
// Nz x Fy x (Fx/2+1) part of the spectrum that the crop can see is ever
// formed ("pruned" FFT).  P is the spectrum row pitch: Fx/2 + 1 rounded up to
// 16 complex values, so every 16-wide column tile of the strided passes
// reads whole 128-byte lines.
#include <cmath>
#include <map>
#include <mutex>
#include <tuple>
#include <vector>

#include <algorithm>

#include "conv_impl.cuh"
#include "tma.cuh"
namespace dk {

// Raised when a bounded mbarrier wait gives up (read by decon_device_status,
// cleared by decon_device_status_clear); such a CTA skips its compute and store.
static __device__ int g_wait_timeout = 0;

}  // namespace dk

#include "yzpass.cuh"

namespace dk {

// ---------------------------------------------------------------------------
// host: axis planning and launches
// ---------------------------------------------------------------------------

bool plan_axis(int L, Axis& ax, int order) {
    ax = Axis{};
    ax.L = L;
    int n = L, e2 = 0;
    while (n % 2 == 0) {
        n /= 2;
        ++e2;
    }
    std::vector<int> r;
    int n8 = e2 / 3, rem = e2 % 3;
    if (rem == 1 && n8 > 0) {
        --n8;
        r.push_back(4);
        r.push_back(4);
    } else if (rem == 1) {
        r.push_back(2);
    } else if (rem == 2) {
        r.push_back(4);
    }
    for (int i = 0; i < n8; ++i) r.insert(r.begin(), 8);
    std::vector<int> odd;
    for (int p : {5, 3, 7}) {
        while (n % p == 0) {
            n /= p;
            odd.push_back(p);
        }
    }
    if (order == 1) r.insert(r.begin(), odd.begin(), odd.end());
    else r.insert(r.end(), odd.begin(), odd.end());
    if (n != 1 || (int)r.size() > kMaxStages) return false;
    ax.nst = (int)r.size();
    for (int i = 0; i < ax.nst; ++i) ax.rad |= (unsigned long long)r[i] << (4 * i);
    ax.tpl = (L + kDynPPT - 1) / kDynPPT;
    return true;
}

static int threads_for(int T, const Axis& ax) {
    int n = T * ax.tpl;
    n = (int)round_up(n, 32);
    return std::max(n, 64);
}

// Kernel-class timing (decon_profile_start / _stop): CUDA events recorded
// on the launching stream around every launch of the selected classes.
struct ProfState {
    int mask = 0;
    std::vector<std::pair<cudaEvent_t, cudaEvent_t>> ev;
    size_t used = 0;
};
static ProfState g_prof;

// Per (device, kernel, dynamic shared memory, block size): the occupancy is
// queried once; per (device, kernel) the shared-memory opt-in only ever rises
// to the largest size launched so far (a launch with less shared memory must
// not lower it under another plan's larger launches).  Later launches,
// including launches recorded into a CUDA graph, only look the entries up.
int kernel_prepare(void* fn, size_t smem, int nthr, int* per_sm) {
    static std::mutex mu;
    static std::map<std::tuple<int, void*, size_t, int>, int> done;
    static std::map<std::pair<int, void*>, size_t> opt_in;
    int dev = 0;
    DK_CUDA(cudaGetDevice(&dev));
    const auto key = std::make_tuple(dev, fn, smem, nthr);
    std::lock_guard<std::mutex> lock(mu);
    auto it = done.find(key);
    if (it != done.end()) {
        if (per_sm) *per_sm = it->second;
        return DECON_OK;
    }
    // the 48 KB default covers static plus dynamic shared memory: opt in
    // whenever their sum exceeds it
    cudaFuncAttributes fa{};
    DK_CUDA(cudaFuncGetAttributes(&fa, fn));
    if (smem + fa.sharedSizeBytes > 48 * 1024) {
        size_t& cur = opt_in[std::make_pair(dev, fn)];
        if (smem > cur) {
            DK_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
            cur = smem;
        }
    }
    int occ = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, nthr, smem) != cudaSuccess) {
        cudaGetLastError();
        occ = 0;
    }
    done[key] = occ;
    if (per_sm) *per_sm = occ;
    return DECON_OK;
}

// Dynamic shared memory that needs no opt-in, whatever the kernel's static part
// (at most a few hundred bytes in the FFT passes; the default limit is 48 KB).
constexpr size_t kNoOptIn = 44 * 1024;

// Launches an FFT pass as a chained kernel.  prepared: its shared memory is
// already opted in (a plan's column passes), or needs no opt-in.
static int launch_chained(void* fn, dim3 grid, int nthr, size_t smem, bool prepared, cudaStream_t st, void* args,
                          int cls) {
    if (!prepared && smem > kNoOptIn) DK_TRY(kernel_prepare(fn, smem, nthr, nullptr));
    void* params[] = {args};
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(nthr);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    chain_attribute(&cfg, at);
    const bool prof = (g_prof.mask & cls) != 0;
    if (prof) {
        if (g_prof.used == g_prof.ev.size()) {
            cudaEvent_t a, b;
            DK_CUDA(cudaEventCreate(&a));
            DK_CUDA(cudaEventCreate(&b));
            g_prof.ev.emplace_back(a, b);
        }
        DK_CUDA(cudaEventRecord(g_prof.ev[g_prof.used].first, st));
    }
    DK_CUDA(cudaLaunchKernelExC(&cfg, fn, params));
    count_launch();
    if (prof) {
        DK_CUDA(cudaEventRecord(g_prof.ev[g_prof.used].second, st));
        ++g_prof.used;
    }
    return DECON_OK;
}

static int launch(void* fn, int64_t nblk, int nthr, size_t smem, cudaStream_t st, void* args, int cls) {
    if (nblk <= 0) return kernel_prepare(fn, smem, nthr, nullptr);
    if (nblk > 0x7fffffffLL) return fail(DECON_ERR_UNSUPPORTED, "grid too large");
    return launch_chained(fn, dim3((unsigned)nblk), nthr, smem, false, st, args, cls);
}

}  // namespace dk

extern "C" int decon_device_status(void* stream) {
    using namespace dk;
    DK_CUDA(cudaStreamSynchronize(as_stream(stream)));
    int flag = 0;
    DK_CUDA(cudaMemcpyFromSymbol(&flag, g_wait_timeout, sizeof(int)));
    if (flag) return fail(DECON_ERR_TIMEOUT, "a bounded TMA wait gave up; results are invalid");
    return DECON_OK;
}

extern "C" int decon_device_status_clear(void* stream) {
    using namespace dk;
    DK_CUDA(cudaStreamSynchronize(as_stream(stream)));
    const int zero = 0;
    DK_CUDA(cudaMemcpyToSymbol(g_wait_timeout, &zero, sizeof(int)));
    return DECON_OK;
}

namespace dk {

// One CTA waits, through the kernels' own bounded wait, on an mbarrier that
// no thread arrives at and no copy completes: every poll fails, the wait
// gives up after `polls` polls, raises g_wait_timeout and the CTA returns.
// Nothing is in flight and nothing is written but the flag.
__global__ void k_wait_probe(unsigned polls) {
    __shared__ uint64_t bar;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        fence_proxy_async_smem();
    }
    __syncthreads();
    if (threadIdx.x == 0) (void)mbar_wait_bounded(&bar, 0, &g_wait_timeout, polls);
}

// One CTA starts a copy of n values into shared memory, gives its wait up at once
// and drains, as the column passes do; then hands on what has arrived.
constexpr int kDrainProbe = 8192;
__global__ void k_drain_probe(const float* __restrict__ src, float* __restrict__ dst, int n) {
    __shared__ __align__(128) float buf[kDrainProbe];
    __shared__ uint64_t bar;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        fence_proxy_async_smem();
    }
    for (int i = threadIdx.x; i < n; i += blockDim.x) buf[i] = 0.f;
    fence_proxy_async_smem();
    __syncthreads();
    if (threadIdx.x == 0) {
        mbar_expect_tx(&bar, (uint32_t)n * 4u);
        bulk_load(buf, src, (uint32_t)n * 4u, &bar);
        if (!mbar_wait_bounded(&bar, 0, &g_wait_timeout, 0)) mbar_drain(&bar, 0);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += blockDim.x) dst[i] = buf[i];
}

}  // namespace dk

extern "C" int decon_test_wait_timeout(unsigned polls, void* stream) {
    using namespace dk;
    if (polls == 0 || polls > (1u << 16))
        return fail(DECON_ERR_VALUE, "decon_test_wait_timeout: polls must be in [1, 65536]");
    k_wait_probe<<<1, 32, 0, as_stream(stream)>>>(polls);
    DK_LAUNCHED();
    return DECON_OK;
}

extern "C" int decon_test_wait_drain(const float* src, float* dst, int n, void* stream) {
    using namespace dk;
    if (!src || !dst) return fail(DECON_ERR_NULL, "null pointer");
    if (n < 4 || n > kDrainProbe || n % 4 != 0 || (reinterpret_cast<uintptr_t>(src) & 15) != 0)
        return fail(DECON_ERR_VALUE, "decon_test_wait_drain: n must be a multiple of 4 up to %d, src 16-byte aligned",
                    kDrainProbe);
    k_drain_probe<<<1, 128, 0, as_stream(stream)>>>(src, dst, n);
    DK_LAUNCHED();
    return DECON_OK;
}

extern "C" int decon_profile_start(int class_mask) {
    dk::g_prof.mask = class_mask;
    dk::g_prof.used = 0;
    return DECON_OK;
}

extern "C" int decon_profile_stop(double* ms_total, int64_t* launches) {
    using namespace dk;
    double tot = 0.0;
    for (size_t i = 0; i < g_prof.used; ++i) {
        DK_CUDA(cudaEventSynchronize(g_prof.ev[i].second));
        float ms = 0.f;
        DK_CUDA(cudaEventElapsedTime(&ms, g_prof.ev[i].first, g_prof.ev[i].second));
        tot += ms;
    }
    if (ms_total) *ms_total = tot;
    if (launches) *launches = (int64_t)g_prof.used;
    g_prof.mask = 0;
    g_prof.used = 0;
    return DECON_OK;
}

namespace dk {

#define DK_XREG_PICK(kind) \
    static XRegKernel pick_xreg_##kind(int L, bool odd, bool kx, int what) { \
        if (kx) return odd ? XRegKernel{} : xreg_##kind##_kx(L, what); \
        if (odd) return xreg_##kind##_odd(L, what); \
        for (auto group : {xreg_##kind##_a, xreg_##kind##_b, xreg_##kind##_c, xreg_##kind##_d, xreg_##kind##_e, \
                           xreg_##kind##_f, xreg_##kind##_g}) { \
            const XRegKernel k = group(L, what); \
            if (k.fn) return k; \
        } \
        return XRegKernel{}; \
    }
DK_XREG_PICK(r2c)
DK_XREG_PICK(c2r)
#undef DK_XREG_PICK

static bool is_full_window(const ConvPlan& p, const Win3& w) {
    return w.oz == 0 && w.oy == 0 && w.ox == 0 && w.wz == p.N[0] && w.wy == p.N[1] && w.wx == p.N[2];
}

static bool pair_aligned(const void* q) { return (reinterpret_cast<uintptr_t>(q) & 7) == 0; }

// The fields both register X passes share.
static XRegArgs xreg_args(const ConvPlan& p, int64_t nrows, int64_t Ny, int64_t Nx, const Win3& w, bool full) {
    XRegArgs a{};
    a.win = full ? 0 : 1;
    a.z0 = full ? 0 : (int)w.oz;
    a.y0 = full ? 0 : (int)w.oy;
    a.x0 = full ? 0 : (int)w.ox;
    a.wz = full ? (int)(nrows / Ny) : (int)w.wz;
    a.wy = full ? (int)Ny : (int)w.wy;
    a.wx = full ? (int)Nx : (int)w.wx;
    const int L = p.ax_x.L;
    a.Ny = Ny;
    a.Nx = Nx;
    a.P = p.P;
    a.nrows = (uint32_t)nrows;
    a.nlines = (uint32_t)(p.odd ? cdiv(nrows, 2) : nrows);
    a.nin = a.nout = (int)std::min<int64_t>(p.odd ? Nx : cdiv(Nx, 2), L);
    a.Hx = (int)p.Hx;
    a.tw = p.ax_x.tw;
    a.tws = p.ax_x.tws;
    a.twx = p.twx;
    return a;
}

int launch_xr2c(const ConvPlan& p, int pro, const float* in, Win3 win, float cval, float bg,
                int64_t nz_rows, float2* out, cudaStream_t st, int64_t kstride) {
    const int src = pro == PRO_KERNEL ? 2 : pro == PRO_UP2 ? 1 : 0;
    const bool full = pro == PRO_KERNEL || pro == PRO_UP2 || is_full_window(p, win);
    const XRegKernel k = full || pro == PRO_ARRAY ? pick_xreg_r2c(p.ax_x.L, p.odd, kstride != 0, src) : XRegKernel{};
    if (k.fn) {
        const int64_t Ny = pro == PRO_KERNEL ? p.F[1] : p.N[1], Nx = pro == PRO_KERNEL ? p.F[2] : p.N[2];
        XRegArgs a = xreg_args(p, nz_rows * Ny, Ny, Nx, win, full);
        a.pro = pro;
        a.in = in;
        a.cval = cval;
        a.bg = bg;
        a.ksum = p.ksum;
        a.Nz = nz_rows;
        a.Kz = p.K[0];
        a.Ky = p.K[1];
        a.Kx = p.K[2];
        a.pz = (p.K[0] + 1) / 2;
        a.py = (p.K[1] + 1) / 2;
        a.px = (p.K[2] + 1) / 2;
        a.out = out;
        if (kstride) a.P = kstride;
        a.vec = a.wx % 2 == 0 && a.x0 % 2 == 0 && pair_aligned(in);
        return launch(k.fn, cdiv(a.nlines, k.TL), k.nt, k.smem, st, &a, PROF_XR2C);
    }
    XR2CArgs a{};
    a.kstride = kstride;
    a.in = in;
    a.cval = cval;
    a.bg = bg;
    a.Nz = nz_rows;
    a.Ny = pro == PRO_KERNEL ? p.F[1] : p.N[1];
    a.Nx = pro == PRO_KERNEL ? p.F[2] : p.N[2];
    a.win = win;
    a.Kz = p.K[0];
    a.Ky = p.K[1];
    a.Kx = p.K[2];
    a.pz = (p.K[0] + 1) / 2;
    a.py = (p.K[1] + 1) / 2;
    a.px = (p.K[2] + 1) / 2;
    a.ksum = p.ksum;
    a.out = out;
    a.P = p.P;
    a.Hx = (int)p.Hx;
    a.odd = p.odd;
    a.ax = p.ax_x;
    a.twx = p.twx;
    a.vec4 = pro == PRO_ARRAY && in != nullptr && !p.odd && (a.Nx % 4) == 0 && win.oz == 0 &&
             win.oy == 0 && win.ox == 0 && win.wz == p.N[0] && win.wy == p.N[1] &&
             win.wx == p.N[2] && (reinterpret_cast<uintptr_t>(in) & 15) == 0;
    // the 2x adjoint prologue reads coarse rows of Nx / 2 floats as float4
    const bool up2_vec = pro == PRO_UP2 && (a.Nx % 8) == 0 && (reinterpret_cast<uintptr_t>(in) & 15) == 0;
    if (pro == PRO_UP2) a.vec4 = up2_vec;
    a.T = p.T_x;
    a.nrows = nz_rows * a.Ny;
    {
        const int L = a.ax.L;
        const int64_t nin = p.odd ? std::min<int64_t>(a.Nx, L) : std::min<int64_t>((a.Nx + 1) / 2, L);
        a.fd_q4 = make_fastdiv(std::max<int64_t>(1, pro == PRO_UP2 ? a.Nx / 8 : a.Nx / 4));
        a.fd_H = make_fastdiv(a.Hx);
        a.fd_nin = make_fastdiv(std::max<int64_t>(1, nin));
        a.fd_np = make_fastdiv(L / 2 + 1);
    }
    const int nthr = threads_for(a.T, a.ax);
    const int64_t nblk = cdiv(a.nrows, a.T);
    const size_t smem = (size_t)a.T * a.ax.L * sizeof(float2);
    void* fn = pick_xr2c_kernel(pro);
    if (!fn) return fail(DECON_ERR_VALUE, "bad prologue %d", pro);
    return launch(fn, nblk, nthr, smem, st, &a, PROF_XR2C);
}

int launch_col(const ConvPlan& p, const Axis& ax, int T, int mode, const float2* src,
               int64_t src_os, int64_t src_js, int nin, float2* dst, int64_t dst_os,
               int64_t dst_js, int nout, int64_t nouter, cudaStream_t st) {
    ColArgs a{};
    a.src = src;
    a.dst = dst;
    a.src_os = src_os;
    a.src_js = src_js;
    a.dst_os = dst_os;
    a.dst_js = dst_js;
    a.nin = nin;
    a.nout = nout;
    a.ncols = (int)p.Hx;
    a.T = T;
    a.ax = ax;
    a.mode = mode;
    a.otf = p.otf;
    a.otf_js = p.F[1] * p.P;
    a.otf_os = p.P;
    a.ntiles = (int)cdiv(p.Hx, T);
    const int nthr = threads_for(T, ax);
    const int64_t nblk = nouter * a.ntiles;
    const size_t smem = (size_t)T * ax.L * sizeof(float2);
    return launch(pick_colfft_kernel(), nblk, nthr, smem, st, &a,
                  (mode == COL_OTF || mode == COL_OTF_CONJ) ? PROF_ZOTF : PROF_COL);
}

// A pass that sums writes one partial per CTA.
static int check_partials(const ConvPlan& p, const double* partials, int64_t nblk) {
    if (partials && nblk > p.npartials) return fail(DECON_ERR_VALUE, "X pass: partials buffer too small");
    return DECON_OK;
}

int launch_xc2r(const ConvPlan& p, int epi, const float2* in, Win3 win, float* out,
                const float* aux0, const float* aux1, float bg, double* partials, int* nblk_out,
                cudaStream_t st) {
    const bool full = is_full_window(p, win);
    const int64_t kstride = use_yz(p) ? p.N[0] * p.N[1] : 0;
    const XRegKernel k = full || epi == EPI_STORE ? pick_xreg_c2r(p.ax_x.L, p.odd, kstride != 0, epi) : XRegKernel{};
    if (k.fn) {
        if (epi == EPI_DOWN2 && (p.odd || (p.N[0] | p.N[1] | p.N[2]) & 1))
            return fail(DECON_ERR_UNSUPPORTED, "2x area-sum epilogue: extents must be even");
        // odd Fx: rows are transformed in the pairs of the whole field, so that a
        // window has its bits; pairs outside are skipped
        const int64_t rows = full || p.odd ? p.N[0] * p.N[1] : win.wz * win.wy;
        XRegArgs a = xreg_args(p, rows, p.N[1], p.N[2], win, full);
        a.spec = in;
        if (kstride) a.P = kstride;
        a.out_real = out;
        a.aux0 = aux0;
        a.aux1 = aux1;
        a.bg = bg;
        a.pred = epi == EPI_PRED;
        a.partials = partials;
        a.scale = (float)(1.0 / ((double)p.F[0] * (double)p.F[1] * (double)p.F[2]));
        a.vec = a.wx % 2 == 0 && a.x0 % 2 == 0 && pair_aligned(out) && pair_aligned(aux0) && pair_aligned(aux1);
        const int64_t nblk = cdiv(a.nlines, k.TL);
        DK_TRY(check_partials(p, partials, nblk));
        if (nblk_out) *nblk_out = (int)nblk;
        return launch(k.fn, nblk, k.nt, k.smem, st, &a, PROF_XC2R);
    }
    XC2RArgs a{};
    a.in = in;
    a.P = p.P;
    a.Ny = p.N[1];
    a.Nx = p.N[2];
    a.nrows = p.N[0] * p.N[1];
    a.Hx = (int)p.Hx;
    a.odd = p.odd;
    a.ax = p.ax_x;
    a.twx = p.twx;
    {
        const bool full = win.oz == 0 && win.oy == 0 && win.ox == 0 && win.wz == p.N[0] &&
                          win.wy == p.N[1] && win.wx == p.N[2];
        auto al = [](const void* q) { return q == nullptr || (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
        a.vec4 = full && !p.odd && (p.N[2] % 4) == 0 && al(out) && al(aux0) && al(aux1);
    }
    a.T = p.T_x;
    a.scale = (float)(1.0 / ((double)p.F[0] * (double)p.F[1] * (double)p.F[2]));
    a.win = win;
    a.out = out;
    a.aux0 = aux0;
    a.aux1 = aux1;
    a.bg = bg;
    a.partials = partials;
    a.kstride = kstride;
    {
        const int L = a.ax.L;
        a.fd_L = make_fastdiv(L);
        a.fd_h2 = make_fastdiv(std::max(1, L / 2));
        a.fd_npair = make_fastdiv(L / 2 + 1);
        a.fd_q4 = make_fastdiv(std::max<int64_t>(1, epi == EPI_DOWN2 ? a.Nx / 2 : a.Nx / 4));
        a.fd_Nx = make_fastdiv(a.Nx);
    }
    if (epi == EPI_DOWN2) {
        // whole 2 x 2 x 2 blocks per CTA: T / 2 lines from each of two planes
        a.vec4 = 0;
        if (p.odd || (p.N[0] | p.N[1] | p.N[2]) & 1 || a.T < 4 || p.N[1] % (a.T / 2) != 0)
            return fail(DECON_ERR_UNSUPPORTED, "2x area-sum epilogue: extents must be even and Ny a "
                                               "multiple of %d", a.T / 2);
    }
    const int nthr = threads_for(a.T, a.ax);
    const int64_t nblk = cdiv(a.nrows, a.T);
    DK_TRY(check_partials(p, partials, nblk));
    if (nblk_out) *nblk_out = (int)nblk;
    const size_t smem = (size_t)a.T * a.ax.L * sizeof(float2);
    void* fn = pick_xc2r_kernel(epi);
    if (!fn) return fail(DECON_ERR_VALUE, "bad epilogue %d", epi);
    return launch(fn, nblk, nthr, smem, st, &a, PROF_XC2R);
}

// Found once, by the first thread that asks; the others wait for it.
static PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
    static const PFN_cuTensorMapEncodeTiled_v12000 enc = [] {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess) {
            cudaGetLastError();
            fn = nullptr;
        }
        return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
    }();
    return enc;
}

bool encode_tile_map(CUtensorMap* map, const void* base, int esize, int64_t pitch, int64_t d1, int64_t d2,
                     int T, int b1, int b2) {
    const PFN_cuTensorMapEncodeTiled_v12000 enc = tensor_map_encoder();
    if (!enc) return false;
    const int f = esize / 4;  // 4-byte map elements per complex value
    cuuint64_t dims[3] = {(cuuint64_t)(f * pitch), (cuuint64_t)d1, (cuuint64_t)d2};
    cuuint64_t strides[2] = {(cuuint64_t)(pitch * esize), (cuuint64_t)(pitch * esize * d1)};
    cuuint32_t box[3] = {(cuuint32_t)(f * T), (cuuint32_t)b1, (cuuint32_t)b2};
    cuuint32_t estr[3] = {1u, 1u, 1u};
    CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<void*>(base), dims, strides, box,
                     estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS;
}

// ---------------------------------------------------------------------------
// register column passes (colreg.cuh)
// ---------------------------------------------------------------------------

// DECON_NO_TMA / DECON_SCHED_NO_TMA: plain loads (and the FP32 OTF for a mixed plan).
static bool no_tma(const ConvPlan& p) { return !p.tma || (p.sched & DECON_SCHED_NO_TMA) != 0; }

// DECON_NO_PIPE / DECON_SCHED_NO_PIPE: the FP32 OTF also for a mixed plan.
static bool no_pipe(const ConvPlan& p) {
    return getenv("DECON_NO_PIPE") != nullptr || (p.sched & DECON_SCHED_NO_PIPE) != 0;
}

static ColRegKernel pick_colreg(int L, int mode, bool plain) {
    for (auto group : {colreg_group_a, colreg_group_b, colreg_group_c, colreg_group_d, colreg_group_e}) {
        const ColRegKernel k = group(L, mode, plain);
        if (k.fn) return k;
    }
    return ColRegKernel{};
}

// Boxes of at most 256 rows covering n rows, each a multiple of 128 bytes (the
// shared-memory alignment of a TMA box); rows past the buffer read as zero.
static void split_rows(int n, int row_bytes, int* box, int* nbox) {
    *nbox = (n + 255) / 256;
    const int even = 128 / std::min(128, row_bytes);
    *box = (int)round_up(cdiv(n, *nbox), even);
}

// A column pass along dimension jdim (1: rows adjacent in a plane, 2: planes)
// of src [s2][s1][P] into dst with the same dimension order.
static bool make_col_pass(const ConvPlan& p, ColPass& c, const Axis& ax, int mode, int jdim,
                          const float2* src, int64_t s1, int64_t s2, int nin, float2* dst, int64_t d1,
                          int nout, int64_t nouter) {
    c.ok = c.maps = false;
    c.k = pick_colreg(ax.L, mode, false);
    if (!c.k.fn) return false;
    ColRegArgs& a = c.a;
    memset(&a, 0, sizeof(a));
    const int T = c.k.T;
    a.src = src;
    a.dst = dst;
    a.src_os = jdim == 1 ? s1 * p.P : p.P;
    a.src_js = jdim == 1 ? p.P : s1 * p.P;
    a.dst_os = jdim == 1 ? d1 * p.P : p.P;
    a.dst_js = jdim == 1 ? p.P : d1 * p.P;
    a.nin = nin;
    a.nout = nout;
    a.nouter = (int)nouter;
    a.jdim = jdim;
    a.tw = ax.tw;
    a.tws = ax.tws;
    a.conj = 1.f;
    a.nfull = (int)(p.Hx / T);
    a.rem = (int)(p.Hx - (int64_t)a.nfull * T);
    a.per = a.rem ? T / a.rem : 1;
    split_rows(nin, T * 8, &a.box, &a.nbox);
    a.in_bytes = a.nbox * a.box * T * 8;
    bool maps = !no_tma(p) && encode_tile_map(&a.srcmap, src, 8, p.P, s1, s2, T, jdim == 1 ? a.box : 1,
                                              jdim == 1 ? 1 : a.box);
    c.smem = c.k.exch + a.in_bytes;
    if (mode == 2 || mode == 3) {
        const int esize = mode == 3 ? 4 : 8;
        a.otf = p.otf;
        a.otf16 = p.otf16;
        a.otf_inv = p.otf_inv;
        a.otf_os = jdim == 1 ? p.F[1] * p.P : p.P;
        a.otf_js = jdim == 1 ? p.P : p.F[1] * p.P;
        split_rows(ax.L, T * esize, &a.obox, &a.onbox);
        maps = maps && encode_tile_map(&a.otfmap, mode == 3 ? (const void*)p.otf16 : (const void*)p.otf, esize,
                                       p.P, p.F[1], p.F[0], T, jdim == 1 ? a.obox : 1, jdim == 1 ? 1 : a.obox);
        c.smem += a.onbox * a.obox * T * esize;
    }
    int64_t nmain = nouter * a.nfull, ntiles = nmain + (a.rem ? cdiv(nouter, a.per) : 0);
    if (!maps) {
        if (mode == 3) return false;
        c.k = pick_colreg(ax.L, mode, true);
        a.nfull = (int)cdiv(p.Hx, T);
        a.rem = (int)p.Hx;
        nmain = 0;
        ntiles = nouter * a.nfull;
    }
    if (ntiles > 0x7fffffffLL - 65536) return false;
    a.nmain = (int)nmain;
    a.ntiles = (int)ntiles;
    void* flag = nullptr;
    int per_sm = 0;
    if (c.smem > 227 * 1024 || cudaGetSymbolAddress(&flag, g_wait_timeout) != cudaSuccess ||
        kernel_prepare(c.k.fn, c.smem, c.k.nt, &per_sm) != DECON_OK || per_sm < 1) {
        cudaGetLastError();
        return false;
    }
    a.flag = static_cast<int*>(flag);
    c.grid = (int)std::min<int64_t>(ntiles, (int64_t)sm_count() * per_sm);
    c.maps = maps;
    return c.ok = true;
}

// No axial transform for one plane: three launches per convolution instead of
// five (forward + adjoint of a 512x640 frame: 59.0 -> 39.6 us), and no S2.
bool make_one_plane_pass(ConvPlan& p) {
    const int64_t Ny = p.N[1];
    return p.F[0] == 1 && make_col_pass(p, p.y_otf, p.ax_y, 2, 1, p.s1, Ny, 1, (int)Ny, p.s1, Ny, (int)Ny, 1);
}

void make_col_passes(ConvPlan& p) {
    const int64_t Nz = p.N[0], Ny = p.N[1], Fy = p.F[1];
    if (make_one_plane_pass(p) || !p.s2) return;
    make_col_pass(p, p.y_fwd, p.ax_y, 0, 1, p.s1, Ny, Nz, (int)Ny, p.s2, Fy, (int)Fy, Nz);
    make_col_pass(p, p.z_otf, p.ax_z, 2, 2, p.s2, Fy, Nz, (int)Nz, p.s2, Fy, (int)Nz, Fy);
    make_col_pass(p, p.y_inv, p.ax_y, 1, 1, p.s2, Fy, Nz, (int)Fy, p.s1, Ny, (int)Ny, Nz);
}

void make_z_otf16(ConvPlan& p) {
    const int64_t Nz = p.N[0], Fy = p.F[1];
    make_col_pass(p, p.z_otf16, p.ax_z, 3, 2, p.s2, Fy, Nz, (int)Nz, p.s2, Fy, (int)Nz, Fy);
}

static int launch_col_pass(const ColPass& c, bool conj, cudaStream_t st) {
    ColRegArgs a = c.a;
    if (conj) a.conj = -1.f;
    return launch_chained(c.k.fn, dim3((unsigned)c.grid), c.k.nt, c.smem, true, st, &a, a.otf ? PROF_ZOTF : PROF_COL);
}

int transform_otf(const ConvPlan& p, int axis, cudaStream_t st) {
    const int64_t Fz = p.F[0], Fy = p.F[1], P = p.P;
    const int n = (int)p.F[axis];
    const Axis& ax = axis == 1 ? p.ax_y : p.ax_z;
    ColPass c;
    if (make_col_pass(p, c, ax, 0, axis == 1 ? 1 : 2, p.otf, Fy, Fz, n, p.otf, Fy, n, axis == 1 ? Fz : Fy))
        return launch_col_pass(c, false, st);
    if (axis == 1)
        return launch_col(p, ax, p.T_y, COL_FWD, p.otf, Fy * P, P, n, p.otf, Fy * P, P, n, Fz, st);
    return launch_col(p, ax, p.T_z, COL_FWD, p.otf, P, Fy * P, n, p.otf, P, Fy * P, n, Fy, st);
}

bool zpass_pipelined(const ConvPlan& p) {
    if (!p.z_otf.maps || no_pipe(p)) return false;
    const int L = p.ax_z.L;
    return L == 64 || L == 256 || (L == 128 && p.N[0] <= 64);
}

// ---------------------------------------------------------------------------
// fused Y / axial pass (yzpass.cuh)
// ---------------------------------------------------------------------------

bool yz_supported(const int64_t N[3], const int64_t F[3]) {
    const bool fy = F[1] == 256 || F[1] == 512, fz = F[0] == 128 || F[0] == 256;
    return fy && fz && N[1] <= F[1] / 2 && N[0] <= F[0] / 2 && N[1] % 2 == 0 && N[0] >= 1 &&
           N[1] >= 2;
}

bool use_yz(const ConvPlan& p) {
    // opt-in: the plan's schedule asks for it, or DECON_YZ=1 for every plan
    // (on the B200 the fused pass measured slower than the separate passes:
    // it is instruction-bound, 15 eight-CTA clusters occupy 120 of 148 SMs)
    const bool want = (p.sched & DECON_SCHED_FUSED) || getenv("DECON_YZ") != nullptr;
    return want && p.otft != nullptr && p.precision == 0 && getenv("DECON_NO_YZ") == nullptr;
}

// out[(kx * Fy + ky) * Fz + kz] = otf[(kz * Fy + ky) * P + kx]: 32 x 32 tiles
// of (kz, kx) per ky through shared memory.
__global__ void k_otf_kmajor(const float2* __restrict__ otf, int Fz, int Fy, int64_t P, int Hx,
                             float2* __restrict__ out) {
    __shared__ float2 t[32][33];
    const int ky = blockIdx.z;
    const int kx0 = blockIdx.x * 32, kz0 = blockIdx.y * 32;
    for (int i = threadIdx.y; i < 32; i += blockDim.y) {
        const int kz = kz0 + i, kx = kx0 + threadIdx.x;
        if (kz < Fz && kx < Hx) t[i][threadIdx.x] = otf[((int64_t)kz * Fy + ky) * P + kx];
    }
    __syncthreads();
    for (int i = threadIdx.y; i < 32; i += blockDim.y) {
        const int kx = kx0 + i, kz = kz0 + threadIdx.x;
        if (kz < Fz && kx < Hx) out[((int64_t)kx * Fy + ky) * Fz + kz] = t[threadIdx.x][i];
    }
}

int build_otf_kmajor(const ConvPlan& p, cudaStream_t st) {
    if (!p.otft) return DECON_OK;
    const dim3 grid((unsigned)cdiv(p.Hx, 32), (unsigned)cdiv(p.F[0], 32), (unsigned)p.F[1]);
    k_otf_kmajor<<<grid, dim3(32, 8), 0, st>>>(p.otf, (int)p.F[0], (int)p.F[1], p.P, (int)p.Hx, p.otft);
    DK_LAUNCHED();
    return DECON_OK;
}

template <int FY, int FZ, int C, int NT>
static void* pick_yz_fz(bool adjoint) {
    return adjoint ? (void*)k_yz<FY, FZ, COL_OTF_CONJ, C, NT> : (void*)k_yz<FY, FZ, COL_OTF, C, NT>;
}

template <int C, int NT>
static void* pick_yz_c(int64_t Fy, int64_t Fz, bool adjoint) {
    if (Fy == 512 && Fz == 256) return pick_yz_fz<512, 256, C, NT>(adjoint);
    if (Fy == 512 && Fz == 128) return pick_yz_fz<512, 128, C, NT>(adjoint);
    if (Fy == 256 && Fz == 256) return pick_yz_fz<256, 256, C, NT>(adjoint);
    if (Fy == 256 && Fz == 128) return pick_yz_fz<256, 128, C, NT>(adjoint);
    return nullptr;
}

// Cluster shape of the fused pass: 8 x 512 threads (default) or, with
// DECON_YZ_CLUSTER=16, 16 x 256 threads (two CTAs per SM).
static int yz_cluster_size() {
    const char* e = getenv("DECON_YZ_CLUSTER");
    return (e && atoi(e) == 16) ? 16 : 8;
}

static void* pick_yz(int64_t Fy, int64_t Fz, bool adjoint, int C) {
    return C == 16 ? pick_yz_c<16, 256>(Fy, Fz, adjoint) : pick_yz_c<8, 512>(Fy, Fz, adjoint);
}

// Clusters of k_yz resident at once on this device (cached per kernel).
static int yz_clusters(void* fn, size_t smem, int C, int NT) {
    static std::mutex mu;
    static std::map<std::pair<int, void*>, int> cache;
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lock(mu);
    auto key = std::make_pair(dev, fn);
    auto it = cache.find(key);
    if (it != cache.end()) return it->second;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(C * 64);
    cfg.blockDim = dim3(NT);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = C;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, fn, &cfg) != cudaSuccess || n < 1) {
        cudaGetLastError();
        n = std::max(1, sm_count() / C);
    }
    cache[key] = n;
    return n;
}

static int launch_yz(const ConvPlan& p, bool adjoint, cudaStream_t st) {
    const int C = yz_cluster_size(), NT = C == 16 ? 256 : 512;
    void* fn = pick_yz(p.F[1], p.F[0], adjoint, C);
    if (!fn) return fail(DECON_ERR_UNSUPPORTED, "fused Y / axial pass: unsupported canvas");
    YZArgs a;
    a.s1t = p.s1;
    a.otft = p.otft;
    a.twy = p.twy;
    a.twz = p.twz;
    a.Nz = (int)p.N[0];
    a.Ny = (int)p.N[1];
    a.Hx = (int)p.Hx;
    const size_t smem = yz_smem_bytes((int)p.F[1], (int)p.F[0], C);
    if (C > 8) {
        static std::mutex mu;
        static std::map<std::pair<int, void*>, bool> done;
        int dev = 0;
        cudaGetDevice(&dev);
        std::lock_guard<std::mutex> lock(mu);
        if (!done[std::make_pair(dev, fn)]) {
            DK_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
            done[std::make_pair(dev, fn)] = true;
        }
    }
    DK_TRY(kernel_prepare(fn, smem, NT, nullptr));
    const int ncl = (int)std::min<int64_t>(p.Hx, yz_clusters(fn, smem, C, NT));
    // a cluster launch, timed like the other passes when profiling is on
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(ncl * C));
    cfg.blockDim = dim3(NT);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = C;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    void* params[] = {&a};
    const bool prof = (g_prof.mask & PROF_ZOTF) != 0;
    if (prof) {
        if (g_prof.used == g_prof.ev.size()) {
            cudaEvent_t e0, e1;
            DK_CUDA(cudaEventCreate(&e0));
            DK_CUDA(cudaEventCreate(&e1));
            g_prof.ev.emplace_back(e0, e1);
        }
        DK_CUDA(cudaEventRecord(g_prof.ev[g_prof.used].first, st));
    }
    DK_CUDA(cudaLaunchKernelExC(&cfg, fn, params));
    count_launch();
    if (prof) {
        DK_CUDA(cudaEventRecord(g_prof.ev[g_prof.used].second, st));
        ++g_prof.used;
    }
    return DECON_OK;
}

static bool one_plane(const ConvPlan& p) { return p.y_otf.ok; }

int schedule_bits(const ConvPlan& p) {
    const bool yz = use_yz(p);
    int bits = 0;
    if (p.precision == 0 && getenv("DECON_NO_YZ") == nullptr && getenv("DECON_YZ") == nullptr &&
        (p.otft != nullptr || (yz_supported(p.N, p.F) && p.F[0] != p.N[0])))
        bits |= DECON_SCHED_FUSED;
    const bool columns = one_plane(p) || (p.y_fwd.ok && p.y_inv.ok && p.z_otf.ok);  // register kernels
    if (!yz && p.tma && (one_plane(p) || p.y_fwd.ok || p.y_inv.ok || p.z_otf.ok)) bits |= DECON_SCHED_NO_TMA;
    if (!yz && p.precision == 1 && p.z_otf16.ok) bits |= DECON_SCHED_NO_PIPE;
    const bool rows = pick_xreg_r2c(p.ax_x.L, p.odd, yz, 0).fn && pick_xreg_c2r(p.ax_x.L, p.odd, yz, EPI_STORE).fn;
    if (!rows || (!yz && !columns)) bits |= DECON_SCHED_ODD_RADIX | DECON_SCHED_HALF_LINES;
    return bits;
}

// Forward spectrum: x (window in N-space) -> S2 (after the Y pass), or, with
// the fused Y / axial pass, -> the kx-major S1 (X pass only).
int spectrum_forward(const ConvPlan& p, int pro, const float* in, Win3 win, float cval, float bg,
                     cudaStream_t st) {
    const int64_t Nz = p.N[0], Ny = p.N[1], Fy = p.F[1], P = p.P;
    if (use_yz(p)) return launch_xr2c(p, pro, in, win, cval, bg, Nz, p.s1, st, Nz * Ny);
    DK_TRY(launch_xr2c(p, pro, in, win, cval, bg, Nz, p.s1, st));
    if (!one_plane(p) && !p.s2) return fail(DECON_ERR_CUDA, "the plan's column pass could not be prepared");
    if (one_plane(p)) return DECON_OK;  // the Y transforms run with the product (spectrum_filter_back)
    if (p.y_fwd.ok) {
        DK_TRY(launch_col_pass(p.y_fwd, false, st));
    } else {
        DK_TRY(launch_col(p, p.ax_y, p.T_y, COL_FWD, p.s1, Ny * P, P, (int)Ny, p.s2, Fy * P, P,
                          (int)Fy, Nz, st));
    }
    return DECON_OK;
}

// Z pass (x OTF or conj OTF) and the inverse Y pass: S2 -> S1.
int spectrum_filter_back(const ConvPlan& p, bool adjoint, cudaStream_t st) {
    if (use_yz(p)) return launch_yz(p, adjoint, st);
    if (one_plane(p)) return launch_col_pass(p.y_otf, adjoint, st);
    const int64_t Nz = p.N[0], Ny = p.N[1], Fy = p.F[1], P = p.P;
    const int mode = adjoint ? COL_OTF_CONJ : COL_OTF;
    if (p.z_otf.ok) {
        const bool h16 = p.precision == 1 && p.z_otf16.ok && p.z_otf.maps && !no_pipe(p);
        DK_TRY(launch_col_pass(h16 ? p.z_otf16 : p.z_otf, adjoint, st));
    } else {
        DK_TRY(launch_col(p, p.ax_z, p.T_z, mode, p.s2, P, Fy * P, (int)Nz, p.s2, P, Fy * P,
                          (int)Nz, Fy, st));
    }
    if (p.y_inv.ok) {
        DK_TRY(launch_col_pass(p.y_inv, false, st));
    } else {
        DK_TRY(launch_col(p, p.ax_y, p.T_y, COL_INV, p.s2, Fy * P, P, (int)Fy, p.s1, Ny * P, P,
                          (int)Ny, Nz, st));
    }
    return DECON_OK;
}

}  // namespace dk
