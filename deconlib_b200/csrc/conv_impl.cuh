// Internal declarations of the convolution passes (conv.cu) shared with the
// C ABI (capi.cu) and the solver kernels.
#pragma once

#include <cuda.h>
#include <cuda_fp16.h>

#include "common.cuh"
#include "fft_engine.cuh"

namespace dk {

constexpr int kSmemElems = 8192;  // complex values per CTA (64 KB)

// Lines per CTA of the runtime-radix passes: the largest power of two <= cap
// whose tile fits kSmemElems complex values and whose threads (T x tpl) fit a
// CTA.
inline int fft_lines_per_cta(const Axis& ax, int cap) {
    int T = 1;
    while (T * 2 <= cap && (T * 2) * ax.L <= kSmemElems && (T * 2) * ax.tpl <= kDynThreads) T *= 2;
    return T;
}

// A float32 array of shape (wz, wy, wx) placed at offset (oz, oy, ox) inside
// the N-space volume; voxels outside the box read as zero / are not written.
struct Win3 {
    int64_t wz, wy, wx;
    int64_t oz, oy, ox;
};

inline Win3 full_window(const int64_t* N) { return Win3{N[0], N[1], N[2], 0, 0, 0}; }

// PRO_UP2: the input is the coarse (Nz/2, Ny/2, Nx/2) array of a 2x fractional-area
// downsample and the X pass reads its adjoint (every fine voxel takes its
// coarse voxel's value).  EPI_DOWN2: the output is the 2x area sum of the
// convolved volume, written at the coarse shape.
enum Prologue { PRO_ARRAY = 0, PRO_CONST = 1, PRO_KERNEL = 2, PRO_RLINIT = 3, PRO_UP2 = 4 };
enum Epilogue { EPI_STORE = 0, EPI_RL_RATIO = 1, EPI_RL_UPDATE = 2, EPI_PRED = 3, EPI_DOWN2 = 4 };
enum ColMode { COL_FWD = 0, COL_INV = 1, COL_OTF = 2, COL_OTF_CONJ = 3 };
// kernel classes for decon_profile_start (bit mask)
enum ProfClass { PROF_XR2C = 1, PROF_COL = 2, PROF_ZOTF = 4, PROF_XC2R = 8 };

__device__ __forceinline__ bool kernel_src(int64_t c, int64_t F, int64_t m, int64_t npos,
                                           int64_t& k) {
    // Corner-origin embedding (utils/padding.py:142-190): canvas index c holds
    // kernel index c (c < npos) or c - F + m (the wrapped negative offsets).
    if (c < npos) {
        k = c;
        return c < m;
    }
    const int64_t nneg = m - npos;
    if (c >= F - nneg) {
        k = c - F + m;
        return true;
    }
    return false;
}

struct XR2CArgs {
    const float* in;
    float cval, bg;
    const double* ksum;  // kernel sum the values are divided by (nullptr: not normalised)
    int64_t Nz, Ny, Nx;  // rows = Nz * Ny, row length Nx (zero-padded to Fx)
    Win3 win;
    int64_t Kz, Ky, Kx, pz, py, px;  // kernel embedding (PRO_KERNEL)
    float2* out;
    int64_t P, nrows;
    int Hx, odd, T, vec4;
    Axis ax;            // length Fx/2 (even Fx) or Fx (odd)
    const float2* twx;  // W_Fx table
    FastDiv fd_q4, fd_H, fd_nin, fd_np;  // Nx / 4, Hx, packed non-zero points, L / 2 + 1
    // 0: spectrum rows of pitch P (element (row, kx) at row * P + kx); > 0:
    // kx-major spectrum, element (row, kx) at kx * kstride + row (kstride =
    // Nz * Ny), the layout of the fused Y / axial pass
    int64_t kstride;
};

struct ColArgs {
    const float2* src;
    float2* dst;
    int64_t src_os, src_js, dst_os, dst_js;
    int nin, nout, ncols, T, mode, ntiles;
    Axis ax;
    const float2* otf;
    int64_t otf_js, otf_os;
};

// Register column pass (k_colreg, colreg.cuh): tile geometry, tensor maps of
// the rows that come by TMA, and the plain addresses of the same rows.
struct ColRegArgs {
    CUtensorMap srcmap, otfmap;
    const float2* src;
    float2* dst;
    int64_t src_os, src_js, dst_os, dst_js;
    int nin, nout, nouter;
    int nfull, rem, per;   // full tiles per plane, columns past them, planes per tile of those
    int nmain, ntiles;     // full tiles, all tiles
    int jdim, box, nbox;   // source map: dimension of the rows, rows per box, boxes
    int obox, onbox, in_bytes;
    const float2* tw;      // W_L table, W_L^m = tw[m * tws]
    int tws;
    float conj;            // -1: multiply by conj(OTF)
    const float2* otf;
    const __half2* otf16;  // mixed precision: OTF = otf16 * otf_inv[kz]
    const float* otf_inv;
    int64_t otf_os, otf_js;
    int* flag;             // raised when a bounded wait gives up
};
struct ColRegKernel {
    void* fn = nullptr;
    int T = 0, nt = 0, exch = 0;
};
// One column pass of a plan, ready to launch.
struct ColPass {
    ColRegKernel k;
    ColRegArgs a;
    int smem = 0, grid = 0;
    bool ok = false, maps = false;  // maps: the rows come by TMA
};
ColRegKernel colreg_group_a(int L, int mode, bool plain);
ColRegKernel colreg_group_b(int L, int mode, bool plain);
ColRegKernel colreg_group_c(int L, int mode, bool plain);
ColRegKernel colreg_group_d(int L, int mode, bool plain);
ColRegKernel colreg_group_e(int L, int mode, bool plain);

// Register X passes (xreg.cuh).
struct XRegArgs {
    int pro;               // Prologue (array, constant or RL start in the array kernel)
    const float* in;       // R2C input
    float cval, bg;
    const double* ksum;  // kernel sum the values are divided by (nullptr: not normalised)
    int64_t Nz, Ny, Nx;
    int64_t Kz, Ky, Kx, pz, py, px;  // kernel embedding (PRO_KERNEL)
    float2* out;           // R2C output spectrum
    const float2* spec;    // C2R input spectrum
    float* out_real;       // C2R output
    const float *aux0, *aux1;
    double* partials;
    int pred;              // EPI_RL_RATIO kernel: store the model, not the ratio
    float scale;
    int64_t P;
    // the real array is the box (wz, wy, wx) at (z0, y0, x0) of the volume; win: a
    // box smaller than the volume (R2C: zero outside; C2R: nothing else is kept)
    int win, z0, y0, x0, wz, wy, wx;
    uint32_t nrows, nlines;  // rows of the volume (C2R: of the box); lines (rows, or pairs for odd Fx)
    int nin, nout;           // points of a line that can be non-zero / are kept
    int Hx;                  // spectrum points of a row
    int vec;                 // rows are 8-byte aligned pairs
    const float2* tw;        // W_L table, W_L^m = tw[m * tws]
    int tws;
    const float2* twx;       // W_Fx table
};
struct XRegKernel {
    void* fn = nullptr;
    int TL = 0, nt = 0, smem = 0;
};
#define DK_XREG_GROUPS(X) X(a) X(b) X(c) X(d) X(e) X(f) X(g) X(odd) X(kx)
#define DK_XREG_DECL(g)                       \
    XRegKernel xreg_r2c_##g(int L, int src);  \
    XRegKernel xreg_c2r_##g(int L, int epi);
DK_XREG_GROUPS(DK_XREG_DECL)
#undef DK_XREG_DECL

struct XC2RArgs {
    const float2* in;
    int64_t P, Ny, Nx, nrows;
    int Hx, odd, T, vec4;
    Axis ax;
    const float2* twx;
    float scale;
    Win3 win;
    float* out;
    const float* aux0;
    const float* aux1;
    float bg;
    double* partials;
    FastDiv fd_L, fd_h2, fd_npair, fd_q4, fd_Nx;  // L, L / 2, L / 2 + 1, Nx / 4, Nx
    int64_t kstride;  // as XR2CArgs::kstride
};

// Device-resident state of one LinearFFTConvolver.
struct ConvPlan {
    int64_t N[3], F[3], K[3];
    int64_t Hx, P;
    int odd;
    Axis ax_x, ax_y, ax_z;
    int T_x, T_y, T_z;
    float2 *otf, *s1, *s2;
    const float2 *twx, *twy, *twz;
    double* dscal;        // device scalars (kernel sum, reductions)
    double* partials;     // per-CTA FP64 partial sums of fused reductions
    int64_t npartials;
    const double* ksum;   // device scalar the kernel is divided by, or nullptr
    double norm_sq;
    int device;
    // Register column passes (ok when the axis length has one): Y forward
    // S1 -> S2, axial in S2 (FP32 and FP16 OTF), Y inverse S2 -> S1; one plane
    // (Fz = 1, images): Y forward, product and Y inverse in one pass over S1
    ColPass y_fwd, z_otf, z_otf16, y_inv, y_otf;
    bool tma = true;  // tensor maps (DECON_NO_TMA was not set when the plan was made)
    // Mixed precision (decon_conv_set_precision): the OTF also stored as FP16
    // complex, scaled per kz plane by a power of two (OTF = otf16 * otf_inv[kz]),
    // read by the axial pass instead of the FP32 OTF.
    int precision = 0;
    __half2* otf16 = nullptr;
    float* otf_inv = nullptr;
    // Fused Y / axial pass (yzpass.cuh): the OTF also stored kx-major
    // [Hx][Fy][Fz]; the spectrum between the X passes is then kx-major too
    // ([Hx][Nz][Ny] in s1).  nullptr: the canvas takes the unfused passes.
    float2* otft = nullptr;
    // Schedule (decon_conv_set_schedule): DECON_SCHED_* bits choosing among
    // equivalent pass families; T*_0 / ax*_0 keep the default lines per CTA
    // and radix plans the schedule modifies.
    int sched = 0;
    int T_x0 = 0, T_y0 = 0, T_z0 = 0;
};

// Canvas and signal extents the fused Y / axial pass implements (Fy in {256,
// 512}, Fz in {128, 256}, the signal in the first half of both axes, Ny even).
bool yz_supported(const int64_t N[3], const int64_t F[3]);
// True when this plan's convolutions run the fused Y / axial pass.
bool use_yz(const ConvPlan& p);
// Fill p.otft from p.otf (after every OTF build).
int build_otf_kmajor(const ConvPlan& p, cudaStream_t st);

// Quantise p.otf into p.otf16 / p.otf_inv (capi.cu).
int quantize_otf(const ConvPlan& p, cudaStream_t st);
// The schedule bits that change a launch of this plan (conv.cu).
int schedule_bits(const ConvPlan& p);
// True when this plan's axial pass can take an FP16 OTF (conv.cu).
bool zpass_pipelined(const ConvPlan& p);

// Shared-memory opt-in (only ever raised per device and kernel) and cached
// occupancy for a launch shape (conv.cu).
int kernel_prepare(void* fn, size_t smem, int nthr, int* per_sm);

// Runtime-radix kernels (fftplain.cu) by prologue / epilogue code; nullptr for
// an unknown code.
void* pick_xr2c_kernel(int pro);
void* pick_xc2r_kernel(int epi);
void* pick_colfft_kernel();

// Column passes of the plan's buffers (after they are allocated), and the
// transform of the OTF buffer along an axis (1: y, 0: z) in place.
void make_col_passes(ConvPlan& p);
// The one pass of a one-plane canvas, which needs no S2; false: there is none.
bool make_one_plane_pass(ConvPlan& p);
void make_z_otf16(ConvPlan& p);
int transform_otf(const ConvPlan& p, int axis, cudaStream_t st);

int launch_xr2c(const ConvPlan& p, int pro, const float* in, Win3 win, float cval, float bg,
                int64_t nz_rows, float2* out, cudaStream_t st, int64_t kstride = 0);
int launch_col(const ConvPlan& p, const Axis& ax, int T, int mode, const float2* src,
               int64_t src_os, int64_t src_js, int nin, float2* dst, int64_t dst_os,
               int64_t dst_js, int nout, int64_t nouter, cudaStream_t st);
int launch_xc2r(const ConvPlan& p, int epi, const float2* in, Win3 win, float* out,
                const float* aux0, const float* aux1, float bg, double* partials, int* nblk_out,
                cudaStream_t st);
int spectrum_forward(const ConvPlan& p, int pro, const float* in, Win3 win, float cval, float bg,
                     cudaStream_t st);
int spectrum_filter_back(const ConvPlan& p, bool adjoint, cudaStream_t st);

// FP64 reductions (reduce.cu)
int reduce_f32(const float* a, const float* b, int64_t n, int op, double* out, double* partials,
               int64_t npartials, cudaStream_t st);
int finish_partials(const double* partials, int n, double* out, cudaStream_t st);
int64_t reduce_partials_needed();

}  // namespace dk

struct decon_conv : dk::ConvPlan {};
