// X passes (real-to-complex and back) with the transform in registers.
//
// Even Fx: a row is packed as L = M = Fx / 2 complex points z[n] = x[2n] +
// i x[2n+1].  Odd Fx: two rows make one line z[n] = xa[n] + i xb[n] of L = Fx
// points.  L = B x S runs as two register DFTs around one exchange through
// shared memory, and the packing is undone (or done) in the same registers:
// spectrum points k and L - k lie in butterflies u and B - u of the radix-S
// stage, so one thread takes both and no second pass over shared memory is
// needed.  Rows are read and written by the threads that transform them, 8 or
// 16 bytes a lane in whole row pieces.
//
//   R2C  stage 1: radix B over n = j + r S (global rows -> exchange)
//        stage 2: radix S, butterflies u and B - u -> X[k], X[L - k]
//   C2R  stage 1: X[k], X[L - k] -> radix S, butterflies u and B - u
//        stage 2: radix B -> x, with the element-wise epilogues
//
// KX: the kx-major spectrum of the fused Y / axial pass, element (k, row) at
// k P + row.  Adjacent threads then take adjacent rows in the spectrum stage, 64
// bytes of a frequency (8 rows) in whole pieces.  A template: as a run-time stride
// it would cost the row-major passes.
//
// The self-paired butterflies (u = 0, and B / 2 for even B) go through the same
// code: their second half repeats the first and is not stored.
#pragma once

#include "codelets.cuh"
#include "conv_impl.cuh"

namespace dk {

// The radix S of which a thread holds two butterflies: the most equal pair with S
// at most 20 (odd lines: 27, one register set per pair of rows), and above 512
// points at most 24, then 32, where 20 leaves no pair: the fewer registers, the
// more lines per SM (800 points as 20 x 40 instead of 25 x 32: R2C of 32768 rows 118 ->
// 88 us, C2R 135 -> 108; 960 as 24 x 40 instead of 30 x 32: 139 -> 108, 148 -> 131).
// Against the runtime-radix passes: 640 points 279 -> 71 and 311 -> 89 us, 1024
// points 381 -> 144 and 410 -> 164.
constexpr int xreg_radix(int L, bool odd) {
    if (odd) return small_radix(L, 27);
    for (int most : {20, 24, 32}) {
        const int s = small_radix(L, most);
        if (s != 0 || L <= 512) return s;
    }
    return 0;
}

// Lines, threads and exchange layout of a CTA.
template <int L, bool ODD>
struct XRegShape {
    static constexpr int S = xreg_radix(L, ODD), B = L / S;
    static constexpr int TPL = B / 2 + 1;  // threads per line in the paired stage
    static constexpr int TL = 32 * TPL <= 160 ? 32 : (16 * TPL <= 160 ? 16 : (8 * TPL <= 160 ? 8 : 4));
    static constexpr int NT = (TL * TPL + 31) / 32 * 32;
    // one exchange row per butterfly of the first stage, an odd number of
    // points apart: consecutive lanes hit different banks
    template <int R>
    struct Ex {
        static constexpr int step = R | 1;               // row length
        static constexpr int need = (L / R) * step;
        // lines start TPL points apart modulo 16, so a half-warp that spans
        // two lines still covers distinct banks
        static constexpr int pitch = need + (((TPL - need) % 16) + 16) % 16;
        static constexpr int bytes = TL * pitch * (int)sizeof(float2);
    };
    static constexpr int blocks_for(int regs) {
        const int b = 65536 / (NT * ((regs + 7) / 8 * 8));
        return b < 1 ? 1 : (b > 10 ? 10 : b);
    }
};

// ---------------------------------------------------------------------------
// pass 1: X R2C
// ---------------------------------------------------------------------------

enum XRegSrc { XS_ARRAY = 0, XS_UP2 = 1, XS_KERNEL = 2 };

// Row of the canvas as the corner-origin embedding of the kernel: nullptr for a
// row of zeros.
__device__ __forceinline__ const float* embedded_row(const XRegArgs& a, int64_t row) {
    if (row >= a.nrows) return nullptr;
    int64_t kz, ky;
    const int64_t z = row / a.Ny, y = row - z * a.Ny;
    if (!kernel_src(z, a.Nz, a.Kz, a.pz, kz) || !kernel_src(y, a.Ny, a.Ky, a.py, ky)) return nullptr;
    return a.in + (kz * a.Ky + ky) * a.Kx;
}
__device__ __forceinline__ float embedded(const XRegArgs& a, const float* p, int x, float sum) {
    int64_t kx;
    if (p == nullptr || x >= a.Nx || !kernel_src(x, a.Nx, a.Kx, a.px, kx)) return 0.f;
    return __ldg(p + kx) / sum;
}

// Bytes lo .. hi of an array of `size` bytes into L2, by one thread.  The rows a
// CTA reads are one piece of memory; its threads ask for them 8 bytes at a time
// and in two or more rounds, and the operands of an epilogue only after the
// transform.  One bulk request ahead of all that (150x600x700, X length 400):
// R2C 138 -> 117 us, update epilogue 274 -> 242, ratio 259 -> 242.  Requesting
// rows of later CTAs instead, or the spectrum rows of the C2R pass, which are
// all asked for at once anyway, gained no more (34.1 vs 35.2 us at 256).
__device__ __forceinline__ void prefetch_l2(const void* p, int64_t lo, int64_t hi, int64_t size) {
    if (hi > size) hi = size;
    const uintptr_t b = (reinterpret_cast<uintptr_t>(p) + lo + 15) & ~(uintptr_t)15;
    const uintptr_t e = (reinterpret_cast<uintptr_t>(p) + hi) & ~(uintptr_t)15;
    if (lo < hi && b < e)
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(b), "r"((uint32_t)(e - b)) : "memory");
}

// Spectrum rows row0 .. row0 + ROWS of zero lines.
template <int ROWS, int NT, bool KX>
__device__ __forceinline__ void zero_rows(const XRegArgs& a, int64_t row0) {
    const int n = (int)(row0 + ROWS < a.nrows ? ROWS : (int64_t)a.nrows - row0);
    for (int i = 0; i < n; ++i)
        for (int k = threadIdx.x; k < a.Hx; k += NT) a.out[KX ? k * a.P + row0 + i : (row0 + i) * a.P + k] = make_float2(0.f, 0.f);
}

// Offset of x = 0 of a row in the real array (its window of the volume: elements
// x0 .. x0 + wx of the row exist), or kNoRow outside of it.
constexpr int64_t kNoRow = INT64_MIN;
__device__ __forceinline__ int64_t array_row(const XRegArgs& a, uint32_t row) {
    if (row >= a.nrows) return kNoRow;
    if (!a.win) return (int64_t)row * a.Nx;
    const uint32_t z = row / (uint32_t)a.Ny, y = row - z * (uint32_t)a.Ny;
    const uint32_t iz = z - (uint32_t)a.z0, iy = y - (uint32_t)a.y0;
    if (iz >= (uint32_t)a.wz || iy >= (uint32_t)a.wy) return kNoRow;
    return (int64_t)(iz * (uint32_t)a.wy + iy) * a.wx - a.x0;
}

template <int L, bool ODD, int SRC, bool KX>
__global__ void __launch_bounds__(XRegShape<L, ODD>::NT, XRegShape<L, ODD>::blocks_for(4 * XRegShape<L, ODD>::S + 44))
    k_xreg_r2c(const XRegArgs a) {
    using H = XRegShape<L, ODD>;
    constexpr int S = H::S, B = H::B, TL = H::TL, NT = H::NT, TPL = H::TPL;
    using E = typename H::template Ex<B>;
    extern __shared__ float2 sm[];
    const int tid = threadIdx.x;
    const uint32_t line0 = blockIdx.x * TL;
    chain_enter();
    float2* stg = sm + TL * E::pitch;  // staged rows (XS_KERNEL)
    if constexpr (SRC == XS_KERNEL) {
        __shared__ const float* rows[2 * TL];
        constexpr int W = ODD ? 2 : 1;  // rows per line
        bool any = false;
        for (int i = tid; i < W * TL; i += NT) {
            rows[i] = embedded_row(a, (int64_t)W * line0 + i);
            any = any || rows[i] != nullptr;
        }
        if (!__syncthreads_or(any)) {
            // the kernel covers a part of the canvas: whole CTAs of zero rows
            // (three quarters of them for a kernel of half the canvas)
            zero_rows<W * TL, NT, KX>(a, (int64_t)W * line0);
            return;
        }
        const float sum = a.ksum ? (float)__ldg(a.ksum) : 1.f;
        for (int q = tid; q < TL * L; q += NT) {
            const int l = q / L, n = q - l * L;
            stg[q] = ODD ? make_float2(embedded(a, rows[2 * l], n, sum), embedded(a, rows[2 * l + 1], n, sum))
                         : make_float2(embedded(a, rows[l], 2 * n, sum), embedded(a, rows[l], 2 * n + 1, sum));
        }
        __syncthreads();
    }

    if constexpr (SRC == XS_ARRAY) {
        if (tid == 0 && !a.win && a.pro != PRO_CONST) {
            constexpr int W = ODD ? 2 : 1;
            const int64_t row = W * (int64_t)line0;
            prefetch_l2(a.in, row * a.Nx * 4, (row + W * TL) * a.Nx * 4, a.nrows * a.Nx * 4);
        }
        if (a.win) {
            constexpr int W = ODD ? 2 : 1;
            bool any = false;
            for (int i = tid; i < W * TL; i += NT) any = any || array_row(a, W * line0 + i) != kNoRow;
            if (!__syncthreads_or(any)) {
                zero_rows<W * TL, NT, KX>(a, (int64_t)W * line0);
                return;
            }
        }
    }

    // stage 1
#pragma unroll 1
    for (int q = tid; q < TL * S; q += NT) {
        const int l = q / S, j = q - l * S;
        const uint32_t line = line0 + l;
        C1 v[B];
        if constexpr (SRC == XS_KERNEL) {
#pragma unroll
            for (int r = 0; r < B; ++r) v[r] = as_c1(stg[l * L + j + r * S]);
        } else if constexpr (SRC == XS_UP2) {
            // fine row (z, y) of the adjoint of the 2x area sum: fine x = 2n and
            // 2n + 1 both take coarse value n of coarse row (z / 2, y / 2)
            const uint32_t z = line / (uint32_t)a.Ny, y = line - z * (uint32_t)a.Ny;
            const float* p = a.in + ((int64_t)(z >> 1) * (a.Ny >> 1) + (y >> 1)) * (a.Nx >> 1);
            const int lim = line < a.nrows ? a.nin : 0;
#pragma unroll
            for (int r = 0; r < B; ++r) {
                const float w = j + r * S < lim ? __ldg(p + j + r * S) : 0.f;
                v[r] = C1{w, w};
            }
        } else if (a.pro == PRO_CONST) {
            const int lim = line < a.nlines ? (ODD ? (int)a.Nx : (int)(a.Nx >> 1)) : 0;
            const bool two = !ODD || 2 * line + 1 < a.nrows, half = !ODD && (a.Nx & 1) && line < a.nlines;
#pragma unroll
            for (int r = 0; r < B; ++r) {
                const int n = j + r * S;
                v[r] = C1{n < lim || (half && n == lim) ? a.cval : 0.f, n < lim && two ? a.cval : 0.f};
            }
        } else {
            // real part: row pa (odd Fx: the first row of the pair), imaginary part: pb
            const int64_t oa = array_row(a, ODD ? 2 * line : line);
            const int64_t ob = ODD ? array_row(a, 2 * line + 1) : oa;
            const float *pa = a.in + (oa == kNoRow ? 0 : oa), *pb = a.in + (ob == kNoRow ? 0 : ob);
            const uint32_t wa = oa == kNoRow ? 0 : a.wx, wb = ob == kNoRow ? 0 : a.wx;
            auto has = [&](uint32_t w, int x) { return (uint32_t)(x - a.x0) < w; };
            if constexpr (ODD) {
#pragma unroll
                for (int r = 0; r < B; ++r) {
                    const int n = j + r * S;
                    v[r] = C1{has(wa, n) ? __ldg(pa + n) : 0.f, has(wb, n) ? __ldg(pb + n) : 0.f};
                }
            } else if (a.vec) {
#pragma unroll
                for (int r = 0; r < B; ++r) {
                    const int x = 2 * (j + r * S);
                    v[r] = has(wa, x) ? as_c1(__ldg(reinterpret_cast<const float2*>(pa + x))) : C1{0.f, 0.f};
                }
            } else {
#pragma unroll
                for (int r = 0; r < B; ++r) {
                    const int x = 2 * (j + r * S);
                    v[r] = C1{has(wa, x) ? __ldg(pa + x) : 0.f, has(wa, x + 1) ? __ldg(pa + x + 1) : 0.f};
                }
            }
            if (a.pro == PRO_RLINIT) {
                // max(y - b, 1e-6) (rl_mlx.py:123-125), after all loads are out
#pragma unroll
                for (int r = 0; r < B; ++r) {
                    const int x = ODD ? j + r * S : 2 * (j + r * S);
                    v[r] = C1{has(wa, x) ? fmaxf(v[r].re - a.bg, 1e-6f) : 0.f,
                              has(wb, ODD ? x : x + 1) ? fmaxf(v[r].im - a.bg, 1e-6f) : 0.f};
                }
            }
        }
        dftn<B, -1>(v);
        float2* e = sm + l * E::pitch + j * E::step;
#pragma unroll
        for (int r = 0; r < B; ++r) e[r] = as_f2(v[r]);
    }
    __syncthreads();

    // stage 2
    const int l = KX ? tid % TL : tid / TPL, u = KX ? tid / TL : tid - l * TPL;
    const uint32_t line = line0 + l;
    if ((KX ? u >= TPL : l >= TL) || line >= a.nlines) return;
    C1 va[S], vb[S];
    {
        const float2* e = sm + l * E::pitch;
        const int m = u == 0 ? 0 : B - u;
#pragma unroll
        for (int r = 0; r < S; ++r) {
            va[r] = as_c1(e[u + r * E::step]);
            vb[r] = as_c1(e[m + r * E::step]);
            if (r > 0) {
                const float2 w = __ldg(&a.tw[(r * u) * a.tws]);
                va[r] = twist<false>(va[r], w);
                // W^(r (B - u)) without its factor W_S^r, which shifts the
                // outputs by one (read below at index + 1)
                vb[r] = twist<true>(vb[r], w);
            }
        }
    }
    dftn<S, -1>(va);
    dftn<S, -1>(vb);
    if constexpr (!ODD) {
        // X[k] = e + W^k o, X[M-k] = conj(e - W^k o) with e = (Z[k] + conj
        // Z[M-k]) / 2, o = -i (Z[k] - conj Z[M-k]) / 2
        float2* out = a.out + (KX ? (int64_t)line : (int64_t)line * a.P);
        const int64_t ks = KX ? a.P : 1;
        const bool second = u > 0 && 2 * u < B;
#pragma unroll
        for (int r = 0; r < S; ++r) {
            const int k = u + r * B;
            const C1 zk = va[r], zm = conj_of(vb[(S - r) % S]);
            const C1 s = zk + zm, d = zk - zm;
            const C1 e{0.5f * s.re, 0.5f * s.im}, o{0.5f * d.im, -0.5f * d.re};
            const C1 t = twist<false>(o, __ldg(&a.twx[k]));
            out[k * ks] = as_f2(e + t);
            if (second || (u == 0 && r == 0)) out[(L - k) * ks] = as_f2(conj_of(e - t));
        }
    } else {
        // Xa = (Z[k] + conj Z[L-k]) / 2, Xb = -i (Z[k] - conj Z[L-k]) / 2
        float2* out = a.out + (int64_t)line * 2 * a.P;
        const bool two = 2 * line + 1 < a.nrows;
#pragma unroll
        for (int r = 0; r < S; ++r) {
            int k = u + r * B;
            const C1 zk = va[r], zm = conj_of(vb[(S - r) % S]);
            const C1 s = zk + zm, d = zk - zm;
            C1 xa{0.5f * s.re, 0.5f * s.im}, xb{0.5f * d.im, -0.5f * d.re};
            if (2 * k > L) {
                if (u == 0) continue;
                k = L - k;
                xa = conj_of(xa);
                xb = conj_of(xb);
            }
            out[k] = as_f2(xa);
            if (two) out[a.P + k] = as_f2(xb);
        }
    }
}

// ---------------------------------------------------------------------------
// pass 5: X C2R with fused epilogues
// ---------------------------------------------------------------------------

// Element-wise epilogues: what a voxel's new value is made of.  The operands of
// several voxels are fetched before any of them is stored: x is read and
// written in place, so the compiler keeps each load behind the store before it
// and the pass waited for HBM once per voxel (150x600x700: 490 us, 140 us for
// the plain store).
template <typename V>
struct XOperands {
    V x, y;
};
template <int EPI, typename V>
__device__ __forceinline__ XOperands<V> x_fetch(const XRegArgs& a, int64_t i) {
    XOperands<V> o{};
    if constexpr (EPI == EPI_RL_UPDATE) {
        o.x = *reinterpret_cast<const V*>(a.aux0 + i);
        o.y = __ldg(reinterpret_cast<const V*>(a.aux1 + i));
    } else if constexpr (EPI != EPI_STORE) {
        o.y = __ldg(reinterpret_cast<const V*>(a.aux0 + i));
    }
    return o;
}
// v: the convolution's value, already scaled
template <int EPI>
__device__ __forceinline__ float x_value(const XRegArgs& a, float v, float x, float y, double& acc) {
    if constexpr (EPI == EPI_STORE) {
        return v;
    } else if constexpr (EPI == EPI_RL_UPDATE) {
        // rl_mlx.py:149-150  x = max(x * where(active, A^T ratio / sens, 0), 1e-10)
        const float c = y > 0.f ? v / y : 0.f;
        return fmaxf(x * c, 1e-10f);
    } else if constexpr (EPI == EPI_RL_RATIO) {
        // rl_mlx.py:147-148  model = A x + b ; ratio = y / max(model, 1e-10)
        return y / fmaxf(v + a.bg, 1e-10f);
    } else {
        const float m = v + a.bg;
        if (a.partials) {
            // rl_mlx.py:75-79: y log(max(y,eps)/max(m,eps)) - (y - max(m,eps))
            const float ys = fmaxf(y, 1e-6f), ms = fmaxf(m, 1e-6f);
            acc += (double)(y * logf(ys / ms) - (y - ms));
        }
        return a.pred ? m : y / fmaxf(m, 1e-10f);
    }
}
template <int EPI>
__device__ __forceinline__ float2 x_value(const XRegArgs& a, float2 v, float2 x, float2 y, double& acc) {
    const float o0 = x_value<EPI>(a, v.x, x.x, y.x, acc);
    return make_float2(o0, x_value<EPI>(a, v.y, x.y, y.y, acc));
}
// Voxels i + r step, r < B, that keep(r) selects; value(r): the convolution there.
template <int EPI, typename V, int B, class Keep, class Value>
__device__ __forceinline__ void x_store(const XRegArgs& a, int64_t i, int step, double& acc, Keep keep, Value value) {
    constexpr int U = EPI == EPI_STORE ? 1 : (EPI == EPI_RL_UPDATE ? 4 : 8);
#pragma unroll
    for (int r0 = 0; r0 < B; r0 += U) {
        XOperands<V> o[U];
#pragma unroll
        for (int e = 0; e < U; ++e)
            if (r0 + e < B && keep(r0 + e)) o[e] = x_fetch<EPI, V>(a, i + (int64_t)(r0 + e) * step);
#pragma unroll
        for (int e = 0; e < U; ++e)
            if (r0 + e < B && keep(r0 + e))
                *reinterpret_cast<V*>(a.out_real + i + (int64_t)(r0 + e) * step) =
                    x_value<EPI>(a, value(r0 + e), o[e].x, o[e].y, acc);
    }
}

// A thread's B points of one line of the real array.
template <int EPI, bool ODD, int B, int S>
__device__ __forceinline__ void c2r_store(const XRegArgs& a, uint32_t line, int j, float s, const C1* v, double& acc) {
    // elements x0 .. x0 + wx of a row are kept (all of them but for a window)
    auto kept = [&](int x) { return (uint32_t)(x - a.x0) < (uint32_t)a.wx; };
    if constexpr (ODD) {
        const int64_t o0 = array_row(a, 2 * line), o1 = array_row(a, 2 * line + 1);
        auto in_row = [&](int r) { return kept(j + r * S); };
        if (o0 != kNoRow) x_store<EPI, float, B>(a, o0 + j, S, acc, in_row, [&](int r) { return v[r].re * s; });
        if (o1 != kNoRow) x_store<EPI, float, B>(a, o1 + j, S, acc, in_row, [&](int r) { return v[r].im * s; });
    } else if (a.vec) {
        x_store<EPI, float2, B>(a, (int64_t)line * a.wx - a.x0 + 2 * j, 2 * S, acc,
                                [&](int r) { return kept(2 * (j + r * S)); },
                                [&](int r) { return make_float2(v[r].re * s, v[r].im * s); });
    } else {
        const int64_t i = (int64_t)line * a.wx - a.x0 + 2 * j;
        x_store<EPI, float, B>(a, i, 2 * S, acc, [&](int r) { return kept(2 * (j + r * S)); },
                               [&](int r) { return v[r].re * s; });
        x_store<EPI, float, B>(a, i + 1, 2 * S, acc, [&](int r) { return kept(2 * (j + r * S) + 1); },
                               [&](int r) { return v[r].im * s; });
    }
}

// Spectrum row of output row `row`: the same, a row of the output's window, or,
// for the 2x area sum, the four rows of one 2 x 2 (z, y) block in lines 4q ..
// 4q + 3.
template <int EPI>
__device__ __forceinline__ uint32_t c2r_row(const XRegArgs& a, uint32_t row) {
    if constexpr (EPI == EPI_DOWN2) {
        const uint32_t q = row >> 2, my = (uint32_t)a.Ny >> 1;
        const uint32_t k = q / my, y = q - k * my;
        return (2 * k + (row & 1)) * (uint32_t)a.Ny + 2 * y + ((row >> 1) & 1);
    } else if constexpr (EPI == EPI_STORE) {
        if (!a.win) return row;
        const uint32_t z = row / (uint32_t)a.wy, y = row - z * (uint32_t)a.wy;
        return (z + (uint32_t)a.z0) * (uint32_t)a.Ny + y + (uint32_t)a.y0;
    } else {
        return row;
    }
}

template <int L, bool ODD, int EPI, bool KX>
__global__ void __launch_bounds__(XRegShape<L, ODD>::NT,
                                  XRegShape<L, ODD>::blocks_for(EPI == EPI_DOWN2 && XRegShape<L, ODD>::B > 12
                                                                    ? 4 * XRegShape<L, ODD>::B + 44
                                                                    : 4 * XRegShape<L, ODD>::S + 44))
    k_xreg_c2r(const XRegArgs a) {
    using H = XRegShape<L, ODD>;
    constexpr int S = H::S, B = H::B, TL = H::TL, NT = H::NT, TPL = H::TPL;
    using E = typename H::template Ex<S>;
    extern __shared__ float2 sm[];
    const int tid = threadIdx.x;
    const uint32_t line0 = blockIdx.x * TL;
    chain_enter();

    if constexpr (EPI == EPI_RL_RATIO || EPI == EPI_RL_UPDATE) {
        if (tid == 0) {
            constexpr int W = ODD ? 2 : 1;
            const int64_t lo = W * (int64_t)line0 * a.Nx * 4, hi = lo + W * TL * a.Nx * 4, size = a.nrows * a.Nx * 4;
            prefetch_l2(a.aux0, lo, hi, size);
            if (EPI == EPI_RL_UPDATE) prefetch_l2(a.aux1, lo, hi, size);
        }
    }
    if constexpr (ODD && EPI == EPI_STORE) {
        if (a.win) {  // pairs of rows outside the window
            bool any = false;
            for (int i = tid; i < 2 * TL; i += NT) any = any || array_row(a, 2 * line0 + i) != kNoRow;
            if (!__syncthreads_or(any)) return;
        }
    }

    // stage 1
    {
        const int l = KX ? tid % TL : tid / TPL, u = KX ? tid / TL : tid - l * TPL;
        const uint32_t line = line0 + l;
        if ((KX ? u < TPL : l < TL) && line < a.nlines) {
            C1 va[S], vb[S];
            if constexpr (!ODD) {
                // Z[k] = e + i d W^-k, Z[M-k] = conj(e) + i conj(d W^-k) with e = X[k] +
                // conj X[M-k], d = X[k] - conj X[M-k]; irfft ignores Im of DC and Nyquist
                const int64_t row = c2r_row<EPI>(a, line), ks = KX ? a.P : 1;
                const float2* in = a.spec + (KX ? row : row * a.P);
#pragma unroll
                for (int r = 0; r < S; ++r) {
                    va[r] = as_c1(__ldg(in + (u + r * B) * ks));
                    vb[r] = as_c1(__ldg(in + (L - u - r * B) * ks));
                }
                if (u == 0) va[0].im = vb[0].im = 0.f;
#pragma unroll
                for (int r = 0; r < S; ++r) {
                    const C1 xm = conj_of(vb[r]);
                    const C1 e = va[r] + xm, d = va[r] - xm;
                    const C1 t = twist<true>(d, __ldg(&a.twx[u + r * B]));
                    va[r] = C1{e.re - t.im, e.im + t.re};
                    vb[r] = C1{e.re + t.im, t.re - e.im};
                }
            } else {
                // Z[k] = Xa[k] + i Xb[k], Z[L-k] = conj(Xa[k]) + i conj(Xb[k])
                const float2* in = a.spec + (int64_t)line * 2 * a.P;
                const bool two = 2 * line + 1 < a.nrows;
#pragma unroll
                for (int r = 0; r < S; ++r) {
                    const int k = u + r * B;
                    const bool up = 2 * k > L;
                    const int h = up ? L - k : k;
                    va[r] = as_c1(__ldg(in + h));
                    vb[r] = two ? as_c1(__ldg(in + a.P + h)) : C1{0.f, 0.f};
                    if (up) {
                        va[r].im = -va[r].im;
                        vb[r].im = -vb[r].im;
                    }
                }
                if (u == 0) va[0].im = vb[0].im = 0.f;
#pragma unroll
                for (int r = 0; r < S; ++r) {
                    const C1 xa = va[r], xb = vb[r];
                    va[r] = C1{xa.re - xb.im, xa.im + xb.re};
                    vb[r] = C1{xa.re + xb.im, xb.re - xa.im};
                }
            }
            float2* e = sm + l * E::pitch;
            dftn<S, +1>(va);
#pragma unroll
            for (int r = 0; r < S; ++r) e[u * E::step + r] = as_f2(va[r]);
            if (u > 0 && 2 * u < B) {
                // butterfly B - u holds Z[L-k] in reverse order
#pragma unroll
                for (int r = 0; r < S / 2; ++r) {
                    const C1 t = vb[r];
                    vb[r] = vb[S - 1 - r];
                    vb[S - 1 - r] = t;
                }
                dftn<S, +1>(vb);
#pragma unroll
                for (int r = 0; r < S; ++r) e[(B - u) * E::step + r] = as_f2(vb[r]);
            }
        }
    }
    __syncthreads();

    // stage 2
    double acc = 0.0;
    auto transform = [&](int l, int j, C1 (&v)[B]) {
        const float2* e = sm + l * E::pitch + j;
#pragma unroll
        for (int r = 0; r < B; ++r) {
            v[r] = as_c1(e[r * E::step]);
            if (r > 0) v[r] = twist<true>(v[r], __ldg(&a.tw[(r * j) * a.tws]));
        }
        dftn<B, +1>(v);
    };
    const float s = a.scale;
    if constexpr (EPI == EPI_DOWN2) {
        // 2x area sum of the scaled output, in the order of the three banded
        // passes (z pairs, then y pairs, then x pairs; unit weights).  Lines
        // 4q, 4q+1: planes 2k, 2k+1 at y = 2j; 4q+2, 4q+3: at y = 2j+1.
        // Round-to-nearest intrinsics: every product and sum is rounded as the
        // stored output and the separate passes round it (no fma).
#pragma unroll 1
        for (int q = tid; q < TL / 4 * S; q += NT) {
            const int b = q / S, j = q - b * S;
            const uint32_t line = line0 + 4 * b;
            if (line >= a.nlines) continue;
            float sx[B], sy[B];
#pragma unroll 1
            for (int h = 0; h < 2; ++h) {
                C1 v[B];
                float px[B], py[B];
                transform(4 * b + 2 * h, j, v);
#pragma unroll
                for (int r = 0; r < B; ++r) {
                    px[r] = __fmul_rn(v[r].re, s);
                    py[r] = __fmul_rn(v[r].im, s);
                }
                transform(4 * b + 2 * h + 1, j, v);
#pragma unroll
                for (int r = 0; r < B; ++r) {
                    px[r] = __fadd_rn(px[r], __fmul_rn(v[r].re, s));
                    py[r] = __fadd_rn(py[r], __fmul_rn(v[r].im, s));
                    sx[r] = h == 0 ? px[r] : __fadd_rn(sx[r], px[r]);
                    sy[r] = h == 0 ? py[r] : __fadd_rn(sy[r], py[r]);
                }
            }
            float* out = a.out_real + (int64_t)(line >> 2) * (a.Nx >> 1) + j;
#pragma unroll
            for (int r = 0; r < B; ++r)
                if (j + r * S < a.nout) out[r * S] = __fadd_rn(sx[r], sy[r]);
        }
    } else {
#pragma unroll 1
        for (int q = tid; q < TL * S; q += NT) {
            const int l = q / S, j = q - l * S;
            const uint32_t line = line0 + l;
            if (line >= a.nlines) continue;
            C1 v[B];
            transform(l, j, v);
            if constexpr (EPI == EPI_RL_RATIO) {
                // the loss and the model in code of their own: in the same loop
                // every iteration jumped over a logarithm per voxel (284 -> 259 us
                // at 150x600x700)
                if (a.partials || a.pred) c2r_store<EPI_PRED, ODD, B, S>(a, line, j, s, v, acc);
                else c2r_store<EPI, ODD, B, S>(a, line, j, s, v, acc);
            } else {
                c2r_store<EPI, ODD, B, S>(a, line, j, s, v, acc);
            }
        }
    }
    if constexpr (EPI == EPI_RL_RATIO) {
        if (a.partials) {
            const double t = block_sum(acc);
            if (tid == 0) a.partials[blockIdx.x] = t;
        }
    }
}

template <int L, bool ODD, bool KX = false>
XRegKernel xreg_r2c_of(int src) {
    using H = XRegShape<L, ODD>;
    constexpr int smem = H::template Ex<H::B>::bytes;
    switch (src) {
        case XS_ARRAY: return XRegKernel{(void*)k_xreg_r2c<L, ODD, XS_ARRAY, KX>, H::TL, H::NT, smem};
        case XS_UP2:
            if constexpr (!ODD) return XRegKernel{(void*)k_xreg_r2c<L, ODD, XS_UP2, KX>, H::TL, H::NT, smem};
            break;
        case XS_KERNEL:
            if constexpr (!KX)
                return XRegKernel{(void*)k_xreg_r2c<L, ODD, XS_KERNEL, KX>, H::TL, H::NT,
                                  smem + H::TL * L * (int)sizeof(float2)};
            break;
    }
    return XRegKernel{};
}

template <int L, bool ODD, bool KX = false>
XRegKernel xreg_c2r_of(int epi) {
    using H = XRegShape<L, ODD>;
    constexpr int smem = H::template Ex<H::S>::bytes;
    switch (epi) {
        case EPI_STORE: return XRegKernel{(void*)k_xreg_c2r<L, ODD, EPI_STORE, KX>, H::TL, H::NT, smem};
        case EPI_PRED:
        case EPI_RL_RATIO: return XRegKernel{(void*)k_xreg_c2r<L, ODD, EPI_RL_RATIO, KX>, H::TL, H::NT, smem};
        case EPI_RL_UPDATE: return XRegKernel{(void*)k_xreg_c2r<L, ODD, EPI_RL_UPDATE, KX>, H::TL, H::NT, smem};
        case EPI_DOWN2:
            if constexpr (!ODD) return XRegKernel{(void*)k_xreg_c2r<L, ODD, EPI_DOWN2, KX>, H::TL, H::NT, smem};
            break;
    }
    return XRegKernel{};
}

}  // namespace dk
