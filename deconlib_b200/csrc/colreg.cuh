// Column FFT pass (Y and axial passes) with the transform in registers.
//
// A tile is T adjacent kx columns of one plane.  An axis of L = R1 x R2 points
// runs as two register DFTs: thread (t, j) takes the R1 points j + r R2 of
// column t (rows past the signal are known zeros), transforms them, exchanges
// once through shared memory and transforms R2 points, which leaves it with
// the spectrum at j + r R1.  The axial pass multiplies by the OTF right there
// and runs the inverse with the radices in reverse, whose first stage needs
// exactly the points the thread holds: two exchanges for the whole pass.
// Results go from registers to global memory in whole row pieces.
//
// The kernel is persistent and its loads run one tile ahead: a TMA copy brings
// the next tile's rows into the input buffer as soon as every thread has taken
// this tile's points out of it, and the next OTF tile as soon as the product
// is formed, so no thread waits for HBM while the SM has arithmetic to do.
// Loading straight into registers instead left the warps on the loads for
// ~45 % of the issue slots (axial pass at 256 points, canvas 256x512x512:
// 150 us; with the TMA buffers 118 us on spectra of its own, 128 us between the
// other passes: 539 MB, 4.2 TB/s; 141 us for the shared-memory FFT before).
// Bound by latency at 0.65 instructions per cycle and scheduler; neither more
// warps (64 registers), nor half the threads for R2 = 2 R1, which idle in that
// stage, nor two columns per thread was faster over the lengths.  Shared-memory
// rows are 128 bytes (T = 16) or 64 (T = 8), read by half-warps in whole rows,
// so no swizzle is needed; the exchange buffer is separate from the input
// buffer, which is what frees the latter early.
#pragma once

#include "codelets.cuh"
#include "conv_impl.cuh"
#include "tma.cuh"

namespace dk {

enum ColRegMode { CR_FWD = 0, CR_INV = 1, CR_OTF = 2, CR_OTF16 = 3 };

template <int L, int MODE>
struct ColRegShape {
    static constexpr int R1 = small_radix(L), R2 = L / R1;
    static constexpr bool OTF = MODE == CR_OTF || MODE == CR_OTF16;
    // 16 columns per tile while two CTAs fit an SM (axial pass: three buffers;
    // Y passes: registers of the longer DFT).  The axial pass strides whole
    // planes, where 64-byte pieces cost DRAM efficiency (200 points over a
    // 200x720x800 canvas: 216 us with 16 columns, 288 us with 8); in the Y
    // passes 8 columns give more CTAs to overlap (240 points: 11.0 vs 11.7 us).
    static constexpr int T = OTF ? (L <= 360 ? 16 : 8) : (R2 < 15 ? 16 : 8);
    static constexpr int NT = T * R2;
    // 64-byte rows: an odd step between the rows of one exchange keeps the two
    // rows of a half-warp on different banks
    static constexpr int pad1 = (T == 8 && R1 % 2 == 0) ? 1 : 0;
    static constexpr int pad2 = (T == 8 && R2 % 2 == 0) ? 1 : 0;
    static constexpr int rows1 = R2 * (R1 + pad1), rows2 = OTF ? R1 * (R2 + pad2) : 0;
    static constexpr int exch = ((rows1 > rows2 ? rows1 : rows2) * T * (int)sizeof(float2) + 127) / 128 * 128;
    // registers per thread that the CTAs per SM are chosen for: the shorter
    // the DFT the more warps fit; 80 hold up to 32 points without spills
    static constexpr int regs = R2 <= 10 ? 64 : (R2 <= 32 ? 80 : 128);
    static constexpr int blocks = 65536 / (NT * regs) < 1 ? 1 : 65536 / (NT * regs);
};

// Rows n < count of one lane's column into shared memory, eight loads in
// flight per thread (each row is a sector of its own: with one load at a time
// these few tiles ran 10 us past the rest of the pass).
template <int STEP, int T, typename V>
__device__ __forceinline__ void gather_rows(V* sm, const V* __restrict__ src, int64_t js, int j, int t,
                                            int count, bool ok) {
    for (int n0 = j; n0 < count; n0 += 8 * STEP) {
        V v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            v[i] = V{};
            if (ok && n0 + i * STEP < count) v[i] = src[(n0 + i * STEP) * js];
        }
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (n0 + i * STEP < count) sm[(n0 + i * STEP) * T + t] = v[i];
    }
}

// PLAIN: every tile by plain loads (a plan without tensor maps); nfull tiles of a
// plane's rem columns.  A kernel of its own: as a run-time choice it cost the TMA
// path 0.5-1.5 %.
template <int L, int MODE, bool PLAIN>
__global__ void __launch_bounds__(ColRegShape<L, MODE>::NT, ColRegShape<L, MODE>::blocks)
    k_colreg(const __grid_constant__ ColRegArgs a) {
    using S = ColRegShape<L, MODE>;
    constexpr int R1 = S::R1, R2 = S::R2, T = S::T;
    constexpr int D = MODE == CR_INV ? +1 : -1;
    constexpr bool OTF = S::OTF;
    extern __shared__ __align__(128) unsigned char smraw[];
    float2* ex = reinterpret_cast<float2*>(smraw);             // exchange buffer
    float2* in = reinterpret_cast<float2*>(smraw + S::exch);   // input rows
    unsigned char* ot = smraw + S::exch + a.in_bytes;          // OTF rows (float2 or half2)
    __shared__ uint64_t full, obar;
    const int tid = threadIdx.x, t = tid % T, j = tid / T;
    if (tid == 0) {
        mbar_init(&full, 1);
        if constexpr (OTF) mbar_init(&obar, 1);
        fence_proxy_async_smem();
    }
    __syncthreads();
    chain_enter();

    // full tiles come by TMA; the tiles of the last Hx % T columns, which hold
    // several planes side by side, by plain loads
    auto issue = [&](int tile) {
        const int o = tile / a.nfull, c0 = (tile - o * a.nfull) * 2 * T;
        mbar_expect_tx(&full, (uint32_t)(a.nbox * a.box * T * sizeof(float2)));
        for (int i = 0; i < a.nbox; ++i) {
            const int r0 = i * a.box;
            if (a.jdim == 1) tma_load_3d(in + r0 * T, &a.srcmap, c0, r0, o, &full);
            else tma_load_3d(in + r0 * T, &a.srcmap, c0, o, r0, &full);
        }
    };
    auto issue_otf = [&](int tile) {
        const int o = tile / a.nfull, c0 = (tile - o * a.nfull) * T;
        constexpr int row = MODE == CR_OTF16 ? T * (int)sizeof(__half2) : T * (int)sizeof(float2);
        constexpr int cs = MODE == CR_OTF16 ? 1 : 2;  // map elements per complex value
        mbar_expect_tx(&obar, (uint32_t)(a.onbox * a.obox * row));
        for (int i = 0; i < a.onbox; ++i) {
            const int r0 = i * a.obox;
            if (a.jdim == 1) tma_load_3d(ot + r0 * row, &a.otfmap, c0 * cs, r0, o, &obar);
            else tma_load_3d(ot + r0 * row, &a.otfmap, c0 * cs, o, r0, &obar);
        }
    };
    if (!PLAIN && tid == 0 && (int)blockIdx.x < a.nmain) {
        issue(blockIdx.x);
        if constexpr (OTF) issue_otf(blockIdx.x);
    }

    uint32_t ph = 0;
    int pending = -1;  // parity of the row copy a CTA that gives up still waits for
    for (int tile = blockIdx.x; tile < a.ntiles; tile += gridDim.x, ph ^= 1) {
        const bool main = !PLAIN && tile < a.nmain;
        const bool more = !PLAIN && tile + (int)gridDim.x < a.nmain;
        int o, kx;
        bool ok = true;
        if (main || PLAIN) {
            o = tile / a.nfull;
            kx = (tile - o * a.nfull) * T + t;
            if constexpr (PLAIN) ok = kx < a.rem;
        } else {
            const int p = t / a.rem;
            o = (tile - a.nmain) * a.per + p;
            kx = a.nfull * T + t - p * a.rem;
            ok = p < a.per && o < a.nouter;
        }

        C1 v[R2 > R1 ? R2 : R1];
        bool arrived = true;
        if (main) {
            arrived = mbar_wait_bounded(&full, ph, a.flag);
        } else {
            // no copy is in flight any more: every thread has passed the last
            // full tile's barriers, or there was none
            __syncthreads();
            const float2* src = a.src + o * a.src_os + kx;
            gather_rows<R2, T>(in, src, a.src_js, j, t, a.nin, ok);
            if constexpr (MODE == CR_OTF)
                gather_rows<R2, T>(reinterpret_cast<float2*>(ot), a.otf + o * a.otf_os + kx, a.otf_js, j, t, L, ok);
            if constexpr (MODE == CR_OTF16)
                gather_rows<R2, T>(reinterpret_cast<__half2*>(ot), a.otf16 + o * a.otf_os + kx, a.otf_js, j, t, L, ok);
            __syncthreads();
        }
        if (j < R2) {
#pragma unroll
            for (int r = 0; r < R1; ++r)
                v[r] = as_c1(j + r * R2 < a.nin ? in[(j + r * R2) * T + t] : make_float2(0.f, 0.f));
        }
        // the refill is an async-proxy write over what the threads just read:
        // each orders its reads before it, then the barrier
        fence_proxy_async_smem();
        if (!__syncthreads_and(arrived)) {
            pending = ph;
            break;
        }
        if (tid == 0 && more) issue(tile + gridDim.x);
        if (j < R2) {
            dftn<R1, D>(v);
#pragma unroll
            for (int r = 0; r < R1; ++r) ex[(j * (R1 + S::pad1) + r) * T + t] = as_f2(v[r]);
        }
        __syncthreads();
        if (j < R1) {
#pragma unroll
            for (int r = 0; r < R2; ++r) {
                v[r] = as_c1(ex[(j + r * (R1 + S::pad1)) * T + t]);
                if (r > 0) v[r] = twist<(D > 0)>(v[r], __ldg(&a.tw[(r * j) * a.tws]));
            }
            dftn<R2, D>(v);
        }
        float2* dst = a.dst + o * a.dst_os + kx + j * a.dst_js;
        const int lim = ok ? a.nout : 0;
        if constexpr (!OTF) {
            if (j < R1) {
                const int64_t step = R1 * a.dst_js;
#pragma unroll
                for (int r = 0; r < R2; ++r)
                    if (j + r * R1 < lim) dst[r * step] = as_f2(v[r]);
            }
        } else {
            if (main) arrived = mbar_wait_bounded(&obar, ph, a.flag);
            if (j < R1) {
#pragma unroll
                for (int r = 0; r < R2; ++r) {
                    const int kz = j + r * R1;
                    float2 w;
                    if constexpr (MODE == CR_OTF) {
                        w = reinterpret_cast<const float2*>(ot)[kz * T + t];
                    } else {
                        w = __half22float2(reinterpret_cast<const __half2*>(ot)[kz * T + t]);
                        w = cscale(w, __ldg(a.otf_inv + kz));
                    }
                    w.y *= a.conj;
                    v[r] = twist<false>(v[r], w);
                }
            }
            // the inverse's twiddles are loaded again: kept across the product
            // they would cost the registers of a whole DFT
            const float2* tw = a.tw;
            asm volatile("" : "+l"(tw));
            fence_proxy_async_smem();
            if (!__syncthreads_and(arrived)) {
                pending = more ? ph ^ 1 : ph;
                break;
            }
            if (tid == 0 && more) issue_otf(tile + gridDim.x);
            if (j < R1) {
                dftn<R2, +1>(v);
#pragma unroll
                for (int r = 0; r < R2; ++r) ex[(j * (R2 + S::pad2) + r) * T + t] = as_f2(v[r]);
            }
            __syncthreads();
            if (j < R2) {
#pragma unroll
                for (int r = 0; r < R1; ++r) {
                    v[r] = as_c1(ex[(j + r * (R2 + S::pad2)) * T + t]);
                    if (r > 0) v[r] = twist<true>(v[r], __ldg(&tw[(r * j) * a.tws]));
                }
                dftn<R1, +1>(v);
                const int64_t step = R2 * a.dst_js;
#pragma unroll
                for (int r = 0; r < R1; ++r)
                    if (j + r * R2 < lim) dst[r * step] = as_f2(v[r]);
            }
        }
    }
    if (pending >= 0 && tid == 0) {
        mbar_drain(&full, pending);
        if constexpr (OTF) mbar_drain(&obar, ph);
    }
}

template <int L, int MODE>
ColRegKernel colreg_one(bool plain) {
    using S = ColRegShape<L, MODE>;
    if constexpr (MODE != CR_OTF16)
        if (plain) return ColRegKernel{(void*)k_colreg<L, MODE, true>, S::T, S::NT, S::exch};
    return ColRegKernel{(void*)k_colreg<L, MODE, false>, S::T, S::NT, S::exch};
}

template <int L>
ColRegKernel colreg_kernel(int mode, bool plain) {
    switch (mode) {
        case CR_FWD: return colreg_one<L, CR_FWD>(plain);
        case CR_INV: return colreg_one<L, CR_INV>(plain);
        case CR_OTF: return colreg_one<L, CR_OTF>(plain);
        case CR_OTF16:
            if constexpr (L == 64 || L == 128 || L == 256) return colreg_one<L, CR_OTF16>(false);
    }
    return ColRegKernel{};
}

}  // namespace dk
