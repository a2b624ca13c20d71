// Register DFTs of composite length, and the split of an axis length into two
// of them.
//
// dftn<N, DIR>(v) transforms N complex values held by one thread, natural
// order in and out, unnormalised.  Two columns per thread in packed f32x2
// instructions halve the issue slots of the arithmetic but not its pipe time,
// and double the registers: no gain (axial pass at 256 points 115 us against
// 118 in the layout that suits them best).  N is a product of the primitive
// codelets 2, 3, 4, 5, 8, 16: co-prime factors combine without twiddles
// (prime-factor indexing, Good 1958), the others by one Cooley-Tukey step
// with twiddles that are compile-time constants.
#pragma once

#include <type_traits>
#include <utility>

#include "common.cuh"

namespace dk {

struct C1 {
    float re, im;
};
__device__ __forceinline__ C1 operator+(C1 a, C1 b) {
    return C1{a.re + b.re, a.im + b.im};
}
__device__ __forceinline__ C1 operator-(C1 a, C1 b) {
    return C1{a.re - b.re, a.im - b.im};
}
// a + DIR i b
template <int DIR>
__device__ __forceinline__ C1 add_i(C1 a, C1 b) {
    return DIR > 0 ? C1{a.re - b.im, a.im + b.re} : C1{a.re + b.im, a.im - b.re};
}
// a * (c + DIR i s)
template <int DIR>
__device__ __forceinline__ C1 spin(C1 a, float c, float s) {
    const float d = DIR > 0 ? s : -s;
    return C1{fmaf(a.re, c, a.im * -d), fmaf(a.im, c, a.re * d)};
}
// a * w, or a * conj(w)
template <bool CONJ>
__device__ __forceinline__ C1 twist(C1 a, float2 w) {
    return spin<CONJ ? -1 : +1>(a, w.x, w.y);
}

__device__ __forceinline__ C1 as_c1(float2 v) { return C1{v.x, v.y}; }
__device__ __forceinline__ float2 as_f2(C1 v) { return make_float2(v.re, v.im); }
__device__ __forceinline__ C1 conj_of(C1 v) { return C1{v.re, -v.im}; }

// ---- compile-time trigonometry ----------------------------------------------

// cos(2 pi m / n), in double: exact reduction to the first octant, then the
// Taylor series (argument <= pi / 4, terms down to 1e-18).
constexpr double turn_series(double x, bool sine) {
    double t = sine ? x : 1.0, s = t;
    for (int i = 1; i < 12; ++i) {
        const double k = sine ? 2.0 * i * (2.0 * i + 1.0) : 2.0 * i * (2.0 * i - 1.0);
        t *= -x * x / k;
        s += t;
    }
    return s;
}
constexpr double cos_turn(int m, int n) {
    m %= n;
    if (m < 0) m += n;
    if (2 * m > n) m = n - m;
    double sign = 1.0;
    if (4 * m > n) {  // cos(pi - a) = -cos a
        sign = -1.0;
        m = n - 2 * m;
        n = 2 * n;
    }
    constexpr double kTurn = 6.283185307179586476925287;
    if (8 * m > n) return sign * turn_series(kTurn * (n - 4 * m) / (4.0 * n), true);
    return sign * turn_series(kTurn * m / n, false);
}
constexpr double sin_turn(int m, int n) { return cos_turn(4 * m - n, 4 * n); }

// v * exp(DIR 2 pi i M / N)
template <int N, int M, int DIR>
__device__ __forceinline__ C1 turn(C1 v) {
    constexpr int m = ((M % N) + N) % N;
    if constexpr (m == 0) {
        return v;
    } else {
        constexpr float c = (float)cos_turn(m, N), s = (float)sin_turn(m, N);
        return spin<DIR>(v, c, s);
    }
}

// ---- codelets -----------------------------------------------------------------

__device__ __forceinline__ void dft_2(C1& a, C1& b) {
    const C1 t = a;
    a = t + b;
    b = t - b;
}
template <int DIR>
__device__ __forceinline__ void dft_4(C1& a, C1& b, C1& c, C1& d) {
    const C1 t0 = a + c, t1 = a - c, t2 = b + d, t3 = b - d;
    a = t0 + t2;
    c = t0 - t2;
    b = add_i<DIR>(t1, t3);
    d = add_i<-DIR>(t1, t3);
}
template <int DIR>
__device__ __forceinline__ void dft_3(C1* v) {
    constexpr float s3 = (float)sin_turn(1, 3);
    const C1 s = v[1] + v[2], d = v[1] - v[2];
    const C1 m{fmaf(s.re, -0.5f, v[0].re), fmaf(s.im, -0.5f, v[0].im)};
    constexpr float k = DIR > 0 ? s3 : -s3;
    v[0] = v[0] + s;
    v[1] = C1{fmaf(d.im, -k, m.re), fmaf(d.re, k, m.im)};
    v[2] = C1{fmaf(d.im, k, m.re), fmaf(d.re, -k, m.im)};
}
template <int DIR>
__device__ __forceinline__ void dft_5(C1* v) {
    constexpr float c1 = (float)cos_turn(1, 5), c2 = (float)cos_turn(2, 5);
    constexpr float s1 = DIR > 0 ? (float)sin_turn(1, 5) : -(float)sin_turn(1, 5);
    constexpr float s2 = DIR > 0 ? (float)sin_turn(2, 5) : -(float)sin_turn(2, 5);
    const C1 b1 = v[1] + v[4], b2 = v[2] + v[3], d1 = v[1] - v[4], d2 = v[2] - v[3];
    const C1 t1{fmaf(b2.re, c2, fmaf(b1.re, c1, v[0].re)), fmaf(b2.im, c2, fmaf(b1.im, c1, v[0].im))};
    const C1 t2{fmaf(b2.re, c1, fmaf(b1.re, c2, v[0].re)), fmaf(b2.im, c1, fmaf(b1.im, c2, v[0].im))};
    v[0] = v[0] + (b1 + b2);
    // i u, u = s1 d1 + s2 d2 and s2 d1 - s1 d2
    const C1 u1{fmaf(d2.re, s2, d1.re * s1), fmaf(d2.im, s2, d1.im * s1)};
    const C1 u2{fmaf(d2.re, -s1, d1.re * s2), fmaf(d2.im, -s1, d1.im * s2)};
    v[1] = add_i<+1>(t1, u1);
    v[4] = add_i<-1>(t1, u1);
    v[2] = add_i<+1>(t2, u2);
    v[3] = add_i<-1>(t2, u2);
}
template <int DIR>
__device__ __forceinline__ void dft_8(C1* v) {
    constexpr float h = (float)cos_turn(1, 8);
    dft_4<DIR>(v[0], v[2], v[4], v[6]);
    dft_4<DIR>(v[1], v[3], v[5], v[7]);
    // odd half: times W8^1 = h (1 + DIR i), W8^2 = DIR i, W8^3 = h (-1 + DIR i);
    // the factor h goes into the last additions
    const C1 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6];
    const C1 o0 = v[1], o2 = v[5];
    const C1 p = add_i<DIR>(v[3], v[3]);   // (1 + DIR i) o1
    const C1 q = add_i<-DIR>(v[7], v[7]);  // (1 - DIR i) o3 = -(-1 + DIR i) o3
    v[0] = e0 + o0;
    v[4] = e0 - o0;
    v[2] = add_i<DIR>(e2, o2);
    v[6] = add_i<-DIR>(e2, o2);
    v[1] = C1{fmaf(p.re, h, e1.re), fmaf(p.im, h, e1.im)};
    v[5] = C1{fmaf(p.re, -h, e1.re), fmaf(p.im, -h, e1.im)};
    v[3] = C1{fmaf(q.re, -h, e3.re), fmaf(q.im, -h, e3.im)};
    v[7] = C1{fmaf(q.re, h, e3.re), fmaf(q.im, h, e3.im)};
}

template <class Fn, int... I>
__device__ __forceinline__ void unrolled(Fn f, std::integer_sequence<int, I...>) {
    (f(std::integral_constant<int, I>{}), ...);
}

constexpr int gcd_of(int a, int b) { return b == 0 ? a : gcd_of(b, a % b); }
// inverse of a modulo m (gcd 1)
constexpr int inverse_mod(int a, int m) {
    for (int x = 1; x < m; ++x)
        if ((a * x) % m == 1) return x;
    return 0;
}
// First factor of the composite codelets (0: primitive).
constexpr int codelet_split(int n) {
    switch (n) {
        case 6: return 2;
        case 9: return 3;
        case 10: return 2;
        case 12: return 4;
        case 15: return 3;
        case 16: return 4;
        case 18: return 2;
        case 20: return 4;
        case 24: return 8;
        case 25: return 5;
        case 27: return 3;
        case 30: return 2;
        case 32: return 4;
        case 36: return 4;
        case 40: return 8;
        default: return 0;
    }
}

template <int N, int DIR>
__device__ __forceinline__ void dftn(C1* v) {
    constexpr int A = codelet_split(N);
    if constexpr (N == 1) {
    } else if constexpr (N == 2) {
        dft_2(v[0], v[1]);
    } else if constexpr (N == 3) {
        dft_3<DIR>(v);
    } else if constexpr (N == 4) {
        dft_4<DIR>(v[0], v[1], v[2], v[3]);
    } else if constexpr (N == 5) {
        dft_5<DIR>(v);
    } else if constexpr (N == 8) {
        dft_8<DIR>(v);
    } else if constexpr (gcd_of(A, N / A) == 1) {
        // n = (B n1 + A n2) mod N;  k = k1 mod A, k2 mod B
        constexpr int B = N / A;
        constexpr int EA = B * inverse_mod(B % A, A), EB = A * inverse_mod(A % B, B);
        C1 y[A][B];
#pragma unroll
        for (int n1 = 0; n1 < A; ++n1) {
#pragma unroll
            for (int n2 = 0; n2 < B; ++n2) y[n1][n2] = v[(B * n1 + A * n2) % N];
            dftn<B, DIR>(y[n1]);
        }
#pragma unroll
        for (int k2 = 0; k2 < B; ++k2) {
            C1 t[A];
#pragma unroll
            for (int n1 = 0; n1 < A; ++n1) t[n1] = y[n1][k2];
            dftn<A, DIR>(t);
#pragma unroll
            for (int k1 = 0; k1 < A; ++k1) v[(EA * k1 + EB * k2) % N] = t[k1];
        }
    } else {
        // n = n1 + A n2;  k = k2 + B k1
        constexpr int B = N / A;
        C1 y[A][B];
        unrolled([&](auto i1) {
            constexpr int n1 = decltype(i1)::value;
#pragma unroll
            for (int n2 = 0; n2 < B; ++n2) y[n1][n2] = v[n1 + A * n2];
            dftn<B, DIR>(y[n1]);
            unrolled([&](auto i2) {
                constexpr int k2 = decltype(i2)::value;
                y[n1][k2] = turn<N, n1 * k2, DIR>(y[n1][k2]);
            }, std::make_integer_sequence<int, B>{});
        }, std::make_integer_sequence<int, A>{});
#pragma unroll
        for (int k2 = 0; k2 < B; ++k2) {
            C1 t[A];
#pragma unroll
            for (int n1 = 0; n1 < A; ++n1) t[n1] = y[n1][k2];
            dftn<A, DIR>(t);
#pragma unroll
            for (int k1 = 0; k1 < A; ++k1) v[k2 + B * k1] = t[k1];
        }
    }
}

constexpr bool is_codelet(int n) {
    return n == 2 || n == 3 || n == 4 || n == 5 || n == 8 || codelet_split(n) != 0;
}

// The smaller radix s of an axis length L = s x big, the two as equal as the
// codelets allow with s <= most (0: no such pair).
constexpr int small_radix(int L, int most = 40) {
    int best = 0;
    for (int s = 2; s * s <= L && s <= most; ++s)
        if (L % s == 0 && is_codelet(s) && is_codelet(L / s)) best = s;
    return best;
}

// Every 5-smooth length from 16 to 1024: each has a pair of codelets.
#define DK_PAIR_LENGTHS_A(X) \
    X(16) X(18) X(20) X(24) X(25) X(27) X(30) X(32) X(36) X(40) X(45) X(48) X(50) X(54) X(60) X(64) X(72) \
    X(75) X(80) X(81) X(90) X(96)
#define DK_PAIR_LENGTHS_B(X) \
    X(100) X(108) X(120) X(125) X(128) X(135) X(144) X(150) X(160) X(162) X(180) X(192) X(200) X(216) X(225)
#define DK_PAIR_LENGTHS_C(X) \
    X(240) X(243) X(250) X(256) X(270) X(288) X(300) X(320) X(324) X(360) X(375) X(384) X(400)
#define DK_PAIR_LENGTHS_D(X) \
    X(405) X(432) X(450) X(480) X(486) X(500) X(512) X(540) X(576) X(600) X(625)
#define DK_PAIR_LENGTHS_E(X) \
    X(640) X(648) X(675) X(720) X(729) X(750) X(768) X(800) X(810) X(864) X(900) X(960) X(972) X(1000) X(1024)

// X lines: even Fx = 2 L up to 2048, and the odd 5-smooth Fx.
#define DK_XREG_LENGTHS_a(X) \
    X(16) X(18) X(20) X(24) X(25) X(27) X(30) X(32) X(36) X(40) X(45) X(48) X(50) X(54) X(60) X(64) X(72)
#define DK_XREG_LENGTHS_b(X) X(75) X(80) X(81) X(90) X(96) X(100) X(108) X(120) X(125) X(128) X(135) X(144) X(150)
#define DK_XREG_LENGTHS_c(X) X(160) X(162) X(180) X(192) X(200) X(216) X(225) X(240) X(243) X(250)
#define DK_XREG_LENGTHS_d(X) X(256) X(270) X(288) X(300) X(320) X(324) X(360) X(375)
#define DK_XREG_LENGTHS_e(X) X(384) X(400) X(405) X(432) X(450) X(480) X(486) X(500) X(512)
#define DK_XREG_LENGTHS_f(X) X(540) X(576) X(600) X(625) X(640) X(648) X(675) X(720) X(729) X(750)
#define DK_XREG_LENGTHS_g(X) X(768) X(800) X(810) X(864) X(900) X(960) X(972) X(1000) X(1024)
// kx-major spectrum (the fused Y / axial pass): 2^a x {1, 3, 5, 15}, the lengths
// that had compile-time kernels for it; the others run on runtime radices.
#define DK_XREG_LENGTHS_kx(X) \
    X(64) X(80) X(96) X(128) X(160) X(192) X(240) X(256) X(320) X(384) X(480) X(512) X(640) X(768) X(960) X(1024)
#define DK_XREG_LENGTHS_odd(X) \
    X(25) X(27) X(45) X(75) X(81) X(125) X(135) X(225) X(243) X(375) X(405) X(625) X(675) X(729)

#define DK_PAIR_CHECK(n) static_assert(small_radix(n) >= 2, "length without a codelet pair");
DK_PAIR_LENGTHS_A(DK_PAIR_CHECK)
DK_PAIR_LENGTHS_B(DK_PAIR_CHECK)
DK_PAIR_LENGTHS_C(DK_PAIR_CHECK)
DK_PAIR_LENGTHS_D(DK_PAIR_CHECK)
DK_PAIR_LENGTHS_E(DK_PAIR_CHECK)
#undef DK_PAIR_CHECK

}  // namespace dk
