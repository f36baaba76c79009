// Register butterflies with literal roots: the radices 2..17 of the runtime-length kernels (qpd_any.cuh) and
// the compile-time passes built on them.
//
// Odd radices use the paired symmetric form, composite ones a prime-factor (Good-Thomas) or a small
// Cooley-Tukey split.  The roots are compile-time constants (a Taylor series evaluated in double by the
// compiler), so no table has to be uploaded per translation unit and device.
#pragma once

#include "qpd_common.cuh"

namespace qpd {

// cos and sin of 2 pi m / R at compile time, |error| below 1e-16: the angle is reduced to [-pi, pi], halved
// twice, and rebuilt with the double-angle formulas.
struct CosSin {
    double c, s;
};
__host__ __device__ constexpr CosSin unit_angle(int m, int R) {
    m %= R;
    if (2 * m > R) m -= R;
    const double a = 2.0 * 3.14159265358979323846 * (double)m / (double)R / 4.0;
    double c = 1.0, s = a, tc = 1.0, ts = a;
    for (int k = 1; k < 14; k++) {
        tc *= -a * a / (double)((2 * k - 1) * (2 * k));
        ts *= -a * a / (double)((2 * k) * (2 * k + 1));
        c += tc;
        s += ts;
    }
    for (int k = 0; k < 2; k++) {
        const double c2 = c * c - s * s, s2 = 2.0 * c * s;
        c = c2;
        s = s2;
    }
    return {c, s};
}

// Multiplications by literals and complex products stay scalar: a packed two-lane multiply needs its real factor
// in both halves of a register pair, which costs the moves that the packed form saves.
template <typename C, typename T> __device__ __forceinline__ C lit_scale(C a, T s) { return cmake<C>(a.x * s, a.y * s); }
template <typename C, typename T> __device__ __forceinline__ void lit_axpy(C& a, T s, C b) {
    a.x = fma(s, b.x, a.x);
    a.y = fma(s, b.y, a.y);
}
template <typename C> __device__ __forceinline__ C tw_mul(C w, C v) {
    return cmake<C>(fma(w.x, v.x, -(w.y * v.y)), fma(w.x, v.y, w.y * v.x));
}
template <typename C> __device__ __forceinline__ void fold_fma(C& a, C w, C v) {
    a.x = fma(w.x, v.x, fma(-w.y, v.y, a.x));
    a.y = fma(w.x, v.y, fma(w.y, v.x, a.y));
}

template <int R, typename C> struct Bfly;

template <typename C> struct Bfly<2, C> {
    __device__ __forceinline__ static void run(C (&x)[2]) {
        const C a = x[0];
        x[0] = cadd(a, x[1]);
        x[1] = csub(a, x[1]);
    }
};

template <typename C> struct Bfly<4, C> {
    __device__ __forceinline__ static void run(C (&x)[4]) {
        const C a = cadd(x[0], x[2]), b = csub(x[0], x[2]), c = cadd(x[1], x[3]), d = csub(x[1], x[3]);
        x[0] = cadd(a, c);
        x[2] = csub(a, c);
        x[1] = cadd_mi(b, d);
        x[3] = cadd_pi(b, d);
    }
};

template <typename C> struct Bfly<8, C> {
    __device__ __forceinline__ static void run(C (&x)[8]) {
        using T = decltype(C::x);
        const T r2 = T(0.70710678118654752440);
        C e[4] = {x[0], x[2], x[4], x[6]}, o[4] = {x[1], x[3], x[5], x[7]};
        Bfly<4, C>::run(e);
        Bfly<4, C>::run(o);
        const C t1 = lit_scale(cadd_mi(o[1], o[1]), r2);                    // exp(-i pi / 4) o1 = (1 - i) o1 / sqrt 2
        const C d3 = cadd_pi(o[3], o[3]);                                // (1 + i) o3
        const C t3 = lit_scale(d3, -r2);                                    // exp(-3 i pi / 4) o3 = -(1 + i) o3 / sqrt 2
        x[0] = cadd(e[0], o[0]);
        x[4] = csub(e[0], o[0]);
        x[1] = cadd(e[1], t1);
        x[5] = csub(e[1], t1);
        x[2] = cadd_mi(e[2], o[2]);
        x[6] = cadd_pi(e[2], o[2]);
        x[3] = cadd(e[3], t3);
        x[7] = csub(e[3], t3);
    }
};

// Odd primes: with a_r = x_r + x_{R-r} and b_r = -i (x_r - x_{R-r}),
//   X_s = x_0 + sum_r cos(2 pi r s / R) a_r + sum_r sin(2 pi r s / R) b_r, X_{R-s} the same with - sin.
template <int R, typename C> struct BflyOdd {
    __device__ __forceinline__ static void run(C (&x)[R]) {
        using T = decltype(C::x);
        constexpr int H = (R - 1) / 2;
        C a[H], b[H];
#pragma unroll
        for (int r = 1; r <= H; r++) {
            a[r - 1] = cadd(x[r], x[R - r]);
            b[r - 1] = cmake<C>(x[r].y - x[R - r].y, x[R - r].x - x[r].x);
        }
        const C x0 = x[0];
        C y = x0;
#pragma unroll
        for (int r = 0; r < H; r++) y = cadd(y, a[r]);
        x[0] = y;
#pragma unroll
        for (int s = 1; s <= H; s++) {
            C A = x0;
            C B = lit_scale(b[0], T(unit_angle(s, R).s));
            lit_axpy(A, T(unit_angle(s, R).c), a[0]);
#pragma unroll
            for (int r = 2; r <= H; r++) {
                lit_axpy(A, T(unit_angle(r * s, R).c), a[r - 1]);
                lit_axpy(B, T(unit_angle(r * s, R).s), b[r - 1]);
            }
            x[s] = cadd(A, B);
            x[R - s] = csub(A, B);
        }
    }
};
template <typename C> struct Bfly<3, C> : BflyOdd<3, C> {};
template <typename C> struct Bfly<5, C> : BflyOdd<5, C> {};
template <typename C> struct Bfly<7, C> : BflyOdd<7, C> {};
template <typename C> struct Bfly<11, C> : BflyOdd<11, C> {};
template <typename C> struct Bfly<13, C> : BflyOdd<13, C> {};
template <typename C> struct Bfly<17, C> : BflyOdd<17, C> {};

// Coprime A, B: input (B i + A j) mod AB is element (i, j) of a twiddle-free A x B transform, output k is
// element (k mod A, k mod B).
template <int A, int B, typename C> struct BflyPfa {
    __device__ __forceinline__ static void run(C (&x)[A * B]) {
        constexpr int N = A * B;
        C v[N];
#pragma unroll
        for (int j = 0; j < B; j++) {
            C t[A];
#pragma unroll
            for (int i = 0; i < A; i++) t[i] = x[(B * i + A * j) % N];
            Bfly<A, C>::run(t);
#pragma unroll
            for (int i = 0; i < A; i++) v[i * B + j] = t[i];
        }
#pragma unroll
        for (int i = 0; i < A; i++) {
            C t[B];
#pragma unroll
            for (int j = 0; j < B; j++) t[j] = v[i * B + j];
            Bfly<B, C>::run(t);
#pragma unroll
            for (int k = 0; k < N; k++)
                if (k % A == i) x[k] = t[k % B];
        }
    }
};
template <typename C> struct Bfly<6, C> : BflyPfa<2, 3, C> {};
template <typename C> struct Bfly<10, C> : BflyPfa<2, 5, C> {};
template <typename C> struct Bfly<12, C> : BflyPfa<4, 3, C> {};
template <typename C> struct Bfly<14, C> : BflyPfa<2, 7, C> {};
template <typename C> struct Bfly<15, C> : BflyPfa<3, 5, C> {};

// Q x Q Cooley-Tukey: x[Q i + j], twiddles exp(-2 pi i j k / Q^2) between the stages, output k + Q s.
template <int Q, typename C> struct BflySquare {
    __device__ __forceinline__ static void run(C (&x)[Q * Q]) {
        using T = decltype(C::x);
        C v[Q * Q];
#pragma unroll
        for (int j = 0; j < Q; j++) {
            C t[Q];
#pragma unroll
            for (int i = 0; i < Q; i++) t[i] = x[Q * i + j];
            Bfly<Q, C>::run(t);
#pragma unroll
            for (int k = 0; k < Q; k++)
                v[k * Q + j] = j * k == 0 ? t[k]
                                          : tw_mul(cmake<C>(T(unit_angle(j * k, Q * Q).c), T(-unit_angle(j * k, Q * Q).s)), t[k]);
        }
#pragma unroll
        for (int k = 0; k < Q; k++) {
            C t[Q];
#pragma unroll
            for (int j = 0; j < Q; j++) t[j] = v[k * Q + j];
            Bfly<Q, C>::run(t);
#pragma unroll
            for (int s = 0; s < Q; s++) x[k + Q * s] = t[s];
        }
    }
};
template <typename C> struct Bfly<9, C> : BflySquare<3, C> {};
template <typename C> struct Bfly<16, C> : BflySquare<4, C> {};

constexpr int kMaxBfly = 17;

}  // namespace qpd
