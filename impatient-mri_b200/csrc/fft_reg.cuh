// Forward DFTs of R points in registers (natural order in and out) for the
// grid FFT and the F^H F engine.  Powers of two are a radix-2 DIT network on
// bit-reversed registers, 3, 5 and 7 direct transforms on the symmetric and
// antisymmetric pairs, other R = A B a compile-time Cooley-Tukey step with A
// the smallest odd prime factor.  All twiddles are compile-time constants
// (Taylor series evaluated by the compiler), so they become immediates.
// The inverse of a vector is the forward of the vector with real and
// imaginary parts exchanged, exchanged back (swap_ri).
#pragma once
#include <cuda_runtime.h>

namespace imp {
namespace fftr {

__host__ __device__ constexpr double csin(double x) {
    double term = x, sum = x;
    for (int k = 1; k < 30; ++k) {
        term *= -x * x / ((2.0 * k) * (2.0 * k + 1.0));
        sum += term;
    }
    return sum;
}
__host__ __device__ constexpr double ccos(double x) {
    double term = 1.0, sum = 1.0;
    for (int k = 1; k < 30; ++k) {
        term *= -x * x / ((2.0 * k - 1.0) * (2.0 * k));
        sum += term;
    }
    return sum;
}

__host__ __device__ constexpr int log2c(int n) { return n <= 1 ? 0 : 1 + log2c(n >> 1); }
__host__ __device__ constexpr int bitrevc(int i, int bits) {
    int r = 0;
    for (int b = 0; b < bits; ++b) r |= ((i >> b) & 1) << (bits - 1 - b);
    return r;
}
__host__ __device__ constexpr int odd_factor(int n) {
    for (int p = 3; p <= n; p += 2)
        if (n % p == 0) return p;
    return 1;
}

__device__ __forceinline__ float2 swap_ri(float2 v, bool on) {
    return on ? make_float2(v.y, v.x) : v;
}

// v * exp(-2 pi i NUM / DEN) with a compile-time angle
template <int NUM, int DEN>
__device__ __forceinline__ float2 mulw(float2 v) {
    constexpr int m = ((NUM % DEN) + DEN) % DEN;
    if constexpr (m == 0) {
        return v;
    } else if constexpr (4 * m == DEN) {
        return make_float2(v.y, -v.x);
    } else if constexpr (2 * m == DEN) {
        return make_float2(-v.x, -v.y);
    } else if constexpr (4 * m == 3 * DEN) {
        return make_float2(-v.y, v.x);
    } else {
        constexpr double ang = -2.0 * 3.14159265358979323846264338327950288 * m / DEN;
        constexpr float c = (float)ccos(ang), s = (float)csin(ang);
        return make_float2(v.x * c - v.y * s, v.x * s + v.y * c);
    }
}

// a' = a + w b, b' = a - w b with w = exp(-2 pi i K / DEN), DEN = 2 HALF.  For a
// general w the larger of its parts is taken out, w = c (1 + i t) or s (t + i)
// with |t| <= 1 (the scaled butterfly of Linzer and Feig, 1993): two FMAs form
// (1 + i t) b and four the outputs, instead of eight multiplications and additions
// (a tenth of a transform's instructions), with one rounding less.
template <int K, int DEN>
__device__ __forceinline__ void butterfly(float2 &a, float2 &b) {
    if constexpr (K == 0 || 4 * K == DEN) {
        const float2 u = mulw<K, DEN>(b);
        b = make_float2(a.x - u.x, a.y - u.y);
        a = make_float2(a.x + u.x, a.y + u.y);
    } else {
        constexpr double ang = -2.0 * 3.14159265358979323846264338327950288 * K / DEN;
        constexpr double cd = ccos(ang), sd = csin(ang);
        constexpr bool big_c = cd * cd >= sd * sd;
        constexpr float m = (float)(big_c ? cd : sd), t = (float)(big_c ? sd / cd : cd / sd);
        const float2 u = big_c ? make_float2(fmaf(-t, b.y, b.x), fmaf(t, b.x, b.y))
                               : make_float2(fmaf(t, b.x, -b.y), fmaf(t, b.y, b.x));
        b = make_float2(fmaf(-m, u.x, a.x), fmaf(-m, u.y, a.y));
        a = make_float2(fmaf(m, u.x, a.x), fmaf(m, u.y, a.y));
    }
}

template <int R, int HALF, int K>
__device__ __forceinline__ void p2_stage(float2 (&v)[R]) {
    if constexpr (HALF < R) {
        if constexpr (K < HALF) {
#pragma unroll
            for (int i = 0; i < R; i += 2 * HALF) butterfly<K, 2 * HALF>(v[i + K], v[i + K + HALF]);
            p2_stage<R, HALF, K + 1>(v);
        } else {
            p2_stage<R, 2 * HALF, 0>(v);
        }
    }
}

// Odd prime P: outputs k and P - k share the pair sums s_j = x_j + x_{P-j},
// d_j = x_j - x_{P-j}: X_k = x_0 + sum s_j cos - i sum d_j sin, X_{P-k} the
// same with + i.
template <int P, int K, int J>
__device__ __forceinline__ void odd_acc(const float2 (&s)[P / 2], const float2 (&d)[P / 2],
                                        float2 &a, float2 &b) {
    if constexpr (J <= P / 2) {
        constexpr double ang = 2.0 * 3.14159265358979323846264338327950288 * ((J * K) % P) / P;
        constexpr float c = (float)ccos(ang), sn = (float)csin(ang);
        a.x = fmaf(s[J - 1].x, c, a.x);
        a.y = fmaf(s[J - 1].y, c, a.y);
        b.x = fmaf(d[J - 1].y, sn, b.x);
        b.y = fmaf(-d[J - 1].x, sn, b.y);
        odd_acc<P, K, J + 1>(s, d, a, b);
    }
}

template <int P, int K>
__device__ __forceinline__ void odd_out(float2 (&v)[P], float2 x0, const float2 (&s)[P / 2],
                                        const float2 (&d)[P / 2]) {
    if constexpr (K <= P / 2) {
        float2 a = x0, b = make_float2(0.f, 0.f);
        odd_acc<P, K, 1>(s, d, a, b);
        v[K] = make_float2(a.x + b.x, a.y + b.y);
        v[P - K] = make_float2(a.x - b.x, a.y - b.y);
        odd_out<P, K + 1>(v, x0, s, d);
    }
}

template <int R>
__device__ __forceinline__ void dft(float2 (&v)[R]);

// u_k1 *= w_R^{J2 k1}
template <int R, int A, int J2, int K1>
__device__ __forceinline__ void ct_twid(float2 (&u)[A]) {
    if constexpr (K1 < A) {
        u[K1] = mulw<J2 * K1, R>(u[K1]);
        ct_twid<R, A, J2, K1 + 1>(u);
    }
}

template <int R, int A, int J2>
__device__ __forceinline__ void ct_inner(float2 (&v)[R]) {
    constexpr int B = R / A;
    if constexpr (J2 < B) {
        float2 u[A];
#pragma unroll
        for (int j = 0; j < A; ++j) u[j] = v[B * j + J2];
        dft<A>(u);
        ct_twid<R, A, J2, 1>(u);
#pragma unroll
        for (int k = 0; k < A; ++k) v[B * k + J2] = u[k];  // t[k1][j2] over the inputs' slots
        ct_inner<R, A, J2 + 1>(v);
    }
}

template <int R>
__device__ __forceinline__ void dft(float2 (&v)[R]) {
    if constexpr (R == 1) {
    } else if constexpr ((R & (R - 1)) == 0) {
        constexpr int LG = log2c(R);
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const int j = bitrevc(i, LG);
            if (j > i) {
                const float2 t = v[i];
                v[i] = v[j];
                v[j] = t;
            }
        }
        p2_stage<R, 1, 0>(v);
    } else if constexpr (odd_factor(R) == R) {
        float2 s[R / 2], d[R / 2];
        float2 x0 = v[0], sum = v[0];
#pragma unroll
        for (int j = 1; j <= R / 2; ++j) {
            s[j - 1] = make_float2(v[j].x + v[R - j].x, v[j].y + v[R - j].y);
            d[j - 1] = make_float2(v[j].x - v[R - j].x, v[j].y - v[R - j].y);
            sum.x += s[j - 1].x;
            sum.y += s[j - 1].y;
        }
        odd_out<R, 1>(v, x0, s, d);
        v[0] = sum;
    } else {
        // j = B j1 + j2, k = k1 + A k2
        constexpr int A = odd_factor(R), B = R / A;
        ct_inner<R, A, 0>(v);
        float2 o[R];
#pragma unroll
        for (int k1 = 0; k1 < A; ++k1) {
            float2 t[B];
#pragma unroll
            for (int j = 0; j < B; ++j) t[j] = v[B * k1 + j];
            dft<B>(t);
#pragma unroll
            for (int k2 = 0; k2 < B; ++k2) o[k1 + A * k2] = t[k2];
        }
#pragma unroll
        for (int i = 0; i < R; ++i) v[i] = o[i];
    }
}

// Mean gain error of the constants above, relative and averaged over all (input,
// output) pairs: rounded to FP32 a constant is not of modulus one, and the powers of
// two share few of them (sqrt(1/2), cos(pi / 8)), which err to the same side: a
// 32-point transform loses 3e-8 of its amplitude, F^H F of 512x512 with its twelve
// passes 3e-7, as much as all its rounding errors.  The twiddle tables between the two
// passes of a line make up for it (their own roundings are as many as the line's
// points, and even out).
constexpr double gain_of(double c, double s, double re, double im) { return c * re + s * im - 1.0; }
constexpr double kStep = -2.0 * 3.14159265358979323846264338327950288;

constexpr double mulw_gain(int num, int den) {  // of mulw<num, den>
    const int m = num % den;
    if (4 * m % den == 0) return 0.0;
    const double c = ccos(kStep * m / den), s = csin(kStep * m / den);
    return gain_of(c, s, (float)c, (float)s);
}
constexpr double butterfly_gain(int k, int den) {  // of butterfly<k, den>'s factor
    if (k == 0 || 4 * k == den) return 0.0;
    const double c = ccos(kStep * k / den), s = csin(kStep * k / den);
    const bool big_c = c * c >= s * s;
    const double m = (float)(big_c ? c : s), t = (float)(big_c ? s / c : c / s);
    return big_c ? gain_of(c, s, m, m * t) : gain_of(c, s, m * t, m);
}
constexpr double dft_gain(int r) {
    double g = 0.0;
    if ((r & (r - 1)) == 0) {  // the lower half of every stage's inputs is multiplied
        for (int half = 2; half < r; half *= 2)
            for (int k = 0; k < half; ++k) g += butterfly_gain(k, 2 * half) / (2 * half);
    } else if (odd_factor(r) == r) {
        for (int j = 1; j < r; ++j)
            for (int k = 1; k < r; ++k) {
                const double c = ccos(kStep * (j * k % r) / r), s = csin(kStep * (j * k % r) / r);
                g += gain_of(c, s, (float)c, (float)s) / (r * r);
            }
    } else {
        const int a = odd_factor(r), b = r / a;
        g = dft_gain(a) + dft_gain(b);
        for (int j = 0; j < b; ++j)
            for (int k = 0; k < a; ++k) g += mulw_gain(j * k, r) / r;
    }
    return g;
}

}  // namespace fftr
}  // namespace imp
