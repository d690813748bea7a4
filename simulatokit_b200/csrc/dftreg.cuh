// dftreg.cuh -- DFTs of a compile-time length held in one thread's registers (float2 or double2, natural order in and out):
// 2, 3, 4, 5 and 8 directly, the other lengths as A x B Cooley-Tukey steps whose twiddles are constants of the
// unrolled code. DIR = -1 forward (e^{-2 pi i jk/R}), +1 inverse, unnormalised.
#pragma once

#include <utility>

#include "fft.cuh"

namespace simk {

// f(integral_constant<int, 0>) ... f(integral_constant<int, N - 1>): an unrolled loop whose index is a constant.
template <typename F, int... I>
__device__ __forceinline__ void sfor_impl(F&& f, std::integer_sequence<int, I...>) {
    (f(std::integral_constant<int, I>{}), ...);
}
template <int N, typename F> __device__ __forceinline__ void sfor(F&& f) {
    sfor_impl(f, std::make_integer_sequence<int, N>{});
}

// cos and sin of 2 pi e / n at compile time: e / n reduced to the first octant exactly, then the Taylor series.
constexpr double series_sin(double x) {
    double term = x, sum = x;
    for (int k = 1; k < 16; ++k) {
        term *= -x * x / ((2.0 * k) * (2.0 * k + 1.0));
        sum += term;
    }
    return sum;
}
constexpr double series_cos(double x) {
    double term = 1.0, sum = 1.0;
    for (int k = 1; k < 16; ++k) {
        term *= -x * x / ((2.0 * k - 1.0) * (2.0 * k));
        sum += term;
    }
    return sum;
}
constexpr double unit_cos(long long e, long long n) {
    e = ((e % n) + n) % n;
    if (2 * e > n) e = n - e;                       // cos(2 pi - x) = cos x
    if (4 * e > n) return -unit_cos(n - 2 * e, 2 * n);  // cos(pi - x) = -cos x
    if (8 * e > n) return series_sin(6.283185307179586476925 * (double)(n - 4 * e) / (4.0 * (double)n));
    return series_cos(6.283185307179586476925 * (double)e / (double)n);
}
constexpr double unit_sin(long long e, long long n) { return unit_cos(4 * e - n, 4 * n); }  // cos(x - pi/2)

// ---- float32 constants ------------------------------------------------------------------------------------------------
// A transform multiplies by the same constants every time, so a constant whose rounding makes its modulus larger or
// smaller than 1 scales the waves by the same factor at every slice, and detector sums drift with it. The constants are
// therefore kept on the unit circle: sqrt(1/2) and sqrt(3/4) as a rounded value plus its remainder (one more packed
// operation), every other cos / sin as the pair of neighbouring floats nearest to modulus 1. The mean energy error of a
// forward 512-point transform falls from 5.9e-8 (cos and sin each rounded to nearest) to 3e-9 (radix-8 passes: 2.6e-8).
constexpr double ulp_of(double x) {  // of |x| <= 1 as a float
    double p = 1.0;
    while (p > (x < 0 ? -x : x)) p *= 0.5;
    return p * 1.1920928955078125e-7;
}
struct UnitPair {
    double c, s;
};
constexpr UnitPair unit_pair(double c, double s) {
    const double cf = (double)(float)c, sf = (double)(float)s, uc = ulp_of(cf), us = ulp_of(sf);
    UnitPair best{cf, sf};
    double least = 1.0;
    for (int i = -1; i <= 1; ++i)
        for (int j = -3; j <= 3; ++j) {
            const double x = cf + i * uc, y = sf + j * us;
            const double m = 0.5 * (x * x + y * y - 1.0), d2 = (x - c) * (x - c) + (y - s) * (y - s);
            if (m * m + 0.02 * d2 < least) {
                least = m * m + 0.02 * d2;
                best = UnitPair{x, y};
            }
        }
    return best;
}
constexpr float kHalfRoot = 0.70710678118654752440f, kHalfRootRest = (float)(0.70710678118654752440 - (double)kHalfRoot);
constexpr float kThreeRoot = 0.86602540378443864676f, kThreeRootRest = (float)(0.86602540378443864676 - (double)kThreeRoot);

// v h, h = sign sqrt(1/2)
__device__ __forceinline__ float2 mul_half_root(float2 v, float sign) {
    return pfma(v, make_float2(sign * kHalfRoot, sign * kHalfRoot),
                pmul(v, make_float2(sign * kHalfRootRest, sign * kHalfRootRest)));
}

// v e^{DIR 2 pi i E / N}: multiples of an eighth turn without general products.
template <int E, int N, int DIR> __device__ __forceinline__ float2 wmul(float2 v) {
    constexpr int e = ((E % N) + N) % N;
    if constexpr (e == 0) return v;
    else if constexpr (2 * e == N) return make_float2(-v.x, -v.y);
    else if constexpr (4 * e == N) return make_float2(-DIR * v.y, DIR * v.x);
    else if constexpr (4 * e == 3 * N) return make_float2(DIR * v.y, -DIR * v.x);
    else if constexpr (8 * e == N || 8 * e == 5 * N)  // +-(1 + i DIR) / sqrt 2
        return mul_half_root(pfma(swp(v), make_float2((float)-DIR, (float)DIR), v), 8 * e == N ? 1.0f : -1.0f);
    else if constexpr (8 * e == 3 * N || 8 * e == 7 * N)  // +-(-1 + i DIR) / sqrt 2
        return mul_half_root(pfma(swp(v), make_float2((float)DIR, (float)-DIR), v), 8 * e == 7 * N ? 1.0f : -1.0f);
    else {
        constexpr UnitPair w = unit_pair(unit_cos(e, N), unit_sin(e, N));
        constexpr float c = (float)w.c, s = (float)(DIR * w.s);
        return make_float2(v.x * c - v.y * s, v.y * c + v.x * s);
    }
}

// radix 3, 5 and 8 on packed pairs; multiplication by +-i as a swapped pair inside the packed FMA
template <int DIR> __device__ __forceinline__ void pbfly3(float2 (&v)[3]) {
    constexpr float h = DIR * kThreeRoot, l = DIR * kThreeRootRest;
    const float2 t = padd(v[1], v[2]), s = swp(psub(v[1], v[2]));
    const float2 m = pfma(t, make_float2(-0.5f, -0.5f), v[0]);
    v[0] = padd(v[0], t);
    v[1] = pfma(s, make_float2(-h, h), pfma(s, make_float2(-l, l), m));
    v[2] = pfma(s, make_float2(h, -h), pfma(s, make_float2(l, -l), m));
}
template <int DIR> __device__ __forceinline__ void pbfly5(float2 (&v)[5]) {
    // sin(2 pi/5), sin(4 pi/5) as the neighbours of the rounded values with the smallest mean energy error (3e-9; nearest:
    // 1.7e-8); the cosines as -1/4 +- sqrt(5)/4, so that a constant line leaves nothing at the other frequencies
    constexpr double s1d = (float)unit_sin(1, 5), s2d = (float)unit_sin(2, 5);
    constexpr float h = 0.55901699437494742410f, s1 = (float)(s1d - ulp_of(s1d)), s2 = (float)(s2d + ulp_of(s2d));
    const float2 a1 = padd(v[1], v[4]), b1 = psub(v[1], v[4]), a2 = padd(v[2], v[3]), b2 = psub(v[2], v[3]);
    const float2 t = padd(a1, a2), d = psub(a1, a2), m = pfma(t, make_float2(-0.25f, -0.25f), v[0]);
    const float2 p1 = pfma(d, make_float2(h, h), m), p2 = pfma(d, make_float2(-h, -h), m);
    const float2 q1 = swp(pfma(b2, make_float2(s2, s2), pmul(b1, make_float2(s1, s1))));
    const float2 q2 = swp(pfma(b2, make_float2(-s1, -s1), pmul(b1, make_float2(s2, s2))));
    v[0] = padd(v[0], t);
    v[1] = pfma(q1, make_float2((float)-DIR, (float)DIR), p1);
    v[4] = pfma(q1, make_float2((float)DIR, (float)-DIR), p1);
    v[2] = pfma(q2, make_float2((float)-DIR, (float)DIR), p2);
    v[3] = pfma(q2, make_float2((float)DIR, (float)-DIR), p2);
}
template <int DIR> __device__ __forceinline__ void pbfly8(float2 (&v)[8]) {
    float2 e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
    bfly4<DIR>(e);
    bfly4<DIR>(o);
    const float2 o1 = wmul<1, 8, DIR>(o[1]), o3 = wmul<3, 8, DIR>(o[3]), s2 = swp(o[2]);
    v[0] = padd(e[0], o[0]);
    v[4] = psub(e[0], o[0]);
    v[1] = padd(e[1], o1);
    v[5] = psub(e[1], o1);
    v[2] = pfma(s2, make_float2((float)-DIR, (float)DIR), e[2]);
    v[6] = pfma(s2, make_float2((float)DIR, (float)-DIR), e[2]);
    v[3] = padd(e[3], o3);
    v[7] = psub(e[3], o3);
}

// The same in float64, with constants rounded to nearest.
template <int E, int N, int DIR> __device__ __forceinline__ double2 wmul(double2 v) {
    constexpr int e = ((E % N) + N) % N;
    constexpr double h = 0.70710678118654752440;
    if constexpr (e == 0) return v;
    else if constexpr (2 * e == N) return make_double2(-v.x, -v.y);
    else if constexpr (4 * e == N) return make_double2(-DIR * v.y, DIR * v.x);
    else if constexpr (4 * e == 3 * N) return make_double2(DIR * v.y, -DIR * v.x);
    else if constexpr (8 * e == N) return make_double2((v.x - DIR * v.y) * h, (v.y + DIR * v.x) * h);
    else if constexpr (8 * e == 3 * N) return make_double2((-v.x - DIR * v.y) * h, (-v.y + DIR * v.x) * h);
    else if constexpr (8 * e == 5 * N) return make_double2((DIR * v.y - v.x) * h, (-v.y - DIR * v.x) * h);
    else if constexpr (8 * e == 7 * N) return make_double2((v.x + DIR * v.y) * h, (v.y - DIR * v.x) * h);
    else {
        constexpr double c = unit_cos(e, N), s = DIR * unit_sin(e, N);
        return make_double2(v.x * c - v.y * s, v.y * c + v.x * s);
    }
}
template <int DIR> __device__ __forceinline__ void pbfly3(double2 (&v)[3]) { bfly3<DIR>(v); }
template <int DIR> __device__ __forceinline__ void pbfly5(double2 (&v)[5]) { bfly5<DIR>(v); }
template <int DIR> __device__ __forceinline__ void pbfly8(double2 (&v)[8]) { bfly8<DIR>(v); }

// The first factor A of the step R = A B.
constexpr int dft_first(int r) {
    return r == 6 ? 2 : r == 10 ? 2 : r == 12 ? 3 : r == 15 ? 3 : r == 16 ? 4 : r == 18 ? 3 : r == 20 ? 4 : r == 24 ? 3
           : r == 25 ? 5 : r == 30 ? 5 : r == 32 ? 4 : r == 40 ? 5 : 0;
}

// X[k1 + A k2] = sum_n2 W_R^{n2 k1} W_B^{n2 k2} sum_n1 x[B n1 + n2] W_A^{n1 k1}
template <int R, int DIR, typename V> __device__ __forceinline__ void dft_reg(V (&v)[R]) {
    if constexpr (R == 1) return;
    else if constexpr (R == 2) bfly2<DIR>(v);
    else if constexpr (R == 3) pbfly3<DIR>(v);
    else if constexpr (R == 4) bfly4<DIR>(v);
    else if constexpr (R == 5) pbfly5<DIR>(v);
    else if constexpr (R == 8) pbfly8<DIR>(v);
    else {
        constexpr int A = dft_first(R), B = R / A;
        static_assert(A > 1 && A * B == R, "a register DFT of this length is not defined");
        V w[R];
        sfor<B>([&](auto n2c) {
            constexpr int n2 = decltype(n2c)::value;
            V u[A];
            sfor<A>([&](auto n1c) { u[decltype(n1c)::value] = v[B * decltype(n1c)::value + n2]; });
            dft_reg<A, DIR>(u);
            sfor<A>([&](auto k1c) {
                constexpr int k1 = decltype(k1c)::value;
                w[k1 * B + n2] = wmul<n2 * k1, R, DIR>(u[k1]);
            });
        });
        sfor<A>([&](auto k1c) {
            constexpr int k1 = decltype(k1c)::value;
            V u[B];
            sfor<B>([&](auto n2c) { u[decltype(n2c)::value] = w[k1 * B + decltype(n2c)::value]; });
            dft_reg<B, DIR>(u);
            sfor<B>([&](auto k2c) { v[k1 + A * decltype(k2c)::value] = u[decltype(k2c)::value]; });
        });
    }
}

}  // namespace simk
