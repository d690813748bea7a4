// dftreg.cuh -- DFTs of a compile-time length held in one thread's registers (float2 or double2, natural order in and out):
// 2, 3, 4, 5 and 8 directly, the other lengths as A x B Cooley-Tukey steps whose twiddles are constants of the
// unrolled code. DIR = -1 forward (e^{-2 pi i jk/R}), +1 inverse, unnormalised.
#pragma once

#include <numeric>
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
// A transform multiplies by the same constants every time. One whose rounding makes its modulus larger or smaller than
// 1 scales the waves by the same factor at every slice, and detector sums drift with it; one whose direction is off
// costs every wave its accuracy. So sqrt(1/2) and sqrt(3/4) are kept to two terms, and every other turn takes the form
// of as few operations that has both small: a and b near its cosine and sine, or h (1 + i t) or i h (1 - i t) with t
// near its tangent or cotangent, each searched over neighbouring floats. Where none has its modulus within 1e-8 the
// turns of 15 and 22.5 degrees are too long and too short by turns, and those of 6 and 7.2 degrees take h to two terms
// (at 22.5 degrees that would cost the 512-point passes 2 %). Forward transforms of random values, relative error and
// mean energy error in 1e-8, all emulated on the CPU (cos and sin each rounded to nearest | as the neighbouring floats
// nearest to modulus 1 | this form): 512 points 10.2, -4.1 | 11.3, -0.7 | 10.2, -0.4; 384 10.0, -4.1 | 11.3, -0.4 |
// 10.0, 0.1; 500 11.5, 6.7 | 13.1, 2.2 | 10.4, 0.5 (radix-8 passes at 512: 10.3, -2.6).
struct Turn {
    int form;       // 0: a + i b, 1: a (1 + i b), 2: i a (1 - i b)
    float a, b, l;  // l: the rest of a
};
constexpr double ulp_of(double x) {  // of |x| < 8 as a float
    double p = 4.0;
    while (p > (x < 0 ? -x : x)) p *= 0.5;
    return p * 1.1920928955078125e-7;
}
constexpr double root_of(double x) {  // of x near 1
    double y = x;
    for (int k = 0; k < 14; ++k) y = 0.5 * (y + x / y);
    return y;
}
// c + i s of squared modulus m; sign > 0 or < 0: none shorter or longer than that.
constexpr Turn turn_of(double c, double s, double m = 1.0, int sign = 0, bool pairs = true) {
    Turn best{};
    double least = 1.0, off = 0.0;
    auto take = [&](int form, double a, double b, double energy, double angle) {
        const double cost = (sign ? 1.0 : 4.0) * energy * energy + angle * angle;
        if (cost >= least || energy * sign < 0.0) return;
        least = cost;
        off = energy < 0 ? -energy : energy;
        best = Turn{form, (float)a, (float)b, 0.0f};
    };
    const double cf = (double)(float)c, sf = (double)(float)s;
    for (int i = pairs ? -1 : 2; i <= 1; ++i)
        for (int j = -2; j <= 2; ++j) {
            const double a = cf + i * ulp_of(cf), b = sf + j * ulp_of(sf);
            take(0, a, b, (a * a + b * b) / m - 1.0, (b - s) * c - (a - c) * s);
        }
    for (int form = 1; form <= 2; ++form) {
        const double big = form == 2 ? s : c, r = form == 2 ? c / s : s / c, near = (double)(float)r;
        if (r < -8.0 || r > 8.0) continue;
        for (int k = -2; k <= 2; ++k) {
            const double t = near + k * ulp_of(near), len = root_of(m / (1.0 + t * t));
            const double h = (double)(float)(big < 0 ? -len : len);
            take(form, h, t, h * h * (1.0 + t * t) / m - 1.0, (t - r) / (1.0 + r * r));
        }
    }
    if (off > 1.1e-8 && sign == 0) {
        const bool steep = c * c < s * s;
        const double t = (double)(float)(steep ? c / s : s / c), len = root_of(m / (1.0 + t * t));
        const double big = (steep ? s : c) < 0 ? -len : len;
        best = Turn{steep ? 2 : 1, (float)big, (float)t, (float)(big - (double)(float)big)};
    }
    return best;
}
constexpr float kHalfRoot = 0.70710678118654752440f, kHalfRootRest = (float)(0.70710678118654752440 - (double)kHalfRoot);
// sqrt(3/4) as 7/8 and the rest, so that s (h + l) + m by two fused operations loses nothing of l (a rest below the
// rounding of m would be rounded away in s l + m nearly every time)
constexpr float kThreeRoot = 0.875f, kThreeRootRest = (float)(0.86602540378443864676 - 0.875);

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
        constexpr double c = unit_cos(e, N), s = DIR * unit_sin(e, N);
        constexpr float h = kThreeRoot, l = kThreeRootRest, p = c < 0 ? -1.0f : 1.0f, q = s < 0 ? -1.0f : 1.0f;
        if constexpr (12 * e % N == 0 && s * s < 0.5) {  // 30 degrees from the real axis: s = +-1/2
            const float2 u = pmul(swp(v), make_float2(-0.5f * q, 0.5f * q));
            return pfma(v, make_float2(p * h, p * h), pfma(v, make_float2(p * l, p * l), u));
        } else if constexpr (12 * e % N == 0) {  // and from the imaginary one: c = +-1/2
            const float2 u = pmul(v, make_float2(0.5f * p, 0.5f * p));
            return pfma(swp(v), make_float2(-q * h, q * h), pfma(swp(v), make_float2(-q * l, q * l), u));
        } else {
            constexpr Turn any = turn_of(c, s);
            constexpr int sign = (e / std::gcd(e, N)) % 4 == 1 ? 1 : -1;
            constexpr Turn w = any.l != 0.0f && 48 * e % N == 0 ? turn_of(c, s, 1.0, sign) : any;
            if constexpr (w.form == 0) return make_float2(v.x * w.a - v.y * w.b, v.y * w.a + v.x * w.b);
            else {
                const float x = w.form == 1 ? fmaf(-w.b, v.y, v.x) : fmaf(w.b, v.x, -v.y);
                const float y = w.form == 1 ? fmaf(w.b, v.x, v.y) : fmaf(w.b, v.y, v.x);
                if constexpr (w.l == 0.0f) return make_float2(w.a * x, w.a * y);
                else return make_float2(fmaf(w.a, x, w.l * x), fmaf(w.a, y, w.l * y));
            }
        }
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
    // 1 + 2 c1 + 2 c2 = 0 also as floats, so that a constant line leaves nothing at the other frequencies; the sines as a
    // Turn h (t, 1), for outputs of mean energy 1 + 2 (c1^2 + c2^2) + 2 h^2 (1 + t^2) = 5
    constexpr float c2 = (float)unit_cos(2, 5), c1 = -0.5f - c2;
    constexpr Turn w = turn_of(unit_sin(1, 5), unit_sin(2, 5), 2.0 - (double)c1 * c1 - (double)c2 * c2, 0, false);
    static_assert(w.form == 2 && w.l == 0.0f, "b = s1 / s2");
    constexpr float h = DIR * w.a;
    const float2 a1 = padd(v[1], v[4]), b1 = psub(v[1], v[4]), a2 = padd(v[2], v[3]), b2 = psub(v[2], v[3]);
    const float2 p1 = pfma(a2, make_float2(c2, c2), pfma(a1, make_float2(c1, c1), v[0]));
    const float2 p2 = pfma(a1, make_float2(c2, c2), pfma(a2, make_float2(c1, c1), v[0]));
    const float2 q1 = swp(pfma(b1, make_float2(w.b, w.b), b2)), q2 = swp(pfma(b2, make_float2(-w.b, -w.b), b1));
    v[0] = padd(v[0], padd(a1, a2));
    v[1] = pfma(q1, make_float2(-h, h), p1);
    v[4] = pfma(q1, make_float2(h, -h), p1);
    v[2] = pfma(q2, make_float2(-h, h), p2);
    v[3] = pfma(q2, make_float2(h, -h), p2);
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
           : r == 25 ? 5 : r == 30 ? 5 : r == 32 ? 4 : 0;
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
