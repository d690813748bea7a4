// linefft.cu -- dispatch of the one-exchange line transforms on the length.
#include "linefft.cuh"

#include <cmath>

namespace simk {

#define SIMK_TWO_PLAN(n, a, b)                                                                    \
    extern template void launch_line<n, false, float2>(const LineArgs<float2>&, bool, cudaStream_t);    \
    extern template void launch_line<n, false, double2>(const LineArgs<double2>&, bool, cudaStream_t);
#include "twopass_plans.inc"
#undef SIMK_TWO_PLAN
#define SIMK_BLUE(n)                                                                             \
    extern template void launch_line<n, true, float2>(const LineArgs<float2>&, bool, cudaStream_t);     \
    extern template void launch_line<n, true, double2>(const LineArgs<double2>&, bool, cudaStream_t);
SIMK_BLUE(256)
SIMK_BLUE(512)
SIMK_BLUE(1024)
#undef SIMK_BLUE

int line_first_radix(int N) {
    switch (N) {
#define SIMK_TWO_PLAN(n, a, b) \
    case n: return a;
#include "twopass_plans.inc"
#undef SIMK_TWO_PLAN
        default: return 0;
    }
}

// Rounded to nearest, then column by column (the values one item of step B multiplies by; j = 0 takes none) single
// values moved to the neighbouring float, the ones nearest to half way between two first, until the column's mean
// squared modulus is scale^2: the moves cost 0.1 % in the error of a transform, and without them the 384-point table
// alone takes 1.2e-8 of the energy a pass, and the column k = 0 of a scaled table, where a plane wave's energy is, has
// every value off alike (1/640^2 is 2.2e-8 off as a float: 1.8e-6 after 40 slices).
std::vector<float2> line_table(int n, int r1, double scale) {
    const int r2 = n / r1;
    std::vector<float2> t(n);
    std::vector<double2> exact(n);
    for (int i = 0; i < n; ++i) {
        double2& x = exact[i];
        host_sincospi(-2.0 * (double)((long long)(i / r1) * (i % r1) % n) / (double)n, &x.y, &x.x);
        x = x * scale;
        t[i] = make_float2((float)x.x, (float)x.y);
    }
    for (int k = 0; k < r1; ++k) {
        double excess = 0.0;  // of the squared moduli
        for (int j = 1; j < r2; ++j) {
            const float2 w = t[j * r1 + k];
            excess += (double)w.x * w.x + (double)w.y * w.y - scale * scale;
        }
        for (;;) {  // the move that costs least for what it brings the excess nearer to 0
            float *at = nullptr, to = 0.0f;
            double least = 0.0, change = 0.0;
            for (int q = 2; q < 2 * r2; ++q) {
                float& w = q & 1 ? t[(q >> 1) * r1 + k].y : t[(q >> 1) * r1 + k].x;
                const double x = q & 1 ? exact[(q >> 1) * r1 + k].y : exact[(q >> 1) * r1 + k].x;
                if (x == 0.0 || std::fabs(x) == 1.0) continue;
                const float next = std::nextafterf(w, excess > 0.0 ? 0.0f : std::copysign(2.0f, w));
                const double step = (double)next * next - (double)w * w;
                if (std::fabs(excess + step) >= std::fabs(excess)) continue;
                const double cost = ((next - x) * (next - x) - (w - x) * (w - x)) / std::fabs(step);
                if (!at || cost < least) {
                    at = &w;
                    to = next;
                    least = cost;
                    change = step;
                }
            }
            if (!at) break;
            *at = to;
            excess += change;
        }
    }
    return t;
}

bool line_bluestein_length(int N) { return N == 256 || N == 512 || N == 1024; }

template <typename V> void launch_line_any(int N, bool blue, const LineArgs<V>& a, bool columns, cudaStream_t stream) {
    if (blue) {
        switch (N) {
            case 256: launch_line<256, true, V>(a, columns, stream); return;
            case 512: launch_line<512, true, V>(a, columns, stream); return;
            default: launch_line<1024, true, V>(a, columns, stream); return;
        }
    }
    switch (N) {
#define SIMK_TWO_PLAN(n, r1, r2) \
    case n: launch_line<n, false, V>(a, columns, stream); return;
#include "twopass_plans.inc"
#undef SIMK_TWO_PLAN
        default: throw Error(SIMK_ERR_INVALID, "no line plan for length " + std::to_string(N));
    }
}
template void launch_line_any<float2>(int, bool, const LineArgs<float2>&, bool, cudaStream_t);
template void launch_line_any<double2>(int, bool, const LineArgs<double2>&, bool, cudaStream_t);

}  // namespace simk
