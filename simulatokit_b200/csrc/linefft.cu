// linefft.cu -- dispatch of the one-exchange line transforms on the length.
#include "linefft.cuh"

namespace simk {

#define SIMK_TWO_PLAN(n, a, b)                                                                    \
    extern template void launch_line<n, false, float2>(const LineArgs<float2>&, bool, cudaStream_t);    \
    extern template void launch_line<n, false, double2>(const LineArgs<double2>&, bool, cudaStream_t);
#include "twopass_plans.inc"
#undef SIMK_TWO_PLAN
#define SIMK_BLUE(n)                                                                             \
    extern template void launch_line<n, true, float2>(const LineArgs<float2>&, bool, cudaStream_t);     \
    extern template void launch_line<n, true, double2>(const LineArgs<double2>&, bool, cudaStream_t);
SIMK_BLUE(128)
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

bool line_bluestein_length(int N) { return N == 128 || N == 256 || N == 512 || N == 1024; }

template <typename V> void launch_line_any(int N, bool blue, const LineArgs<V>& a, bool columns, cudaStream_t stream) {
    if (blue) {
        switch (N) {
            case 128: launch_line<128, true, V>(a, columns, stream); return;
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
