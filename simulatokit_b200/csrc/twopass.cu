// twopass.cu -- the two-pass engine's tables and its dispatch on the line length.
#include "twopass.cuh"

#include "linefft.cuh"

namespace simk {

// Each length's launches are instantiated in one of the twopass_*.cu files (built side by side).
#define SIMK_TWO_PLAN(n, a, b)                                                                                        \
    template <int N> bool launch_two_rows(Context&, const float2*, float2*, const float2*, int, long long, int, int,  \
                                          float);                                                                     \
    template <int N> bool launch_two_cols(Context&, const float2*, const TwoPassCols&, int*);                         \
    extern template bool launch_two_rows<n>(Context&, const float2*, float2*, const float2*, int, long long, int,     \
                                            int, float);                                                              \
    extern template bool launch_two_cols<n>(Context&, const float2*, const TwoPassCols&, int*);
#include "twopass_plans.inc"
#undef SIMK_TWO_PLAN

namespace {
// R1 of the plan of n, 0 where there is none.
int first_radix(int n) {
    switch (n) {
#define SIMK_TWO_PLAN(n, a, b) \
    case n: return a;
#include "twopass_plans.inc"
#undef SIMK_TWO_PLAN
        default: return 0;
    }
}
}  // namespace

bool twopass_length(int n) { return first_radix(n) != 0; }

const float2* twopass_table(Context& ctx, int n, long long points) {
    DeviceBuffer& buf = ctx.twopass_tables[{n, points}];
    if (!buf.ptr) {
        const int r1 = first_radix(n);
        SIMK_REQUIRE(r1 != 0, "no two-pass plan for length " + std::to_string(n));
        const std::vector<float2> h = line_table(n, r1, 1.0 / (double)points);
        DeviceBuffer made(n * sizeof(float2));
        copy_to_device(made.ptr, h.data(), n * sizeof(float2));
        buf = std::move(made);
    }
    return buf.as<float2>();
}

bool twopass_rows(Context& ctx, float2* psi, const float2* tmul, int nx, int ny, long long nrows, int inv, int fwd,
                  float scale) {
    if (!inv && !fwd) return false;
    switch (ny) {
#define SIMK_TWO_PLAN(n, a, b) \
    case n: return launch_two_rows<n>(ctx, twopass_table(ctx, n), psi, tmul, nx, nrows, inv, fwd, scale);
#include "twopass_plans.inc"
#undef SIMK_TWO_PLAN
        default: return false;
    }
}

bool twopass_cols(Context& ctx, int nx, const TwoPassCols& a, int* groups) {
    switch (nx) {
#define SIMK_TWO_PLAN(n, r1, r2)                                                                               \
    case n:                                                                                                    \
        if constexpr (n > kTwoColsAbove) return launch_two_cols<n>(ctx, twopass_table(ctx, n), a, groups);     \
        else return false;
#include "twopass_plans.inc"
#undef SIMK_TWO_PLAN
        default: return false;
    }
}

}  // namespace simk
