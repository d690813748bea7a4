// twopass_d.cu -- two-pass kernels of the lengths 200, 360, 1024.
#include "twopass_kernels.cuh"

namespace simk {

template bool launch_two_rows<200>(Context&, const float2*, float2*, const float2*, int, long long, int, int, float);
template bool launch_two_cols<200>(Context&, const float2*, const TwoPassCols&, int*);
template bool launch_two_rows<360>(Context&, const float2*, float2*, const float2*, int, long long, int, int, float);
template bool launch_two_cols<360>(Context&, const float2*, const TwoPassCols&, int*);
template bool launch_two_rows<1024>(Context&, const float2*, float2*, const float2*, int, long long, int, int, float);
template bool launch_two_cols<1024>(Context&, const float2*, const TwoPassCols&, int*);

}  // namespace simk
