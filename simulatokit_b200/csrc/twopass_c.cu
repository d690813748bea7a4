// twopass_c.cu -- two-pass kernels of the lengths 192, 320, 500.
#include "twopass_kernels.cuh"

namespace simk {

template bool launch_two_rows<192>(Context&, const float2*, float2*, const float2*, int, long long, int, int, float);
template bool launch_two_cols<192>(Context&, const float2*, const TwoPassCols&, int*);
template bool launch_two_rows<320>(Context&, const float2*, float2*, const float2*, int, long long, int, int, float);
template bool launch_two_cols<320>(Context&, const float2*, const TwoPassCols&, int*);
template bool launch_two_rows<500>(Context&, const float2*, float2*, const float2*, int, long long, int, int, float);
template bool launch_two_cols<500>(Context&, const float2*, const TwoPassCols&, int*);

}  // namespace simk
