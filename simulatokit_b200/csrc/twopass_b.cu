// twopass_b.cu -- two-pass kernels of the lengths 160, 300, 384, 768.
#include "twopass_kernels.cuh"

namespace simk {

template bool launch_two_rows<160>(Context&, const float2*, float2*, const float2*, int, long long, int, int, float);
template bool launch_two_cols<160>(Context&, const float2*, const TwoPassCols&, int*);
template bool launch_two_rows<300>(Context&, const float2*, float2*, const float2*, int, long long, int, int, float);
template bool launch_two_cols<300>(Context&, const float2*, const TwoPassCols&, int*);
template bool launch_two_rows<384>(Context&, const float2*, float2*, const float2*, int, long long, int, int, float);
template bool launch_two_cols<384>(Context&, const float2*, const TwoPassCols&, int*);
template bool launch_two_rows<768>(Context&, const float2*, float2*, const float2*, int, long long, int, int, float);
template bool launch_two_cols<768>(Context&, const float2*, const TwoPassCols&, int*);

}  // namespace simk
