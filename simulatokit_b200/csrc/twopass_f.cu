// twopass_f.cu -- two-pass kernels of the lengths 450, 576, 800.
#include "twopass_kernels.cuh"

namespace simk {

template bool launch_two_rows<450>(Context&, const float2*, float2*, const float2*, int, long long, int, int, float);
template bool launch_two_cols<450>(Context&, const float2*, const TwoPassCols&, int*);
template bool launch_two_rows<576>(Context&, const float2*, float2*, const float2*, int, long long, int, int, float);
template bool launch_two_cols<576>(Context&, const float2*, const TwoPassCols&, int*);
template bool launch_two_rows<800>(Context&, const float2*, float2*, const float2*, int, long long, int, int, float);
template bool launch_two_cols<800>(Context&, const float2*, const TwoPassCols&, int*);

}  // namespace simk
