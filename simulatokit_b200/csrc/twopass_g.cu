// twopass_g.cu -- two-pass kernels of the lengths 480, 600, 960.
#include "twopass_kernels.cuh"

namespace simk {

template bool launch_two_rows<480>(Context&, const float2*, float2*, const float2*, int, long long, int, int, float);
template bool launch_two_cols<480>(Context&, const float2*, const TwoPassCols&, int*);
template bool launch_two_rows<600>(Context&, const float2*, float2*, const float2*, int, long long, int, int, float);
template bool launch_two_cols<600>(Context&, const float2*, const TwoPassCols&, int*);
template bool launch_two_rows<960>(Context&, const float2*, float2*, const float2*, int, long long, int, int, float);
template bool launch_two_cols<960>(Context&, const float2*, const TwoPassCols&, int*);

}  // namespace simk
