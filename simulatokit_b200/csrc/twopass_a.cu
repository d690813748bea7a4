// twopass_a.cu -- two-pass kernels of the lengths 128 (rows), 250, 256, 512.
#include "twopass_kernels.cuh"

namespace simk {

template bool launch_two_rows<128>(Context&, const float2*, float2*, const float2*, int, long long, int, int, float);
template bool launch_two_rows<250>(Context&, const float2*, float2*, const float2*, int, long long, int, int, float);
template bool launch_two_cols<250>(Context&, const float2*, const TwoPassCols&, int*);
template bool launch_two_rows<256>(Context&, const float2*, float2*, const float2*, int, long long, int, int, float);
template bool launch_two_cols<256>(Context&, const float2*, const TwoPassCols&, int*);
template bool launch_two_rows<512>(Context&, const float2*, float2*, const float2*, int, long long, int, int, float);
template bool launch_two_cols<512>(Context&, const float2*, const TwoPassCols&, int*);

}  // namespace simk
