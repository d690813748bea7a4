// twopass_h.cu -- two-pass kernels of the lengths 720, 750.
#include "twopass_kernels.cuh"

namespace simk {

template bool launch_two_rows<720>(Context&, const float2*, float2*, const float2*, int, long long, int, int, float);
template bool launch_two_cols<720>(Context&, const float2*, const TwoPassCols&, int*);
template bool launch_two_rows<750>(Context&, const float2*, float2*, const float2*, int, long long, int, int, float);
template bool launch_two_cols<750>(Context&, const float2*, const TwoPassCols&, int*);

}  // namespace simk
