// twopass_e.cu -- two-pass kernels of the lengths 240, 400, 640, 900.
#include "twopass_kernels.cuh"

namespace simk {

template bool launch_two_rows<240>(Context&, const float2*, float2*, const float2*, int, long long, int, int, float);
template bool launch_two_cols<240>(Context&, const float2*, const TwoPassCols&, int*);
template bool launch_two_rows<400>(Context&, const float2*, float2*, const float2*, int, long long, int, int, float);
template bool launch_two_cols<400>(Context&, const float2*, const TwoPassCols&, int*);
template bool launch_two_rows<640>(Context&, const float2*, float2*, const float2*, int, long long, int, int, float);
template bool launch_two_cols<640>(Context&, const float2*, const TwoPassCols&, int*);
template bool launch_two_rows<900>(Context&, const float2*, float2*, const float2*, int, long long, int, int, float);
template bool launch_two_cols<900>(Context&, const float2*, const TwoPassCols&, int*);

}  // namespace simk
