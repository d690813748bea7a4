// linefft_c.cu -- line transforms of the lengths 192, 320, 500, 750.
#include "linefft_kernels.cuh"

namespace simk {

template void launch_line<192, false, float2>(const LineArgs<float2>&, bool, cudaStream_t);
template void launch_line<192, false, double2>(const LineArgs<double2>&, bool, cudaStream_t);
template void launch_line<320, false, float2>(const LineArgs<float2>&, bool, cudaStream_t);
template void launch_line<320, false, double2>(const LineArgs<double2>&, bool, cudaStream_t);
template void launch_line<500, false, float2>(const LineArgs<float2>&, bool, cudaStream_t);
template void launch_line<500, false, double2>(const LineArgs<double2>&, bool, cudaStream_t);
template void launch_line<750, false, float2>(const LineArgs<float2>&, bool, cudaStream_t);
template void launch_line<750, false, double2>(const LineArgs<double2>&, bool, cudaStream_t);

}  // namespace simk
