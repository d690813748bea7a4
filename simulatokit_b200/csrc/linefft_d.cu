// linefft_d.cu -- line transforms of the lengths 200, 360, 1024.
#include "linefft_kernels.cuh"

namespace simk {

template void launch_line<200, false, float2>(const LineArgs<float2>&, bool, cudaStream_t);
template void launch_line<200, false, double2>(const LineArgs<double2>&, bool, cudaStream_t);
template void launch_line<360, false, float2>(const LineArgs<float2>&, bool, cudaStream_t);
template void launch_line<360, false, double2>(const LineArgs<double2>&, bool, cudaStream_t);
template void launch_line<1024, false, float2>(const LineArgs<float2>&, bool, cudaStream_t);
template void launch_line<1024, false, double2>(const LineArgs<double2>&, bool, cudaStream_t);

}  // namespace simk
