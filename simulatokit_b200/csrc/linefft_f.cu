// linefft_f.cu -- line transforms of the lengths 450, 576, 800.
#include "linefft_kernels.cuh"

namespace simk {

template void launch_line<450, false, float2>(const LineArgs<float2>&, bool, cudaStream_t);
template void launch_line<450, false, double2>(const LineArgs<double2>&, bool, cudaStream_t);
template void launch_line<576, false, float2>(const LineArgs<float2>&, bool, cudaStream_t);
template void launch_line<576, false, double2>(const LineArgs<double2>&, bool, cudaStream_t);
template void launch_line<800, false, float2>(const LineArgs<float2>&, bool, cudaStream_t);
template void launch_line<800, false, double2>(const LineArgs<double2>&, bool, cudaStream_t);

}  // namespace simk
