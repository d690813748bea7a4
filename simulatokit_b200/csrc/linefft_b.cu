// linefft_b.cu -- line transforms of the lengths 160, 300, 384, 768.
#include "linefft_kernels.cuh"

namespace simk {

template void launch_line<160, false, float2>(const LineArgs<float2>&, bool, cudaStream_t);
template void launch_line<160, false, double2>(const LineArgs<double2>&, bool, cudaStream_t);
template void launch_line<300, false, float2>(const LineArgs<float2>&, bool, cudaStream_t);
template void launch_line<300, false, double2>(const LineArgs<double2>&, bool, cudaStream_t);
template void launch_line<384, false, float2>(const LineArgs<float2>&, bool, cudaStream_t);
template void launch_line<384, false, double2>(const LineArgs<double2>&, bool, cudaStream_t);
template void launch_line<768, false, float2>(const LineArgs<float2>&, bool, cudaStream_t);
template void launch_line<768, false, double2>(const LineArgs<double2>&, bool, cudaStream_t);

}  // namespace simk
