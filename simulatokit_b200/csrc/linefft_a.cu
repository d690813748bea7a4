// linefft_a.cu -- line transforms of the lengths 128, 250, 256, 512.
#include "linefft_kernels.cuh"

namespace simk {

template void launch_line<128, false, float2>(const LineArgs<float2>&, bool, cudaStream_t);
template void launch_line<128, false, double2>(const LineArgs<double2>&, bool, cudaStream_t);
template void launch_line<250, false, float2>(const LineArgs<float2>&, bool, cudaStream_t);
template void launch_line<250, false, double2>(const LineArgs<double2>&, bool, cudaStream_t);
template void launch_line<256, false, float2>(const LineArgs<float2>&, bool, cudaStream_t);
template void launch_line<256, false, double2>(const LineArgs<double2>&, bool, cudaStream_t);
template void launch_line<512, false, float2>(const LineArgs<float2>&, bool, cudaStream_t);
template void launch_line<512, false, double2>(const LineArgs<double2>&, bool, cudaStream_t);

}  // namespace simk
