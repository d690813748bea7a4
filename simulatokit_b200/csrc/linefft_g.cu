// linefft_g.cu -- line transforms of the lengths 480, 600, 960, 720.
#include "linefft_kernels.cuh"

namespace simk {

template void launch_line<480, false, float2>(const LineArgs<float2>&, bool, cudaStream_t);
template void launch_line<480, false, double2>(const LineArgs<double2>&, bool, cudaStream_t);
template void launch_line<600, false, float2>(const LineArgs<float2>&, bool, cudaStream_t);
template void launch_line<600, false, double2>(const LineArgs<double2>&, bool, cudaStream_t);
template void launch_line<960, false, float2>(const LineArgs<float2>&, bool, cudaStream_t);
template void launch_line<960, false, double2>(const LineArgs<double2>&, bool, cudaStream_t);
template void launch_line<720, false, float2>(const LineArgs<float2>&, bool, cudaStream_t);
template void launch_line<720, false, double2>(const LineArgs<double2>&, bool, cudaStream_t);

}  // namespace simk
