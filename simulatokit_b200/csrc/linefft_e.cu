// linefft_e.cu -- line transforms of the lengths 240, 400, 640, 900.
#include "linefft_kernels.cuh"

namespace simk {

template void launch_line<240, false, float2>(const LineArgs<float2>&, bool, cudaStream_t);
template void launch_line<240, false, double2>(const LineArgs<double2>&, bool, cudaStream_t);
template void launch_line<400, false, float2>(const LineArgs<float2>&, bool, cudaStream_t);
template void launch_line<400, false, double2>(const LineArgs<double2>&, bool, cudaStream_t);
template void launch_line<640, false, float2>(const LineArgs<float2>&, bool, cudaStream_t);
template void launch_line<640, false, double2>(const LineArgs<double2>&, bool, cudaStream_t);
template void launch_line<900, false, float2>(const LineArgs<float2>&, bool, cudaStream_t);
template void launch_line<900, false, double2>(const LineArgs<double2>&, bool, cudaStream_t);

}  // namespace simk
