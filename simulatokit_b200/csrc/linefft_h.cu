// linefft_h.cu -- Bluestein's transforms on work lengths 256 to 1024.
#include "linefft_kernels.cuh"

namespace simk {

template void launch_line<256, true, float2>(const LineArgs<float2>&, bool, cudaStream_t);
template void launch_line<256, true, double2>(const LineArgs<double2>&, bool, cudaStream_t);
template void launch_line<512, true, float2>(const LineArgs<float2>&, bool, cudaStream_t);
template void launch_line<512, true, double2>(const LineArgs<double2>&, bool, cudaStream_t);
template void launch_line<1024, true, float2>(const LineArgs<float2>&, bool, cudaStream_t);
template void launch_line<1024, true, double2>(const LineArgs<double2>&, bool, cudaStream_t);

}  // namespace simk
