// FP32 kernels of three fields (kernels_wide.cuh).
#include "kernels_wide.cuh"

namespace pfcg {

template cudaError_t wide_launch_x<3>(int, const XArgs<float>&, const LaunchCfg&, cudaStream_t);
template cudaError_t wide_launch_y<3>(int, const YArgs<float>&, const LaunchCfg&, cudaStream_t);

} // namespace pfcg
