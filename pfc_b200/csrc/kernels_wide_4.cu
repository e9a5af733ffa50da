// FP32 kernels of four fields (kernels_wide.cuh).
#include "kernels_wide.cuh"

namespace pfcg {

template cudaError_t wide_launch_x<4>(int, const XArgs<float>&, const LaunchCfg&, cudaStream_t);
template cudaError_t wide_launch_y<4>(int, const YArgs<float>&, const LaunchCfg&, cudaStream_t);

} // namespace pfcg
