// Kernels of run-time lengths, F32, 3 fields (kernels_rt.cuh); one file per
// field count so that they compile in parallel.
#include "kernels_rt.cuh"

namespace pfcg {

template cudaError_t rt_launch_x<float, 3>(int, const XArgs<float>&, const LaunchCfg&, cudaStream_t);
template cudaError_t rt_launch_y<float, 3>(int, const YArgs<float>&, const LaunchCfg&, cudaStream_t);

} // namespace pfcg
