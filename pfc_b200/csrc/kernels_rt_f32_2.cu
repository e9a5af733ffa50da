// Kernels of run-time lengths, F32, 2 fields (kernels_rt.cuh); one file per
// field count so that they compile in parallel.
#include "kernels_rt.cuh"

namespace pfcg {

template cudaError_t rt_launch_x<float, 2>(int, const XArgs<float>&, const LaunchCfg&, cudaStream_t);
template cudaError_t rt_launch_y<float, 2>(int, const YArgs<float>&, const LaunchCfg&, cudaStream_t);

} // namespace pfcg
