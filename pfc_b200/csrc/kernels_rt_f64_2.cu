// Kernels of run-time lengths, F64, 2 fields (kernels_rt.cuh); one file per
// field count so that they compile in parallel.
#include "kernels_rt.cuh"

namespace pfcg {

template cudaError_t rt_launch_x<double, 2>(int, const XArgs<double>&, const LaunchCfg&, cudaStream_t);
template cudaError_t rt_launch_y<double, 2>(int, const YArgs<double>&, const LaunchCfg&, cudaStream_t);

} // namespace pfcg
