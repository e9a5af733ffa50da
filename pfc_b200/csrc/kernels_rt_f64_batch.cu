// Batched STEP kernels of run-time lengths, F64 (kernels_rt_batch.cuh).
#include "kernels_rt_batch.cuh"

namespace pfcg {

template cudaError_t launch_generic_batch<double>(int, int, const void*, const int*, const int*, int, const LaunchCfg&,
                                           cudaStream_t);

} // namespace pfcg
