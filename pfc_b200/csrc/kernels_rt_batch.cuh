// Batched STEP kernels of run-time lengths.
#pragma once

#include "kernels_wide.cuh"

namespace pfcg {

// Many independent relaxations of runtime sizes in one launch: block b runs
// tile (x-pass) or column group (y-pass) blk_local[b] of problem blk_prob[b],
// whose arguments sit in global memory. Launched with the largest thread count
// and shared memory any problem needs; the bodies use whatever threads they get.
template <typename T>
__global__ void __launch_bounds__(MAXNT, 1)
    xrt_batch_kernel(const XArgs<T>* __restrict__ probs, const int* __restrict__ blk_prob, const int* __restrict__ blk_local) {
	const XArgs<T>& a = probs[blk_prob[blockIdx.x]];
	const int local = blk_local[blockIdx.x];
	switch (a.m.U) {
	case 1: rt_xpass<T, 1, true>(a, XP_STEP, local); break;
	case 2: rt_xpass<T, 2, true>(a, XP_STEP, local); break;
	case 3:
		if constexpr (sizeof(T) == 4) {
			if (a.wtw) { wide::xpass<3, XP_STEP>(a, local); break; }
		}
		rt_xpass<T, 3, true>(a, XP_STEP, local);
		break;
	case 4:
		if constexpr (sizeof(T) == 4) {
			if (a.wtw) { wide::xpass<4, XP_STEP>(a, local); break; }
		}
		rt_xpass<T, 4, true>(a, XP_STEP, local);
		break;
	}
}

template <typename T>
__global__ void __launch_bounds__(MAXNT, 1)
    yrt_batch_kernel(const YArgs<T>* __restrict__ probs, const int* __restrict__ blk_prob, const int* __restrict__ blk_local) {
	const YArgs<T>& a = probs[blk_prob[blockIdx.x]];
	const int local = blk_local[blockIdx.x];
	switch (a.m.U) {
	case 1: rt_ypass<T, 1, true>(a, YP_STEP, local); break;
	case 2: rt_ypass<T, 2, true>(a, YP_STEP, local); break;
	case 3:
		if constexpr (sizeof(T) == 4) {
			if (a.wtw) { wide::ypass<3, YP_STEP>(a, local); break; }
		}
		rt_ypass<T, 3, true>(a, YP_STEP, local);
		break;
	case 4:
		if constexpr (sizeof(T) == 4) {
			if (a.wtw) { wide::ypass<4, YP_STEP>(a, local); break; }
		}
		rt_ypass<T, 4, true>(a, YP_STEP, local);
		break;
	}
}

template <typename T>
cudaError_t launch_generic_batch(int pass, const void* probs, const int* bp, const int* bl, int nblk, int threads,
                                 int smem, cudaStream_t s) {
	static unsigned long long mx = 0, my = 0;
	smem_attr(xrt_batch_kernel<T>, mx);
	smem_attr(yrt_batch_kernel<T>, my);
	if (nblk <= 0) return cudaGetLastError();
	if (pass == 0) xrt_batch_kernel<T><<<nblk, threads, smem, s>>>((const XArgs<T>*)probs, bp, bl);
	else yrt_batch_kernel<T><<<nblk, threads, smem, s>>>((const YArgs<T>*)probs, bp, bl);
	return cudaGetLastError();
}

} // namespace pfcg
