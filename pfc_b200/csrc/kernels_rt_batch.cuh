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

// The same where every block's problem has U fields: those kernels need no more
// registers than U takes.
template <typename T, int U>
__global__ void __launch_bounds__(MAXNT, 1)
    xrt_batch_kernel_u(const XArgs<T>* __restrict__ probs, const int* __restrict__ blk_prob, const int* __restrict__ blk_local) {
	rt_xpass<T, U, true>(probs[blk_prob[blockIdx.x]], XP_STEP, blk_local[blockIdx.x]);
}
template <typename T, int U>
__global__ void __launch_bounds__(MAXNT, 1)
    yrt_batch_kernel_u(const YArgs<T>* __restrict__ probs, const int* __restrict__ blk_prob, const int* __restrict__ blk_local) {
	rt_ypass<T, U, true>(probs[blk_prob[blockIdx.x]], YP_STEP, blk_local[blockIdx.x]);
}

template <typename A, typename K>
static cudaError_t batch_launch(K k, unsigned long long& mask, const void* probs, const int* bp, const int* bl, int nblk,
                                const LaunchCfg& c, cudaStream_t s) {
	smem_attr(k, mask);
	if (nblk > 0) k<<<nblk, c.block, c.smem, s>>>((const A*)probs, bp, bl);
	return cudaGetLastError();
}

template <typename T>
cudaError_t launch_generic_batch(int pass, int U, const void* probs, const int* bp, const int* bl, int nblk, const LaunchCfg& c,
                                 cudaStream_t s) {
	static unsigned long long m[6] = {};
	if constexpr (sizeof(T) == 8) {
		if (U == 1)
			return pass ? batch_launch<YArgs<T>>(yrt_batch_kernel_u<T, 1>, m[0], probs, bp, bl, nblk, c, s)
			            : batch_launch<XArgs<T>>(xrt_batch_kernel_u<T, 1>, m[1], probs, bp, bl, nblk, c, s);
		if (U == 2)
			return pass ? batch_launch<YArgs<T>>(yrt_batch_kernel_u<T, 2>, m[2], probs, bp, bl, nblk, c, s)
			            : batch_launch<XArgs<T>>(xrt_batch_kernel_u<T, 2>, m[3], probs, bp, bl, nblk, c, s);
	}
	return pass ? batch_launch<YArgs<T>>(yrt_batch_kernel<T>, m[4], probs, bp, bl, nblk, c, s)
	            : batch_launch<XArgs<T>>(xrt_batch_kernel<T>, m[5], probs, bp, bl, nblk, c, s);
}

} // namespace pfcg
