// F32 instantiation of the relaxation kernels (kernels_impl.cuh).
#include "kernels_impl.cuh"

namespace pfcg {

template cudaError_t launch_xpass<float>(int, const XArgs<float>&, const LaunchCfg&, cudaStream_t);
template cudaError_t launch_ypass<float>(int, const YArgs<float>&, const LaunchCfg&, cudaStream_t);
template cudaError_t launch_kspace_energy<float>(const cplx<float>*, long long, const Model&, const Geom&, int, const double*,
                                               const double*, double*, double*, cudaStream_t);

// One launch of the batched STEP pass (pass 0 = x, 1 = y) of the class of
// problems with U fields and length N; cudaErrorInvalidValue where the size
// has no specialised kernel.
template <int U>
static cudaError_t ct_batch_u(int pass, int N, const void* probs, const int* bp, const int* bl, int nblk,
                              const LaunchCfg& c, cudaStream_t s) {
#define PFCG_CT_CASE(NN)                                                                                              \
	case NN:                                                                                                           \
		return pass == 0 ? ct_xbatch<float, U, NN>((const XArgs<float>*)probs, bp, bl, nblk, c, s)                    \
		                 : ct_ybatch<float, U, NN>((const YArgs<float>*)probs, bp, bl, nblk, c, s);
	switch (N) {
		PFCG_CT_CASE(4096)
		PFCG_CT_CASE(2048)
		PFCG_CT_CASE(1536)
		PFCG_CT_CASE(1024)
		PFCG_CT_CASE(768)
		PFCG_CT_CASE(512)
		PFCG_CT_CASE(384)
		PFCG_CT_CASE(256)
	}
#undef PFCG_CT_CASE
	return cudaErrorInvalidValue;
}
cudaError_t launch_ct_batch(int pass, int U, int N, const void* probs, const int* bp, const int* bl, int nblk,
                            const LaunchCfg& c, cudaStream_t s) {
	if (U == 1) return ct_batch_u<1>(pass, N, probs, bp, bl, nblk, c, s);
	if (U == 2) return ct_batch_u<2>(pass, N, probs, bp, bl, nblk, c, s);
	return cudaErrorInvalidValue;
}

} // namespace pfcg
