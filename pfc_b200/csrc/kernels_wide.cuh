// FP32 STEP, r2c and first-spectrum kernels of systems of three and four fields.
//
// They keep the order of operations that these systems' FP32 results were made
// with: passes of radix 16, then the power-of-two rest, then 3, 5 and 7, twiddles
// from an n-entry table, inverse transforms with their own signs, field pairs in the
// order of the row tile. Which products are fused is the compiler's choice, and
// pfcg_autotune may take another row tile, so the last bits can differ between
// builds, a single problem and a batch, and tuned and untuned handles.
// The kernels of kernels_rt.cuh step these systems about three times as fast and
// are as close to 64 bits (1.5e-5 against 1.4e-5 after 50 steps), but three or
// four coupled fields amplify a difference in rounding of 1e-7 to 4e-5 of the
// field and 2e-3 of a point within 100 steps, which no longer counts as the same
// FP32 result (2e-5 of the field); one and two fields stay within 4e-6.
#pragma once

#include "kernels_rt.cuh"

namespace pfcg {
namespace wide {

using T = float;
constexpr int MAXE = 16;

// One Stockham pass over P sequences (sequence p starts at buf + p*ld, padded
// indexing inside a sequence), NB butterflies per thread; threads without one
// repeat the last and store nothing (rt_pass_nb tells why).
template <int R, int NB, int SIGN, typename T>
__device__ __forceinline__ void stockham_nb(cplx<T>* buf, int ld, int total, int n, int Ns, const cplx<T>* __restrict__ tw,
                                            int t, int nthreads) {
	const int nR = n / R;
	const int tstep = n / (Ns * R);
	cplx<T> v[NB][R];
#pragma unroll
	for (int i = 0; i < NB; i++) {
		const int b = min(t + i * nthreads, total - 1);
		const int p = b / nR, j = b - p * nR;
		const cplx<T>* in = buf + p * ld;
#pragma unroll
		for (int r = 0; r < R; r++) v[i][r] = in[pad<T>(j + r * nR)];
	}
	__syncthreads();
#pragma unroll
	for (int i = 0; i < NB; i++) {
		const int b = min(t + i * nthreads, total - 1);
		const int p = b / nR, j = b - p * nR;
		const int jm = j % Ns;
		if (jm > 0) {
			const cplx<T>* twj = tw + jm * tstep;
#pragma unroll
			for (int r = 1; r < R; r++) {
				cplx<T> w = __ldg(twj + (r - 1) * jm * tstep);
				if (SIGN > 0) w.y = -w.y;
				v[i][r] = cmul(v[i][r], w);
			}
		}
		dft<R, SIGN, T>(v[i]);
		if (t + i * nthreads < total) {
			cplx<T>* out = buf + p * ld;
			const int d0 = (j - jm) * R + jm;
#pragma unroll
			for (int r = 0; r < R; r++) out[pad<T>(d0 + r * Ns)] = v[i][r];
		}
	}
	__syncthreads();
}

template <int R, int SIGN, int MAXE, typename T>
__device__ __forceinline__ void stockham_pass(cplx<T>* buf, int ld, int P, int n, int Ns, const cplx<T>* __restrict__ tw, int t,
                                              int nthreads) {
	const int total = P * (n / R);
	if (MAXE / R == 1 || total <= nthreads) stockham_nb<R, 1, SIGN, T>(buf, ld, total, n, Ns, tw, t, nthreads);
	else stockham_nb<R, MAXE / R, SIGN, T>(buf, ld, total, n, Ns, tw, t, nthreads);
}

// Full transform of P sequences of length plan.n in place in shared memory.
// RMAIN = MAXE; requires ceil(P * n / (R * nthreads)) <= MAXE / R for each radix R.
template <int SIGN, int MAXE, typename T>
__device__ __forceinline__ void fft_batch(cplx<T>* buf, int ld, int P, const RadixPlan& plan,
                                          const cplx<T>* __restrict__ tw, int t, int nthreads) {
	constexpr int RM = MAXE;
	const int n = plan.n;
	int Ns = 1;
	for (int s = 0; s < plan.nmain; s++) {
		stockham_pass<RM, SIGN, MAXE, T>(buf, ld, P, n, Ns, tw, t, nthreads);
		Ns *= RM;
	}
	if constexpr (RM > 8) {
		if (plan.rtail == 8) { stockham_pass<8, SIGN, MAXE, T>(buf, ld, P, n, Ns, tw, t, nthreads); Ns *= 8; }
	}
	if (plan.rtail == 4) { stockham_pass<4, SIGN, MAXE, T>(buf, ld, P, n, Ns, tw, t, nthreads); Ns *= 4; }
	else if (plan.rtail == 2) { stockham_pass<2, SIGN, MAXE, T>(buf, ld, P, n, Ns, tw, t, nthreads); Ns *= 2; }
	for (int s = 0; s < plan.n3; s++) { stockham_pass<3, SIGN, MAXE, T>(buf, ld, P, n, Ns, tw, t, nthreads); Ns *= 3; }
	for (int s = 0; s < plan.n5; s++) { stockham_pass<5, SIGN, MAXE, T>(buf, ld, P, n, Ns, tw, t, nthreads); Ns *= 5; }
	for (int s = 0; s < plan.n7; s++) { stockham_pass<7, SIGN, MAXE, T>(buf, ld, P, n, Ns, tw, t, nthreads); Ns *= 7; }
}

// Transforms S resident sequences in sub-batches of at most SB (so that the
// thread count needed by one fft_batch call stays within the CTA).
template <int SIGN, int MAXE, typename T>
__device__ __forceinline__ void fft_batches(cplx<T>* buf, int ld, int S, int SB, const RadixPlan& plan,
                                            const cplx<T>* __restrict__ tw, int t, int nthreads) {
	for (int b0 = 0; b0 < S; b0 += SB) {
		const int nb = (S - b0) < SB ? (S - b0) : SB;
		fft_batch<SIGN, MAXE, T>(buf + b0 * ld, ld, nb, plan, tw, t, nthreads);
	}
}


// the coefficients of entry_coef, with the compiler's choice of fused products
template <typename T, int U>
__device__ __forceinline__ void entry_coef_w(const StepK<T>& K, T k2, T (&A)[U], T (&Bn)[U],
                                           T (&cu)[npairs<T, U>()]) {
	if constexpr (U > 1) {
		const T G = expT<T>(K.ag * k2);
		const T G2 = G * G;
		int p = 0;
#pragma unroll
		for (int u = 0; u < U - 1; u++)
#pragma unroll
			for (int v = u + 1; v < U; v++) {
				T d2 = K.mu2[u][v] - k2;
				d2 *= d2;
				cu[p++] = K.beta[u][v] * d2 + K.eps[u][v] * G2;
			}
	}
	const T o = K.cc - (T)1 - K.cc * k2;
#pragma unroll
	for (int u = 0; u < U; u++) {
		T P = (T)1;
#pragma unroll
		for (int w = 0; w < MAXW; w++)
			if (w < K.W[u]) {
				const T q = K.nu2[u][w] - k2;
				P *= K.omega[u][w] * q * q + K.phi[u][w];
			}
		const T av = K.alpha[u] + K.betad[u] * P;
		const T x = o * av * K.dt;
		if (K.semi) {
			A[u] = (T)1 / ((T)1 - x);
			Bn[u] = o * K.dt * A[u];
			continue;
		}
		A[u] = expT<T>(x);
		if constexpr (sizeof(T) == 4) Bn[u] = o * K.dt * phi1f(x, A[u]);
		else Bn[u] = (av == (T)0) ? o * K.dt : etd_b<T>(A[u], x, av);
	}
}

__device__ __forceinline__ float k2_step_w(int kx, int ky, int Ny, float dkx, float dky) {
	const float kxv = (float)kx * dkx;
	const float kyv = (float)(ky < Ny / 2 ? ky : ky - Ny) * dky;
	return kxv * kxv + kyv * kyv;
}

template <int U, int MODE> __device__ __forceinline__ void xpass(const XArgs<T>& a, const int tile) {
	extern __shared__ __align__(128) unsigned char smem_raw[];
	cplx<T>* sm = reinterpret_cast<cplx<T>*>(smem_raw);
	const int Nx = a.g.Nx, Ny = a.g.Ny, R = a.g.R;
	const int H = Nx / 2 + 1;
	const int CH = U * R;
	const int P = (CH + 1) >> 1;
	const int ld = padded_len<T>(Nx);
	const int y0 = tile * R;
	const int tid = threadIdx.x, nt = blockDim.x;
	const long long tofs = (long long)tile * H * R;
	double off[U];
#pragma unroll
	for (int u = 0; u < U; u++) off[u] = a.off ? a.off[u] : 0.0;

	if constexpr (MODE == XP_R2C) {
		// real rows (minus their mean) -> pairs of channels in one complex sequence
		for (int x = tid; x < Nx; x += nt) {
#pragma unroll
			for (int p = 0; p < MAX_CH / 2; p++) {
				if (p < P) {
					const int c0 = 2 * p, c1 = 2 * p + 1;
					const int u0 = c0 % U, r0 = c0 / U, u1 = c1 % U, r1 = c1 / U;
					const double v0 = a.real[((long long)u0 * Ny + y0 + r0) * Nx + x] - (a.off ? a.off[u0] : 0.0);
					const double v1 = (c1 < CH) ? a.real[((long long)u1 * Ny + y0 + r1) * Nx + x] - (a.off ? a.off[u1] : 0.0) : 0.0;
					sm[p * ld + pad<T>(x)] = mk<T>((T)v0, (T)v1);
				}
			}
		}
	} else {
		// Hermitian-extended spectra of channel pairs: C = A + iB on 0..Nx/2,
		// conj(A) + i conj(B) on Nx/2+1..Nx-1; imaginary parts of the kx = 0 and
		// kx = Nx/2 entries are dropped like a c2r transform does.
		for (int k = tid; k < H; k += nt) {
			cplx<T> y[MAX_CH];
#pragma unroll
			for (int c = 0; c < MAX_CH; c++) {
				y[c] = mk<T>((T)0, (T)0);
				if (c < CH) {
					const int u = c % U, r = c / U;
					y[c] = a.work[u * a.wstride + tofs + (long long)k * R + r];
				}
			}
			const bool selfc = (k == 0) || (2 * k == Nx);
#pragma unroll
			for (int p = 0; p < MAX_CH / 2; p++) {
				if (p < P) {
					cplx<T> A = y[2 * p], B = y[2 * p + 1];
					if (selfc) { A.y = (T)0; B.y = (T)0; }
					sm[p * ld + pad<T>(k)] = mk<T>(A.x - B.y, A.y + B.x);
					if (k > 0 && 2 * k < Nx) sm[p * ld + pad<T>(Nx - k)] = mk<T>(A.x + B.y, B.x - A.y);
				}
			}
		}
		__syncthreads();
		fft_batches<+1, MAXE, T>(sm, ld, P, a.wsb, a.wplan, a.wtw, tid, nt);
	}

	if constexpr (MODE == XP_STEP) {
		double acc[U];
#pragma unroll
		for (int i = 0; i < U; i++) acc[i] = 0.0;
		bool nan = false;
		T lam[U], del[U], gam[U][U], alp[U][U], offT[U];
#pragma unroll
		for (int u = 0; u < U; u++) {
			offT[u] = (T)off[u];
			lam[u] = (T)a.m.lambda[u];
			del[u] = (T)a.m.delta[u];
#pragma unroll
			for (int v = 0; v < U; v++) { gam[u][v] = (T)a.m.gamma[u][v]; alp[u][v] = (T)a.m.alpha[u][v]; }
		}
		for (int x = tid; x < Nx; x += nt) {
			T z[MAX_CH];
#pragma unroll
			for (int p = 0; p < MAX_CH / 2; p++) {
				if (p < P) {
					const cplx<T> v = sm[p * ld + pad<T>(x)];
					z[2 * p] = v.x;
					z[2 * p + 1] = v.y;
				}
			}
#pragma unroll
			for (int r = 0; r < MAX_CH / U; r++) {
				if (r < R) {
					T mv[U], mc[U];
#pragma unroll
					for (int u = 0; u < U; u++) {
						mv[u] = z[r * U + u] + offT[u];
						nan |= (mv[u] != mv[u]);
						mc[u] = (T)0;
					}
#pragma unroll
					for (int u = 0; u < U - 1; u++)
#pragma unroll
						for (int v = u + 1; v < U; v++) {
							mc[u] += alp[u][v] * mv[v] + (T)0.5 * gam[u][v] * ((T)2 * mv[u] * mv[v] + mv[v] * mv[v]);
							mc[v] += alp[u][v] * mv[u] + (T)0.5 * gam[u][v] * ((T)2 * mv[v] * mv[u] + mv[u] * mv[u]);
						}
#pragma unroll
					for (int u = 0; u < U; u++) {
						const T m2 = mv[u] * mv[u];
						const T nl = lam[u] + gam[u][u] * m2 + del[u] * mv[u] * m2 + mc[u];
						z[r * U + u] = nl;
						acc[u] += (double)nl;
					}
				}
			}
#pragma unroll
			for (int p = 0; p < MAX_CH / 2; p++)
				if (p < P) sm[p * ld + pad<T>(x)] = mk<T>(z[2 * p], (2 * p + 1 < CH) ? z[2 * p + 1] : (T)0);
		}
		if (nan) atomicOr(a.flag, FLAG_NAN);
		block_reduce_put<U>(acc, a.part ? a.part + (long long)tile * U : a.acc, a.part != nullptr);
	}

	__syncthreads();
	fft_batches<-1, MAXE, T>(sm, ld, P, a.wsb, a.wplan, a.wtw, tid, nt);
	// split each pair: Za = (C[k] + conj C[-k]) / 2, Zb = (C[k] - conj C[-k]) / (2i)
	const T half = (T)0.5;
	for (int k = tid; k < H; k += nt) {
		const int km = (k == 0) ? 0 : Nx - k;
		cplx<T> zz[MAX_CH];
#pragma unroll
		for (int p = 0; p < MAX_CH / 2; p++) {
			if (p < P) {
				const cplx<T> Ck = sm[p * ld + pad<T>(k)];
				const cplx<T> Cm = sm[p * ld + pad<T>(km)];
				zz[2 * p] = mk<T>(half * (Ck.x + Cm.x), half * (Ck.y - Cm.y));
				zz[2 * p + 1] = mk<T>(half * (Ck.y + Cm.y), half * (Cm.x - Ck.x));
			}
		}
#pragma unroll
		for (int c = 0; c < MAX_CH; c++) {
			if (c < CH) {
				const int u = c % U, r = c / U;
				a.work[u * a.wstride + tofs + (long long)k * R + r] = zz[c];
			}
		}
	}
}

template <int U, int MODE> __device__ __forceinline__ void ypass(const YArgs<T>& a, const int grp) {
	extern __shared__ __align__(128) unsigned char smem_raw[];
	cplx<T>* sm = reinterpret_cast<cplx<T>*>(smem_raw);
	const int Nx = a.g.Nx, H = a.g.H, Ny = a.g.Ny, R = a.g.R, CC = a.g.CC;
	const int tid = threadIdx.x, nt = blockDim.x;
	const int kx0 = grp * CC;
	if (MODE == YP_STEP && kx0 >= H) { // the CTA of the k = 0 update
		ypass_mean_update<T, U>(a, tid, nt);
		return;
	}
	const int S = U * CC;
	const int ld = padded_len<T>(Ny);
	const int ncol = min(CC, H - kx0);
	const int ntile = Ny / R;
	const long long tileH = (long long)H * R;
	const int chunk = CC * R;
#pragma unroll
	for (int u = 0; u < U; u++) {
		const cplx<T>* src = a.work + u * a.wstride + (long long)kx0 * R;
		for (int e = tid; e < ntile * chunk; e += nt) {
			const int t = e / chunk, rem = e - t * chunk;
			const int c = rem / R, r = rem - c * R;
			cplx<T> v = mk<T>((T)0, (T)0);
			if (c < ncol) v = src[t * tileH + rem];
			sm[(u * CC + c) * ld + pad<T>(t * R + r)] = v;
		}
	}
	__syncthreads();
	fft_batches<-1, MAXE, T>(sm, ld, S, a.wsb, a.wplan, a.wtw, tid, nt);
	if constexpr (MODE == YP_STEP) {
		const StepK<T>& K = a.k;
		const T dkxT = K.dkx, dkyT = K.dky;
		auto apply = [&](int c, int kx, int ky, const cplx<T>(&Nv)[U], const T(&A)[U], const T(&Bn)[U],
		                 const T(&cu)[npairs<T, U>()]) {
			cplx<T> Mv[U];
#pragma unroll
			for (int u = 0; u < U; u++) Mv[u] = cscale(sm[(u * CC + c) * ld + pad<T>(ky)], K.invN);
			int p = 0;
#pragma unroll
			for (int u = 0; u < U - 1; u++)
#pragma unroll
				for (int v = u + 1; v < U; v++, p++) {
					Mv[u] = cadd(Mv[u], cscale(Nv[v], cu[p]));
					Mv[v] = cadd(Mv[v], cscale(Nv[u], cu[p]));
				}
			const bool origin = (kx == 0 && ky == 0);
#pragma unroll
			for (int u = 0; u < U; u++) {
				cplx<T> nn = cadd(cscale(Nv[u], A[u]), cscale(Mv[u], Bn[u]));
				if (origin) nn = mk<T>((T)0, (T)0);
				__stcs(a.spec + u * a.sstride + (long long)kx * Ny + ky, nn);
				sm[(u * CC + c) * ld + pad<T>(ky)] = nn;
			}
		};
		for (int e = tid; e < CC * Ny; e += nt) {
			const int c = e / Ny, ky = e - c * Ny;
			if (c >= ncol) continue;
			const int kx = kx0 + c;
			cplx<T> Nv[U];
#pragma unroll
			for (int u = 0; u < U; u++) Nv[u] = a.spec[u * a.sstride + (long long)kx * Ny + ky];
			T A[U], Bn[U], cu[npairs<T, U>()];
			entry_coef_w<T, U>(K, k2_step_w(kx, ky, Ny, dkxT, dkyT), A, Bn, cu);
			apply(c, kx, ky, Nv, A, Bn, cu);
		}
	} else {
		const T invN = (T)(1.0 / ((double)Nx * (double)Ny));
		for (int e = tid; e < CC * Ny; e += nt) {
			const int c = e / Ny, ky = e - c * Ny;
			if (c >= ncol) continue;
			const int kx = kx0 + c;
			const long long si = (long long)kx * Ny + ky;
#pragma unroll
			for (int u = 0; u < U; u++) {
				cplx<T> nn = cscale(sm[(u * CC + c) * ld + pad<T>(ky)], invN);
				if (kx == 0 && ky == 0) nn = mk<T>((T)0, (T)0);
				a.spec[u * a.sstride + si] = nn;
				sm[(u * CC + c) * ld + pad<T>(ky)] = nn;
			}
		}
	}
	// kx = 0 and kx = Nx/2 columns: keep them exactly Hermitian
	const bool has0 = (kx0 == 0);
	const int kn = Nx / 2;
	const bool hasn = (kn >= kx0 && kn < kx0 + ncol);
	if (has0 || hasn) {
		__syncthreads();
#pragma unroll
		for (int u = 0; u < U; u++) {
			if (has0) hermitian_column<T>(sm + (u * CC) * ld, a.spec + u * a.sstride, Ny, tid, nt);
			if (hasn)
				hermitian_column<T>(sm + (u * CC + (kn - kx0)) * ld, a.spec + u * a.sstride + (long long)kn * Ny, Ny, tid, nt);
		}
	}
	__syncthreads();
	fft_batches<+1, MAXE, T>(sm, ld, S, a.wsb, a.wplan, a.wtw, tid, nt);
#pragma unroll
	for (int u = 0; u < U; u++) {
		cplx<T>* dst = a.work + u * a.wstride + (long long)kx0 * R;
		for (int e = tid; e < ntile * chunk; e += nt) {
			const int t = e / chunk, rem = e - t * chunk;
			const int c = rem / R, r = rem - c * R;
			if (c < ncol) dst[t * tileH + rem] = sm[(u * CC + c) * ld + pad<T>(t * R + r)];
		}
	}
}

template <int U, int MODE> __global__ void __launch_bounds__(MAXNT, 1) xwide_kernel(const XArgs<T> a, int) {
	asm volatile("griddepcontrol.wait;" ::: "memory");
	asm volatile("griddepcontrol.launch_dependents;");
	xpass<U, MODE>(a, blockIdx.x);
}
template <int U, int MODE> __global__ void __launch_bounds__(MAXNT, 1) ywide_kernel(const YArgs<T> a, int) {
	asm volatile("griddepcontrol.wait;" ::: "memory");
	asm volatile("griddepcontrol.launch_dependents;");
	ypass<U, MODE>(a, blockIdx.x);
}

template <int U, int MODE> cudaError_t xlaunch(const XArgs<T>& a, const LaunchCfg& c, cudaStream_t s) {
	auto k = xwide_kernel<U, MODE>;
	static unsigned long long mask = 0;
	smem_attr(k, mask);
	return pdl_launch(k, c.grid, c.block, c.smem, s, a, 0);
}
template <int U, int MODE> cudaError_t ylaunch(const YArgs<T>& a, const LaunchCfg& c, cudaStream_t s) {
	auto k = ywide_kernel<U, MODE>;
	static unsigned long long mask = 0;
	smem_attr(k, mask);
	return pdl_launch(k, c.grid, c.block, c.smem, s, a, 0);
}

} // namespace wide

template <int U> cudaError_t wide_launch_x(int mode, const XArgs<float>& a, const LaunchCfg& c, cudaStream_t s) {
	return mode == XP_STEP ? wide::xlaunch<U, XP_STEP>(a, c, s) : wide::xlaunch<U, XP_R2C>(a, c, s);
}
template <int U> cudaError_t wide_launch_y(int mode, const YArgs<float>& a, const LaunchCfg& c, cudaStream_t s) {
	return mode == YP_STEP ? wide::ylaunch<U, YP_STEP>(a, c, s) : wide::ylaunch<U, YP_INIT>(a, c, s);
}

} // namespace pfcg
