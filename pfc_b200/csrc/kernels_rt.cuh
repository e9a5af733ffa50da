// x- and y-pass kernels of run-time lengths (fft_rt.cuh's plans): every mode at
// sizes without specialised STEP kernels, and the other modes (evaluate, c2r,
// r2c, the first spectrum, weighted spectra) at every size.
//
// Both keep the swapped form of fft_rt.cuh between an inverse transform's load
// and its use: element (re, im) is held as (im, re).
//
// x-pass: R rows of U fields make P = ceil(U R / 2) complex sequences. For even U
// (and at R = 1) a sequence is fields 2h, 2h + 1 of a row, as in the specialised
// kernels, so that results don't depend on R; for odd U it is rows 2q, 2q + 1 of
// one field. Rows 2q and 2q + 1 are adjacent in `work` (one 16-byte access in FP32).
// y-pass: CC columns of U fields; entries ky and Ny - ky have the same k^2, so a
// thread takes such pairs and evaluates the update's coefficients once.
// The k = 0 update (FP64, all row tiles' sums) is a CTA of its own: it depends
// on nothing the column groups compute, and in the group of kx = 0 it would
// lengthen the kernel's longest chain.
#pragma once

#include "kernels_impl.cuh"

namespace pfcg {

// two complexes at an even element index (16-byte aligned in FP32)
__device__ __forceinline__ void ld2(const float2* p, float2& a, float2& b) {
	const float4 q = *reinterpret_cast<const float4*>(p);
	a = make_float2(q.x, q.y);
	b = make_float2(q.z, q.w);
}
__device__ __forceinline__ void ld2(const double2* p, double2& a, double2& b) {
	a = p[0];
	b = p[1];
}
__device__ __forceinline__ void st2(float2* p, float2 a, float2 b) { *reinterpret_cast<float4*>(p) = make_float4(a.x, a.y, b.x, b.y); }
__device__ __forceinline__ void st2(double2* p, double2 a, double2 b) {
	p[0] = a;
	p[1] = b;
}

// Brings the plan's twiddles into L1 (one load per 128-byte line). Issued before
// the wait for the previous kernel, which must not be the one that writes the table:
// tables are written when a handle is made, and a launch that follows a kernel
// writing one is plain (LaunchCfg), since L1 could keep the lines of before.
template <typename T> __device__ __forceinline__ void rt_warm_twiddles(const cplx<T>* tw, int ntw, int t, int nt) {
	const char* p = reinterpret_cast<const char*>(tw);
	const int bytes = ntw * (int)sizeof(cplx<T>);
	for (int b = t * 128; b < bytes; b += nt * 128) {
		unsigned v;
		asm volatile("ld.global.nc.u32 %0, [%1];" : "=r"(v) : "l"(p + b));
	}
}

// nonlinear term of U fields at one point, pfc-relax.c:1188-1209
template <typename T, int U> __device__ __forceinline__ void nl_terms(const NlK<T>& K, const T (&m)[U], T (&nl)[U]) {
	T mc[U];
#pragma unroll
	for (int u = 0; u < U; u++) mc[u] = (T)0;
#pragma unroll
	for (int u = 0; u < U - 1; u++)
#pragma unroll
		for (int v = u + 1; v < U; v++) {
			// alpha m_v + gamma / 2 (2 m_u m_v + m_v^2)
			const T g = mul_rn((T)0.5, K.gam[u][v]), uv2 = mul_rn((T)2, mul_rn(m[u], m[v]));
			mc[u] = fma_rn(g, fma_rn(m[v], m[v], uv2), fma_rn(K.alp[u][v], m[v], mc[u]));
			mc[v] = fma_rn(g, fma_rn(m[u], m[u], uv2), fma_rn(K.alp[u][v], m[u], mc[v]));
		}
#pragma unroll
	for (int u = 0; u < U; u++) {
		const T m2 = mul_rn(m[u], m[u]);
		nl[u] = fma_rn(mul_rn(K.del[u], m[u]), m2, fma_rn(K.gam[u][u], m2, K.lam[u])) + mc[u];
	}
}

// local energy terms of U fields at one point (FP64), pfc-relax.c:1094-1118
template <int U> __device__ __forceinline__ double local_energy(const Model& m, const double (&n)[U]) {
	double f = 0.0;
#pragma unroll
	for (int u = 0; u < U; u++) {
		const double n1 = n[u], n2 = n1 * n1;
		f += m.lambda[u] * n1 + 0.5 * m.alpha[u][u] * n2 + (1.0 / 3.0) * m.gamma[u][u] * n1 * n2 + 0.25 * m.delta[u] * n2 * n2;
#pragma unroll
		for (int v = u + 1; v < U; v++) {
			const double nv = n[v];
			f += m.alpha[u][v] * n1 * nv + 0.5 * m.gamma[u][v] * (n2 * nv + n1 * nv * nv);
		}
	}
	return f;
}

template <typename T, int U, bool STEP>
__device__ __forceinline__ void rt_xpass(const XArgs<T>& a, const int mode_, const int tile) {
	extern __shared__ __align__(128) unsigned char smem_raw[];
	cplx<T>* sm = reinterpret_cast<cplx<T>*>(smem_raw);
	const int mode = STEP ? XP_STEP : mode_;
	const int Nx = a.g.Nx, Ny = a.g.Ny, H = a.g.H, R = a.g.R;
	const int ld = a.plan.ld, sh = a.plan.sh;
	const int tid = threadIdx.x, nt = blockDim.x;
	const int P = (U * R + 1) >> 1;
	const int hq = R >> 1, lq = R > 1 ? __ffs(hq) - 1 : 0; // row pairs of a tile
	const int y0 = tile * R;
	constexpr bool IL = WORK_IL<T, U>;
	const long long tofs = (long long)tile * H * (IL ? U * R : R), us = IL ? R : a.wstride;
	constexpr int F = (U + 1) / 2;             // sequences per row when fields are paired
	const bool byrow = U % 2 == 1 && R > 1;    // rows paired
	T offT[U];
	double off[U];
	constexpr int NACC = STEP ? U : 1 + U;
	double acc[NACC];
#pragma unroll
	for (int i = 0; i < NACC; i++) acc[i] = 0.0;
	bool nan = false;
	// The first transform (the inverse one, or R2C's forward one), then the
	// pointwise work, then the second one: one copy of the transform's code.
	// With `warm` a turn before them transforms whatever shared memory holds, to
	// fetch that code, the plan's constants and the twiddles while the previous
	// kernel still runs (cold, the first transform of 512 points took 4700 cycles,
	// the second 2900).
#pragma unroll 1
	for (int turn = STEP && a.warm ? -1 : 0; turn < 2; turn++) {
		if (turn == 0) {
			// programmatic dependent launch (pdl_launch): the previous kernel's results
			// are complete and visible after this wait; a plain launch returns at once
			asm volatile("griddepcontrol.wait;" ::: "memory");
			asm volatile("griddepcontrol.launch_dependents;");
#pragma unroll
			for (int u = 0; u < U; u++) {
				off[u] = a.off ? a.off[u] : 0.0;
				offT[u] = (T)off[u];
			}

			if (mode == XP_R2C) {
				// real rows less their mean, two to a sequence
				if (byrow) {
#pragma unroll
					for (int u = 0; u < U; u++)
						for (int e = tid; e < Nx * hq; e += nt) {
							const int q = hq > 1 ? rt_div(e, a.plan.mn) : 0, x = e - q * Nx;
							const double* r = a.real + ((long long)u * Ny + y0 + 2 * q) * Nx + x;
							sm[(u * hq + q) * ld + rt_pad(x, sh)] = mk<T>((T)(r[0] - off[u]), (T)(r[Nx] - off[u]));
						}
				} else {
					for (int e = tid; e < Nx * R; e += nt) {
						const int r = R > 1 ? rt_div(e, a.plan.mn) : 0, x = e - r * Nx;
						const double* v = a.real + ((long long)(y0 + r)) * Nx + x;
#pragma unroll
						for (int h = 0; h < F; h++) {
							const double v0 = v[(long long)(2 * h) * Ny * Nx] - off[2 * h];
							const double v1 = 2 * h + 1 < U ? v[(long long)(2 * h + 1) * Ny * Nx] - off[2 * h + 1 < U ? 2 * h + 1 : 0] : 0.0;
							sm[(r * F + h) * ld + rt_pad(x, sh)] = mk<T>((T)v0, (T)v1);
						}
					}
				}
			} else {
				// Hermitian-extended spectra of the pairs, C = A + iB on 0 .. Nx/2 and
				// conj A + i conj B above, swapped; the imaginary parts of the kx = 0 and
				// kx = Nx/2 entries are dropped like a c2r transform does
				auto put = [&](cplx<T>* s, int k, cplx<T> A, cplx<T> B) {
					if (k == 0 || 2 * k == Nx) { A.y = (T)0; B.y = (T)0; }
					s[rt_pad(k, sh)] = mk<T>(A.y + B.x, A.x - B.y);
					if (k > 0 && 2 * k < Nx) s[rt_pad(Nx - k, sh)] = mk<T>(B.x - A.y, A.x + B.y);
				};
				if (byrow) {
#pragma unroll
					for (int u = 0; u < U; u++) {
						const cplx<T>* src = a.work + u * a.wstride + tofs;
#pragma unroll 4
						for (int e = tid; e < H << lq; e += nt) {
							cplx<T> A, B;
							ld2(src + 2 * e, A, B);
							put(sm + (u * hq + (e & (hq - 1))) * ld, e >> lq, A, B);
						}
					}
				} else if (U % 2 == 0 && R > 1) {
#pragma unroll
					for (int h = 0; h < F; h++) {
						const cplx<T>* src = a.work + (2 * h) * us + tofs;
#pragma unroll 4
						for (int e = tid; e < H << lq; e += nt) {
							const int at = 2 * (IL ? e + (e >> lq) * (U - 1) * hq : e);
							cplx<T> A0, A1, B0, B1;
							ld2(src + at, A0, A1);
							ld2(src + us + at, B0, B1);
							cplx<T>* s = sm + (2 * (e & (hq - 1)) * F + h) * ld;
							put(s, e >> lq, A0, B0);
							put(s + F * ld, e >> lq, A1, B1);
						}
					}
				} else {
#pragma unroll
					for (int h = 0; h < F; h++) {
						const cplx<T>* s0 = a.work + (2 * h) * us + tofs;
						const cplx<T>* s1 = s0 + us;
						constexpr int ks = IL ? U : 1;
#pragma unroll 4
						for (int k = tid; k < H; k += nt) put(sm + h * ld, k, s0[k * ks], 2 * h + 1 < U ? s1[k * ks] : mk<T>((T)0, (T)0));
					}
				}
			}

		} else if (turn == 1) {
			// the real fields: item (q, x) holds two rows of every field, or item (r, x) one
			if (byrow) {
				for (int e = tid; e < Nx * hq; e += nt) {
					const int q = hq > 1 ? rt_div(e, a.plan.mn) : 0, x = e - q * Nx;
					cplx<T>* s = sm + q * ld + rt_pad(x, sh);
					if (STEP) {
						T m0[U], m1[U], n0[U], n1[U];
#pragma unroll
						for (int u = 0; u < U; u++) {
							const cplx<T> z = s[u * hq * ld];
							m0[u] = z.y + offT[u];
							m1[u] = z.x + offT[u];
							nan |= (m0[u] != m0[u]) | (m1[u] != m1[u]);
						}
						nl_terms<T, U>(a.k, m0, n0);
						nl_terms<T, U>(a.k, m1, n1);
#pragma unroll
						for (int u = 0; u < U; u++) {
							acc[u] += (double)n0[u];
							acc[u] += (double)n1[u];
							s[u * hq * ld] = mk<T>(n0[u], n1[u]);
						}
					} else if (mode == XP_EVAL) {
						double m0[U], m1[U];
#pragma unroll
						for (int u = 0; u < U; u++) {
							const cplx<T> z = s[u * hq * ld];
							m0[u] = (double)z.y + off[u];
							m1[u] = (double)z.x + off[u];
							acc[NACC - U + u] += m0[u];
							acc[NACC - U + u] += m1[u];
						}
						acc[0] += local_energy<U>(a.m, m0);
						acc[0] += local_energy<U>(a.m, m1);
					} else {
#pragma unroll
						for (int u = 0; u < U; u++) {
							const cplx<T> z = s[u * hq * ld];
							double* r = a.real + ((long long)u * Ny + y0 + 2 * q) * Nx + x;
							r[0] = (double)z.y + off[u];
							r[Nx] = (double)z.x + off[u];
						}
					}
				}
			} else {
				for (int e = tid; e < Nx * R; e += nt) {
					const int r = R > 1 ? rt_div(e, a.plan.mn) : 0, x = e - r * Nx;
					cplx<T>* s = sm + r * F * ld + rt_pad(x, sh);
					T z[U + 1];
#pragma unroll
					for (int h = 0; h < F; h++) {
						z[2 * h] = s[h * ld].y;
						z[2 * h + 1 < U ? 2 * h + 1 : U] = s[h * ld].x;
					}
					if (STEP) {
						T m[U], n[U];
#pragma unroll
						for (int u = 0; u < U; u++) {
							m[u] = z[u] + offT[u];
							nan |= m[u] != m[u];
						}
						nl_terms<T, U>(a.k, m, n);
#pragma unroll
						for (int u = 0; u < U; u++) acc[u] += (double)n[u];
#pragma unroll
						for (int h = 0; h < F; h++) s[h * ld] = mk<T>(n[2 * h], 2 * h + 1 < U ? n[2 * h + 1 < U ? 2 * h + 1 : 0] : (T)0);
					} else if (mode == XP_EVAL) {
						double m[U];
#pragma unroll
						for (int u = 0; u < U; u++) {
							m[u] = (double)z[u] + off[u];
							acc[NACC - U + u] += m[u];
						}
						acc[0] += local_energy<U>(a.m, m);
					} else {
#pragma unroll
						for (int u = 0; u < U; u++) a.real[((long long)u * Ny + y0 + r) * Nx + x] = (double)z[u] + off[u];
					}
				}
			}
			if (!STEP) break;
		}
		__syncthreads();
		rt_fft<T>(sm, a.plan, P, a.sb, a.tw, tid, nt);
		if (!STEP && mode == XP_R2C) break;
	}
	if (STEP && nan) atomicOr(a.flag, FLAG_NAN);

	if (STEP || mode == XP_R2C) {
		// split each pair: Za = (C[k] + conj C[-k]) / 2, Zb = (C[k] - conj C[-k]) / (2i)
		const T half = (T)0.5;
		auto split = [&](const cplx<T>* s, int k, cplx<T>& za, cplx<T>& zb) {
			const cplx<T> Ck = s[rt_pad(k, sh)], Cm = s[rt_pad(k == 0 ? 0 : Nx - k, sh)];
			za = mk<T>(half * (Ck.x + Cm.x), half * (Ck.y - Cm.y));
			zb = mk<T>(half * (Ck.y + Cm.y), half * (Cm.x - Ck.x));
		};
		if (byrow) {
#pragma unroll
			for (int u = 0; u < U; u++) {
				cplx<T>* dst = a.work + u * a.wstride + tofs;
				for (int e = tid; e < H << lq; e += nt) {
					cplx<T> za, zb;
					split(sm + (u * hq + (e & (hq - 1))) * ld, e >> lq, za, zb);
					st2(dst + 2 * e, za, zb);
				}
			}
		} else if (U % 2 == 0 && R > 1) {
#pragma unroll
			for (int h = 0; h < F; h++) {
				cplx<T>* dst = a.work + (2 * h) * us + tofs;
				for (int e = tid; e < H << lq; e += nt) {
					const int at = 2 * (IL ? e + (e >> lq) * (U - 1) * hq : e);
					cplx<T> a0, a1, b0, b1;
					const cplx<T>* s = sm + (2 * (e & (hq - 1)) * F + h) * ld;
					split(s, e >> lq, a0, b0);
					split(s + F * ld, e >> lq, a1, b1);
					st2(dst + at, a0, a1);
					st2(dst + us + at, b0, b1);
				}
			}
		} else {
#pragma unroll
			for (int h = 0; h < F; h++) {
				cplx<T>* d0 = a.work + (2 * h) * us + tofs;
				constexpr int ks = IL ? U : 1;
				for (int k = tid; k < H; k += nt) {
					cplx<T> za, zb;
					split(sm + h * ld, k, za, zb);
					d0[k * ks] = za;
					if (2 * h + 1 < U) d0[us + k * ks] = zb;
				}
			}
		}
	}
	if (STEP || mode == XP_EVAL) block_reduce_put<NACC>(acc, a.part ? a.part + (long long)tile * NACC : a.acc, a.part != nullptr);
}

// Hermitian projection of a resident column in swapped form, and of its spectral state (hermitian_column)
template <typename T>
__device__ __forceinline__ void rt_hermitian_column(cplx<T>* col, cplx<T>* spec_col, int Ny, int sh, int tid, int nt) {
	const int half = Ny / 2;
	for (int j = tid; j <= half; j += nt) {
		// thread j reads and writes entries j and Ny - j, which no other thread touches
		const int jn = j == 0 ? 0 : Ny - j;
		const cplx<T> a = col[rt_pad(j, sh)], b = col[rt_pad(jn, sh)];
		const cplx<T> p = mk<T>((T)0.5 * (a.y + b.y), (T)0.5 * (a.x - b.x));
		col[rt_pad(j, sh)] = mk<T>(p.y, p.x);
		spec_col[j] = p;
		if (jn != j) {
			col[rt_pad(jn, sh)] = mk<T>(-p.y, p.x);
			spec_col[jn] = cconj(p);
		}
	}
}

// the k-space weight of one entry (YP_WEIGHT) times the spectral state
template <typename T> __device__ __forceinline__ cplx<T> weighted_entry(const YArgs<T>& a, int kx, int ky) {
	const int Ny = a.g.Ny;
	const long long si = (long long)kx * Ny + ky;
	const double kxv = kx * a.g.dkx, kyv = (ky < Ny / 2 ? ky : ky - Ny) * a.g.dky;
	const double k2 = kxv * kxv + kyv * kyv;
	if (a.wkind == W_OR) {
		// orientation kernel K = exp(-(|k| - 1)^2 / (2 sk^2)) exp(i fold phi),
		// fields.c:143-153; real and imaginary parts are even in k
		// for even fold, so each part maps the field pair to a real field
		const double q = sqrt(k2) - 1.0;
		const double rad = exp(-0.5 * q * q / (a.wp.sk * a.wp.sk));
		double sn, cs;
		sincos(a.wp.fold * atan2(kyv, kxv), &sn, &cs);
		const T kr = (T)(rad * cs), ki = (T)(rad * sn);
		const cplx<T> s0 = a.spec[si], s1 = a.spec[a.sstride + si];
		return a.wp.part == 0 ? csub(cscale(s0, kr), cscale(s1, ki)) : cadd(cscale(s0, ki), cscale(s1, kr));
	}
	const cplx<T> v = a.spec[a.wsrc * a.sstride + si];
	double w = 1.0;
	if (a.wkind == W_P) {
#pragma unroll
		for (int q = 0; q < MAXW; q++)
			if (q < a.wp.W) {
				const double d = a.wp.nu2[q] - k2;
				w *= a.wp.omega[q] * d * d + a.wp.phi[q];
			}
	} else if (a.wkind == W_G) {
		w = exp(-0.5 / a.m.sigma / a.m.sigma * k2);
	} else if (a.wkind == W_Q) {
		const double d = a.wp.mu2 - k2;
		w = d * d;
	} else if (a.wkind == W_GS || a.wkind == W_DG) {
		w = exp(-0.5 * k2 / (a.wp.gs * a.wp.gs));
	}
	if (a.wkind == W_DG) {
		// i k_dir G(k) times the field (fields.c:260-271 on the smoothed spectrum)
		const T f = (T)((a.wp.dir == 0 ? kxv : kyv) * w);
		return mk<T>(-f * v.y, f * v.x);
	}
	return cscale(v, (T)w);
}

template <typename T, int U, bool STEP>
__device__ __forceinline__ void rt_ypass(const YArgs<T>& a, const int mode_, const int grp) {
	extern __shared__ __align__(128) unsigned char smem_raw[];
	cplx<T>* sm = reinterpret_cast<cplx<T>*>(smem_raw);
	const int mode = STEP ? YP_STEP : mode_;
	const int H = a.g.H, Ny = a.g.Ny, R = a.g.R, CC = a.g.CC;
	const int ld = a.plan.ld, sh = a.plan.sh;
	const int tid = threadIdx.x, nt = blockDim.x;
	const int S = U * CC, kx0 = grp * CC;
	if (STEP && kx0 >= H) { // the CTA of the k = 0 update
		asm volatile("griddepcontrol.wait;" ::: "memory"); // as in rt_xpass
		asm volatile("griddepcontrol.launch_dependents;");
		ypass_mean_update<T, U>(a, tid, nt);
		return;
	}
	const int ncol = min(CC, H - kx0);
	const long long tileH = (long long)H * (WORK_IL<T, U> ? U * R : R);
	const int lR = __ffs(R) - 1, lC = __ffs(CC) - 1;
	const int nh = Ny / 2;

	// With `early`, before the wait for the x-pass: the spectral state into shared
	// memory (asynchronous copies), the update's coefficients, and a transform of
	// nothing as in rt_xpass. The state is that of the y-pass before: the x-pass in
	// between lets this kernel start only after its own wait for that y-pass.
	cplx<T>* eN = sm + ((S * ld + 1) & ~1);                 // [u][c][ky], on 16 bytes
	T* eK = reinterpret_cast<T*>(eN + S * Ny);              // [coefficient][pair]
	const int nk = (nh << lC) + CC;
	if (STEP && a.early) {
#pragma unroll
		for (int u = 0; u < U; u++) {
			const char* src = reinterpret_cast<const char*>(a.spec + u * a.sstride + (long long)kx0 * Ny);
			const unsigned dst = (unsigned)__cvta_generic_to_shared(eN + u * CC * Ny);
			for (int i = tid * 16; i < ncol * Ny * (int)sizeof(cplx<T>); i += nt * 16)
				asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + i), "l"(src + i) : "memory");
		}
		asm volatile("cp.async.commit_group;" ::: "memory");
		for (int e = tid; e < nk; e += nt) {
			const bool second = e >= nh << lC; // ky = Ny / 2 of column e - CC nh
			const int c = second ? e - (nh << lC) : CC > 1 ? rt_div(e, a.plan.mnh) : 0;
			T A[U], Bn[U], cu[npairs<T, U>()];
			entry_coef<T, U>(a.k, k2_step<T>(kx0 + c, second ? nh : e - c * nh, Ny, a.k.dkx, a.k.dky), A, Bn, cu);
#pragma unroll
			for (int u = 0; u < U; u++) {
				eK[u * nk + e] = A[u];
				eK[(U + u) * nk + e] = Bn[u];
			}
#pragma unroll
			for (int p = 0; p < U * (U - 1) / 2; p++) eK[(2 * U + p) * nk + e] = cu[p];
		}
	}

#pragma unroll 1
	for (int turn = STEP && a.early ? -1 : 0; turn < 2; turn++) {
		if (turn == 0) {
			asm volatile("griddepcontrol.wait;" ::: "memory"); // as in rt_xpass
			asm volatile("griddepcontrol.launch_dependents;");
			if (mode == YP_WEIGHT) continue;
			if (STEP && !a.early) {
				// this group's spectral state into L2 while the forward transform runs
				const int lines = ncol * Ny * (int)sizeof(cplx<T>) / 128;
#pragma unroll
				for (int u = 0; u < U; u++) {
					const char* p = reinterpret_cast<const char*>(a.spec + u * a.sstride + (long long)kx0 * Ny);
					for (int i = tid; i < lines; i += nt) asm volatile("prefetch.global.L2 [%0];" ::"l"(p + i * 128));
				}
			}
			// CC columns of every row tile of `work`, two rows at a time where the tile has them
			if constexpr (WORK_IL<T, U>) {
				const cplx<T>* src = a.work + kx0 * U * R;
				if (R > 1) {
#pragma unroll 4
					for (int e = tid; e < nh * U << lC; e += nt) {
						const int r = 2 * e & (R - 1), i = e >> (lR - 1), u = i % U, c = i / U & (CC - 1), t = i / U >> lC;
						cplx<T> v0 = mk<T>((T)0, (T)0), v1 = v0;
						if (c < ncol) ld2(src + t * tileH + (c * U + u) * R + r, v0, v1);
						cplx<T>* d = sm + (u * CC + c) * ld + rt_pad(t * R + r, sh);
						d[0] = v0;
						d[1] = v1;
					}
				} else {
#pragma unroll 4
					for (int e = tid; e < Ny * U << lC; e += nt) {
						const int u = e % U, c = e / U & (CC - 1), t = e / U >> lC;
						sm[(u * CC + c) * ld + rt_pad(t, sh)] = c < ncol ? src[t * tileH + c * U + u] : mk<T>((T)0, (T)0);
					}
				}
			} else {
#pragma unroll
				for (int u = 0; u < U; u++) {
					const cplx<T>* src = a.work + u * a.wstride + (long long)kx0 * R;
					cplx<T>* dst = sm + u * CC * ld;
					if (R > 1) {
#pragma unroll 4
						for (int i = tid; i < nh << lC; i += nt) {
							const int e = 2 * i, r = e & (R - 1), c = (e >> lR) & (CC - 1), t = e >> (lR + lC);
							cplx<T> v0 = mk<T>((T)0, (T)0), v1 = v0;
							if (c < ncol) ld2(src + t * tileH + c * R + r, v0, v1);
							cplx<T>* d = dst + c * ld + rt_pad(t * R + r, sh);
							d[0] = v0;
							d[1] = v1;
						}
					} else {
#pragma unroll 4
						for (int e = tid; e < Ny << lC; e += nt) {
							const int c = e & (CC - 1), t = e >> lC;
							dst[c * ld + rt_pad(t, sh)] = c < ncol ? src[t * tileH + c] : mk<T>((T)0, (T)0);
						}
					}
				}
			}
		} else if (turn == 1) {
			if (STEP) {
				if (a.early) {
					asm volatile("cp.async.wait_all;" ::: "memory");
					__syncthreads();
				}
				// coupling and update of pfc-relax.c:1215-1244 for the entries ky = h and
				// Ny - h (h = 0: 0 and Ny / 2, whose k^2 differ) of column c
				const StepK<T>& K = a.k;
				for (int e = tid; e < nh << lC; e += nt) {
					const int c = CC > 1 ? rt_div(e, a.plan.mnh) : 0, h = e - c * nh;
					if (c >= ncol) continue;
					const int kx = kx0 + c, k2nd = h ? Ny - h : nh;
					cplx<T>* sp = a.spec + (long long)kx * Ny;
					cplx<T> N0[U], N1[U];
					T A[U], Bn[U], cu[npairs<T, U>()];
					auto stored = [&](int at) {
#pragma unroll
						for (int u = 0; u < U; u++) {
							A[u] = eK[u * nk + at];
							Bn[u] = eK[(U + u) * nk + at];
						}
#pragma unroll
						for (int p = 0; p < U * (U - 1) / 2; p++) cu[p] = eK[(2 * U + p) * nk + at];
					};
					if (a.early) {
						const cplx<T>* s = eN + c * Ny;
#pragma unroll
						for (int u = 0; u < U; u++) {
							N0[u] = s[u * CC * Ny + h];
							N1[u] = s[u * CC * Ny + k2nd];
						}
						stored(e);
					} else {
#pragma unroll
						for (int u = 0; u < U; u++) {
							N0[u] = __ldcs(sp + u * a.sstride + h);
							N1[u] = __ldcs(sp + u * a.sstride + k2nd);
						}
						entry_coef<T, U>(K, k2_step<T>(kx, h, Ny, K.dkx, K.dky), A, Bn, cu);
					}
					auto apply = [&](int ky, const cplx<T>(&N)[U]) {
						cplx<T> M[U];
						cplx<T>* s = sm + c * ld + rt_pad(ky, sh);
#pragma unroll
						for (int u = 0; u < U; u++) M[u] = cmul_rn(s[u * CC * ld], K.invN);
						if constexpr (U > 1) {
							int p = 0;
#pragma unroll
							for (int u = 0; u < U - 1; u++)
#pragma unroll
								for (int v = u + 1; v < U; v++, p++) {
									M[u] = cfma_rn(N[v], cu[p], M[u]);
									M[v] = cfma_rn(N[u], cu[p], M[v]);
								}
						}
#pragma unroll
						for (int u = 0; u < U; u++) {
							cplx<T> nn = cfma_rn(M[u], Bn[u], cmul_rn(N[u], A[u]));
							if (kx == 0 && ky == 0) nn = mk<T>((T)0, (T)0);
							__stcs(sp + u * a.sstride + ky, nn);
							s[u * CC * ld] = mk<T>(nn.y, nn.x);
						}
					};
					apply(h, N0);
					if (h == 0) {
						if (a.early) stored((nh << lC) + c);
						else entry_coef<T, U>(K, k2_step<T>(kx, nh, Ny, K.dkx, K.dky), A, Bn, cu);
					}
					apply(k2nd, N1);
				}
			} else {
				const T invN = (T)(1.0 / ((double)a.g.Nx * (double)Ny));
				for (int e = tid; e < Ny << lC; e += nt) {
					const int c = CC > 1 ? rt_div(e, a.plan.mn) : 0, ky = e - c * Ny;
					const int kx = kx0 + c;
					cplx<T>* s = sm + c * ld + rt_pad(ky, sh);
					const bool origin = kx == 0 && ky == 0;
					if (mode == YP_WEIGHT) {
						const cplx<T> nn = c < ncol && !origin ? weighted_entry<T>(a, kx, ky) : mk<T>((T)0, (T)0);
						s[0] = mk<T>(nn.y, nn.x);
					} else if (c < ncol) {
#pragma unroll
						for (int u = 0; u < U; u++) {
							cplx<T> nn = cscale(s[u * CC * ld], invN);
							if (origin) nn = mk<T>((T)0, (T)0);
							a.spec[u * a.sstride + (long long)kx * Ny + ky] = nn;
							s[u * CC * ld] = mk<T>(nn.y, nn.x);
						}
					}
				}
			}
			if (mode != YP_WEIGHT) {
				// kx = 0 and kx = Nx/2 (= H - 1): keep them exactly Hermitian
				const int kn = H - 1;
				const bool has0 = kx0 == 0, hasn = kn >= kx0 && kn < kx0 + ncol;
				if (has0 || hasn) {
					__syncthreads();
#pragma unroll
					for (int u = 0; u < U; u++) {
						if (has0) rt_hermitian_column<T>(sm + u * CC * ld, a.spec + u * a.sstride, Ny, sh, tid, nt);
						if (hasn)
							rt_hermitian_column<T>(sm + (u * CC + kn - kx0) * ld, a.spec + u * a.sstride + (long long)kn * Ny, Ny, sh,
							                       tid, nt);
					}
				}
			}
		}
		__syncthreads();
		rt_fft<T>(sm, a.plan, S, a.sb, a.tw, tid, nt);
		}
	if constexpr (WORK_IL<T, U>) {
		cplx<T>* dst = a.work + kx0 * U * R;
		if (R > 1) {
			for (int e = tid; e < nh * U << lC; e += nt) {
				const int r = 2 * e & (R - 1), i = e >> (lR - 1), u = i % U, c = i / U & (CC - 1), t = i / U >> lC;
				const cplx<T>* s = sm + (u * CC + c) * ld + rt_pad(t * R + r, sh);
				if (c < ncol) st2(dst + t * tileH + (c * U + u) * R + r, mk<T>(s[0].y, s[0].x), mk<T>(s[1].y, s[1].x));
			}
		} else {
			for (int e = tid; e < Ny * U << lC; e += nt) {
				const int u = e % U, c = e / U & (CC - 1), t = e / U >> lC;
				const cplx<T> v = sm[(u * CC + c) * ld + rt_pad(t, sh)];
				if (c < ncol) dst[t * tileH + c * U + u] = mk<T>(v.y, v.x);
			}
		}
	} else {
#pragma unroll
		for (int u = 0; u < U; u++) {
			cplx<T>* dst = a.work + u * a.wstride + (long long)kx0 * R;
			const cplx<T>* src = sm + u * CC * ld;
			if (R > 1) {
				for (int i = tid; i < nh << lC; i += nt) {
					const int e = 2 * i, r = e & (R - 1), c = (e >> lR) & (CC - 1), t = e >> (lR + lC);
					const cplx<T>* s = src + c * ld + rt_pad(t * R + r, sh);
					if (c < ncol) st2(dst + t * tileH + c * R + r, mk<T>(s[0].y, s[0].x), mk<T>(s[1].y, s[1].x));
				}
			} else {
				for (int e = tid; e < Ny << lC; e += nt) {
					const int c = e & (CC - 1), t = e >> lC;
					const cplx<T> v = src[c * ld + rt_pad(t, sh)];
					if (c < ncol) dst[t * tileH + c] = mk<T>(v.y, v.x);
				}
			}
		}
	}
}

// -------------------------------------------------------------- kernels --

// CTAs of MAXNT threads per SM: 64 registers in FP32 (no spills; 128 are 0.98 of
// the time at 512^2 but 1.45 at 2000^2 U=1), 128 in FP64
template <typename T> constexpr int RT_MINB = sizeof(T) == 4 ? 2 : 1;

template <typename T, int U, bool STEP> __global__ void __launch_bounds__(MAXNT, RT_MINB<T>) xrt_kernel(const XArgs<T> a, int mode) {
	rt_warm_twiddles<T>(a.tw, a.plan.ntw, threadIdx.x, blockDim.x);
	rt_xpass<T, U, STEP>(a, mode, blockIdx.x);
}

template <typename T, int U, bool STEP> __global__ void __launch_bounds__(MAXNT, RT_MINB<T>) yrt_kernel(const YArgs<T> a, int mode) {
	rt_warm_twiddles<T>(a.tw, a.plan.ntw, threadIdx.x, blockDim.x);
	rt_ypass<T, U, STEP>(a, mode, blockIdx.x);
}

template <typename T, int U, bool STEP> cudaError_t xrt_launch(int mode, const XArgs<T>& a, const LaunchCfg& c, cudaStream_t s) {
	auto k = xrt_kernel<T, U, STEP>;
	static unsigned long long mask = 0;
	smem_attr(k, mask);
	return pdl_launch(k, c.grid, c.block, c.smem, s, a, mode, c.plain);
}
template <typename T, int U, bool STEP> cudaError_t yrt_launch(int mode, const YArgs<T>& a, const LaunchCfg& c, cudaStream_t s) {
	auto k = yrt_kernel<T, U, STEP>;
	static unsigned long long mask = 0;
	smem_attr(k, mask);
	return pdl_launch(k, c.grid, c.block, c.smem, s, a, mode, c.plain);
}

// launchers of one precision and field count, instantiated in kernels_rt_<f32|f64>_<U>.cu
template <typename T, int U> cudaError_t rt_launch_x(int mode, const XArgs<T>& a, const LaunchCfg& c, cudaStream_t s) {
	return mode == XP_STEP ? xrt_launch<T, U, true>(mode, a, c, s) : xrt_launch<T, U, false>(mode, a, c, s);
}
template <typename T, int U> cudaError_t rt_launch_y(int mode, const YArgs<T>& a, const LaunchCfg& c, cudaStream_t s) {
	return mode == YP_STEP ? yrt_launch<T, U, true>(mode, a, c, s) : yrt_launch<T, U, false>(mode, a, c, s);
}

} // namespace pfcg
