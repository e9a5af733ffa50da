// Shared-memory FFT of a length known at run time: a plan of Stockham passes
// (fft_core.cuh) with every index constant prepared on the host.
//
// What bounded the kernels that use it before this form was instruction fetch
// and latency: with both directions and every radix unrolled in line a
// 1440-point transform took five passes (16, 2, 3, 3, 5), divided by run-time
// lengths and gathered its twiddles from an n-entry table. Here
//  - a plan has as few passes as radices up to 16 allow (1440 = 9 * 10 * 16),
//    composite radices being prime-factor DFTs in registers;
//  - only forward transforms exist: swap(x) = i conj(x) turns an inverse one
//    into a forward one (inverse(x) = swap(forward(swap(x)))), and the callers
//    fold the swap into their loads and stores, so one copy of the code serves
//    both directions;
//  - divisions are multiplications by reciprocals rounded up (exact for the
//    ranges used, see rt_magic), strides are precomputed, and the twiddles of a
//    pass are laid out so that consecutive lanes read consecutive entries.
#pragma once

#include "fft_core.cuh"

namespace pfcg {

constexpr int RT_MAXP = 12;  // passes of a plan (8192 = 2^13 needs 4)
constexpr int RT_MAXE = 16;  // elements a thread holds in a pass, and the largest radix

struct RtPass {
	int r;          // radix
	int ns;         // product of the radices before this pass
	int nr;         // n / r
	int two;        // first twiddle of the pass
	unsigned mnr;   // reciprocals of nr and ns (rt_magic)
	unsigned mns;
	int sin, sout;  // padded strides of a butterfly's inputs and outputs
	int sx;         // radix 16 in a first pass with period 8: the spare element between outputs 7 and 8
};

struct FftPlan {
	int n, npass;
	int sh;        // one spare element after every 2^sh (31: no padding)
	int ld;        // padded length of a sequence
	int ntw;       // twiddles in all
	unsigned mn;   // reciprocals of n and n / 2
	unsigned mnh;
	RtPass p[RT_MAXP];
};

// x / d = umulhi(x, rt_magic(d)) for d >= 2 and x * d < 2^32: with
// m = ceil(2^32 / d), m d - 2^32 < d, so x m / 2^32 exceeds x / d by less than
// x / 2^32 < 1 / d, which cannot reach the next integer.
__host__ __device__ __forceinline__ unsigned rt_magic(unsigned d) { return d < 2 ? 0u : (unsigned)(((1ull << 32) + d - 1) / d); }
__host__ __device__ __forceinline__ int rt_div(int x, unsigned m) {
#ifdef __CUDA_ARCH__
	return (int)__umulhi((unsigned)x, m);
#else
	return (int)(((unsigned long long)(unsigned)x * m) >> 32);
#endif
}

__host__ __device__ __forceinline__ int rt_pad(int i, int sh) { return i + (i >> sh); }

// Tabulated twiddle powers of a radix-r pass: w^1 .. w^(r-1), or in FP32 at
// radix 16 the six that ct_twiddle multiplies the others from (fewer loads than
// products there; FP64 keeps every power as tabulated).
__host__ __device__ constexpr int rt_twcnt(int r, bool fp64) { return r == 16 && !fp64 ? 6 : r - 1; }

// Position of butterfly j of a pass: twiddle index jm, first output d.
__host__ __device__ __forceinline__ void rt_place(int r, int ns, unsigned mns, int j, int& jm, int& d) {
	if (ns > 1) {
		const int b = rt_div(j, mns);
		jm = j - b * ns;
		d = j + b * ns * (r - 1);
	} else {
		jm = 0;
		d = j * r;
	}
}

template <int R, typename T>
__host__ __device__ __forceinline__ void rt_butterfly(cplx<T>* v, const cplx<T>* tw, int ns, bool twiddled) {
	if (twiddled) {
		if constexpr (R == 16 && sizeof(T) == 4) {
			cplx<T> b[6];
#pragma unroll
			for (int k = 0; k < 6; k++) b[k] = tw[k * ns];
			v[1] = cmul(v[1], b[0]);
			v[2] = cmul(v[2], b[1]);
			v[3] = cmul(v[3], b[2]);
#pragma unroll
			for (int h = 0; h < 3; h++) {
				v[4 * h + 4] = cmul(v[4 * h + 4], b[3 + h]);
#pragma unroll
				for (int k = 0; k < 3; k++) v[4 * h + 5 + k] = cmul(v[4 * h + 5 + k], cmul(b[3 + h], b[k]));
			}
		} else {
#pragma unroll
			for (int r = 1; r < R; r++) v[r] = cmul(v[r], tw[(r - 1) * ns]);
		}
	}
	dft<R, -1, T>(v);
}

// One pass over P sequences (at buf + p * ld), in place: inputs, twiddles and the
// DFT before the barrier, the stores after it, NB butterflies per thread.
// Threads without a butterfly repeat the last one and store nothing: with every
// value defined on every path none counts as carried over from the pass before
// (as conditionally loaded ones did, which held every radix's elements through
// the loop over the passes: 128 registers and 1.2 KB of spills a thread).
template <int R, int NB, typename T>
__device__ __forceinline__ void rt_pass_nb(cplx<T>* buf, const RtPass& q, int ld, int sh, int total,
                                           const cplx<T>* __restrict__ tw, int t, int nt) {
	const int nr = q.nr, ns = q.ns, sin = q.sin, sout = q.sout;
	cplx<T> v[NB][R];
	int dst[NB];
#pragma unroll
	for (int i = 0; i < NB; i++) {
		const int b = min(t + i * nt, total - 1);
		const int p = rt_div(b, q.mnr), j = b - p * nr;
		const cplx<T>* in = buf + p * ld + rt_pad(j, sh);
#pragma unroll
		for (int r = 0; r < R; r++) v[i][r] = in[r * sin];
		int jm, d;
		rt_place(R, ns, q.mns, j, jm, d);
		rt_butterfly<R, T>(v[i], tw + q.two + jm, ns, ns > 1);
		dst[i] = p * ld + rt_pad(d, sh);
	}
	__syncthreads();
#pragma unroll
	for (int i = 0; i < NB; i++)
		if (t + i * nt < total) {
			cplx<T>* out = buf + dst[i];
#pragma unroll
			for (int r = 0; r < R; r++) out[r * sout + (R == 16 && r >= 8 ? q.sx : 0)] = v[i][r];
		}
	__syncthreads();
}

template <int R, typename T>
__device__ __forceinline__ void rt_pass(cplx<T>* buf, const RtPass& q, int ld, int sh, int P,
                                        const cplx<T>* __restrict__ tw, int t, int nt) {
	const int total = P * q.nr;
	if (RT_MAXE / R == 1 || total <= nt) rt_pass_nb<R, 1, T>(buf, q, ld, sh, total, tw, t, nt);
	else rt_pass_nb<R, RT_MAXE / R, T>(buf, q, ld, sh, total, tw, t, nt);
}

// Forward transforms of S resident sequences, SB at a time (SB such that the
// passes fit the CTA's threads).
template <typename T>
__device__ __forceinline__ void rt_fft(cplx<T>* buf, const FftPlan& pl, int S, int SB, const cplx<T>* __restrict__ tw, int t,
                                       int nt) {
	const int ld = pl.ld, sh = pl.sh;
#pragma unroll 1
	for (int b0 = 0; b0 < S; b0 += SB) {
		const int P = S - b0 < SB ? S - b0 : SB;
		cplx<T>* b = buf + b0 * ld;
#pragma unroll 1
		for (int s = 0; s < pl.npass; s++) {
			const RtPass& q = pl.p[s];
#define PFCG_RT_CASE(R) \
	case R: rt_pass<R, T>(b, q, ld, sh, P, tw, t, nt); break;
			switch (q.r) {
				PFCG_RT_CASE(16)
				PFCG_RT_CASE(15)
				PFCG_RT_CASE(14)
				PFCG_RT_CASE(12)
				PFCG_RT_CASE(10)
				PFCG_RT_CASE(9)
				PFCG_RT_CASE(8)
				PFCG_RT_CASE(7)
				PFCG_RT_CASE(6)
				PFCG_RT_CASE(5)
				PFCG_RT_CASE(4)
				PFCG_RT_CASE(3)
				PFCG_RT_CASE(2)
			}
#undef PFCG_RT_CASE
		}
	}
}

// ------------------------------------------------------------ host planning --

// threads that one pass of radix r over P sequences needs
inline int rt_threads(int n, int r, int P) {
	const long long b = (long long)P * (n / r);
	const int nb = RT_MAXE / r;
	return (int)((b + nb - 1) / nb);
}

inline int rt_plan_threads(const FftPlan& pl, int P) {
	int nt = 32;
	for (int s = 0; s < pl.npass; s++) {
		const int k = rt_threads(pl.n, pl.p[s].r, P);
		nt = k > nt ? k : nt;
	}
	return (nt + 31) / 32 * 32;
}

// Fills the passes' constants for an order of radices. The padding period is
// 2^3 or 2^4 elements where every stride is a multiple of it (a stride then
// grows by stride >> sh whatever the start) and the first pass's outputs stay
// inside one period or, at radix 16, two; otherwise there is none, and an odd first radix keeps the
// stride-r stores of the first pass off each other's banks.
inline void rt_fill(FftPlan* pl, int n, const int* rad, int k, bool fp64) {
	pl->n = n;
	pl->npass = k;
	pl->mn = rt_magic(n);
	pl->mnh = rt_magic(n / 2);
	pl->sh = 31;
	for (int sh = fp64 ? 3 : 4; sh >= 3 && pl->sh == 31; sh--) {
		bool ok = true;
		for (int s = 0, ns = 1; s < k; ns *= rad[s++]) {
			ok = ok && (n / rad[s]) % (1 << sh) == 0;
			ok = ok && (s == 0 ? (1 << sh) % rad[0] == 0 || rad[0] == 16 : ns % (1 << sh) == 0);
		}
		if (ok) pl->sh = sh;
	}
	pl->ld = rt_pad(n, pl->sh) + 1;
	int two = 0;
	for (int s = 0, ns = 1; s < k; ns *= rad[s++]) {
		RtPass& q = pl->p[s];
		q.r = rad[s];
		q.ns = ns;
		q.nr = n / rad[s];
		q.mnr = rt_magic(q.nr);
		q.mns = rt_magic(ns);
		q.two = two;
		q.sin = rt_pad(q.nr, pl->sh);
		q.sout = rt_pad(ns, pl->sh);
		q.sx = s == 0 && rad[s] == 16 && pl->sh == 3 ? 1 : 0;
		if (s) two += rt_twcnt(rad[s], fp64) * ns;
	}
	pl->ntw = two;
}

// The order of radices with the lowest cost: fewest passes first, then the
// largest smallest radix (balanced passes need the fewest threads), then
// padding, then an odd first radix. Radices whose pass of one sequence needs
// more than max_threads threads are left out. Returns false where none is left.
inline bool rt_make_plan(int n, bool fp64, int max_threads, int max_radix, FftPlan* pl) {
	static const int all[13] = {16, 15, 14, 12, 10, 9, 8, 7, 6, 5, 4, 3, 2};
	int cur[RT_MAXP], best[RT_MAXP];
	long long best_cost = -1;
	struct Search {
		int n, max_threads, max_radix;
		bool fp64;
		int *cur, *best;
		long long* best_cost;
		void go(int rest, int k, int limit) {
			if (*best_cost >= 0 && k > *best_cost / 1000000) return;
			if (rest == 1) {
				// every order of this set of radices
				int ord[RT_MAXP];
				for (int i = 0; i < k; i++) ord[i] = cur[i];
				// ord is descending; walk the distinct permutations in lexicographic order from the ascending one
				for (int i = 0; i < k / 2; i++) { const int t = ord[i]; ord[i] = ord[k - 1 - i]; ord[k - 1 - i] = t; }
				for (;;) {
					FftPlan t;
					rt_fill(&t, n, ord, k, fp64);
					int mn = 99, mx = 0;
					for (int i = 0; i < k; i++) {
						const int need = rt_threads(n, ord[i], 1);
						mx = need > mx ? need : mx;
						mn = ord[i] < mn ? ord[i] : mn;
					}
					// conflicts of the first pass's stores without padding
					int g = 1;
					if (t.sh == 31)
						while (g < 16 && ord[0] % (2 * g) == 0) g *= 2;
					const long long c = k * 1000000ll + (long long)(16 - mn) * 10000 + (t.sh == 31 ? 2000 : 0) + g * 100 + (16 - ord[k - 1]);
					if (*best_cost < 0 || c < *best_cost) {
						*best_cost = c;
						for (int i = 0; i < k; i++) best[i] = ord[i];
						best[k] = 0;
					}
					int i = k - 2;
					while (i >= 0 && ord[i] >= ord[i + 1]) i--;
					if (i < 0) break;
					int j = k - 1;
					while (ord[j] <= ord[i]) j--;
					{ const int t2 = ord[i]; ord[i] = ord[j]; ord[j] = t2; }
					for (int a = i + 1, b = k - 1; a < b; a++, b--) { const int t2 = ord[a]; ord[a] = ord[b]; ord[b] = t2; }
				}
				return;
			}
			if (k >= RT_MAXP - 1) return;
			for (int q = 0; q < 13; q++) {
				const int r = all[q];
				if (r > limit || r > max_radix || rest % r || r == n || rt_threads(n, r, 1) > max_threads) continue;
				cur[k] = r;
				go(rest / r, k + 1, r);
			}
		}
	} s{n, max_threads, max_radix, fp64, cur, best, &best_cost};
	s.go(n, 0, 16);
	if (best_cost < 0) return false;
	rt_fill(pl, n, best, (int)(best_cost / 1000000), fp64);
	return true;
}

// entry i of the plan's twiddle table as (numerator, denominator): exp(-2 pi i num / den)
__host__ __device__ inline void rt_twiddle_of(const FftPlan& pl, bool fp64, int i, int* num, int* den) {
	int s = pl.npass - 1;
	while (s > 1 && i < pl.p[s].two) s--;
	const RtPass& q = pl.p[s];
	const int e = i - q.two, k = e / q.ns, jm = e - k * q.ns;
	int pw = k + 1;
	if (q.r == 16 && !fp64) pw = k < 4 ? k + 1 : 4 * (k - 2); // 1, 2, 3, 4, 8, 12
	*num = pw * jm;
	*den = q.ns * q.r;
}

} // namespace pfcg
