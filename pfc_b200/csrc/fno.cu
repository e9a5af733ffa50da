// Fourier neural operator warm start: forward, backward, Adam and tiled apply.
//
// Network (fixed shape; two fields on a T x T periodic tile):
//   v0 = P x + p                            lift, 2 -> C channels per pixel
//   z_l = W_l v_l + b_l + K_l v_l,  v_{l+1} = gelu(z_l)  (l < L-1), v_L = z_{L-1}
//   y = x + Q v_L + q                       projection C -> 2, added to the input
// K_l v = irfft2 of R_l (complex C x C per retained mode) times rfft2(v) on the
// retained modes kx in [0, MX), ky in {0..MY/2-1} u {T-MY/2..T-1}; all other
// modes are dropped. The truncated transforms are direct sums against
// twiddle matrices; the adjoint of each linear step is the transform of the
// other direction, which is how the backward pass is built. A layer is two kinds
// of kernel: one pass over the activations (layer_fwd, or layer_grad and
// layer_bwd on the way back), which does everything per row (channel product,
// inverse x transform of the mixed modes, GELU, forward x transform of the result,
// at the ends the lift and the projection), and the small kernels between two
// passes, which work on the rows' eight retained modes (dft_y_fwd, mix, dft_y_inv).
// Activations and sums are FP32; the kernels read a BF16 copy of the FP32
// master weights, which Adam updates.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cmath>
#include <string>
#include <vector>

#include "../../include/pfc_b200.h"
#include "fno.cuh"
#include "fno_gelu.cuh"

namespace {

using pfcg::gelu;
using pfcg::gelu_d;

constexpr int C = PFCG_FNO_CHANNELS;
constexpr int L = PFCG_FNO_LAYERS;
constexpr int MX = PFCG_FNO_MODES_X;
constexpr int MY = PFCG_FNO_MODES_Y;
constexpr int NK = MX * MY; // retained modes per channel pair

// parameter layout, in floats: P [C][2], p [C], per layer {W [C][C], b [C],
// Rr [C][C][NK], Ri [C][C][NK]} with R indexed [in][out][ky-row][kx], Q [2][C], q [2]
constexpr size_t OFF_P = 0;
constexpr size_t OFF_PB = OFF_P + C * 2;
constexpr size_t OFF_L0 = OFF_PB + C;
constexpr size_t LAYER = C * C + C + 2 * (size_t)C * C * NK;
constexpr size_t OFF_Q = OFF_L0 + L * LAYER;
constexpr size_t OFF_QB = OFF_Q + 2 * C;
constexpr size_t NPARAM = OFF_QB + 2;
static_assert(NPARAM == PFCG_FNO_PARAMS, "parameter count");

__host__ __device__ constexpr size_t off_W(int l) { return OFF_L0 + l * LAYER; }
__host__ __device__ constexpr size_t off_b(int l) { return off_W(l) + C * C; }
__host__ __device__ constexpr size_t off_Rr(int l) { return off_b(l) + C; }
__host__ __device__ constexpr size_t off_Ri(int l) { return off_Rr(l) + (size_t)C * C * NK; }

constexpr int MAXT = 512; // largest tile (twiddle table in shared memory)

__device__ __forceinline__ float wld(const __nv_bfloat16* w, size_t i) { return __bfloat162float(w[i]); }

// wave number of retained row k along y
__device__ __forceinline__ int ky_of(int k, int T) { return k < MY / 2 ? k : T - MY + k; }

template <typename A> __device__ __forceinline__ A warp_sum(A a) {
	for (int o = 16; o; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
	return a;
}

// ------------------------------------------------------------- kernels ---

// tw[j] = (cos, sin)(2 pi j / T), from FP64
__global__ void twiddle_kernel(float2* tw, int T) {
	for (int j = threadIdx.x + blockIdx.x * blockDim.x; j < T; j += blockDim.x * gridDim.x) {
		double s, c;
		sincospi(2.0 * j / (double)T, &s, &c);
		tw[j] = make_float2((float)c, (float)s);
	}
}

// --------------------------------------------------- tensor-core products --
// The per-pixel channel contractions (z = W v, dv = W^T dz, dW = dz v^T) and the
// x transforms (whose other operand is a fixed matrix of twiddles) are GEMMs on
// the tensor cores, mma.sync m16n8k16 with BF16 operands and FP32 accumulation.
// An FP32 operand is split into a BF16 high part and a BF16 remainder (x = hi +
// lo to about 2^-16 relative) and the products that matter are summed: with the
// BF16 weights, which are exact, W hi + W lo; with two FP32 operands, hi hi +
// hi lo + lo hi. Fragment layouts are those of the PTX ISA for m16n8k16: g =
// lane / 4, t = lane % 4; A (16 x 16, row major) holds rows g, g + 8 and columns
// 2t, 2t + 1, 2t + 8, 2t + 9; B (16 x 8) holds rows 2t, 2t + 1, 2t + 8, 2t + 9
// of column g; the accumulator holds rows g, g + 8 and columns 2t, 2t + 1.

__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
	asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
	             "{%0,%1,%2,%3};\n"
	             : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
	             : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// two FP32 values (the lower index first) as BF16 pairs: high parts and remainders
__device__ __forceinline__ void split2(float x0, float x1, uint32_t& hi, uint32_t& lo) {
	const __nv_bfloat162 h = __floats2bfloat162_rn(x0, x1);
	const float2 hf = __bfloat1622float2(h);
	const __nv_bfloat162 l = __floats2bfloat162_rn(x0 - hf.x, x1 - hf.y);
	hi = *reinterpret_cast<const uint32_t*>(&h);
	lo = *reinterpret_cast<const uint32_t*>(&l);
}

// two BF16 weights as one B-fragment register (the first in the low half)
__device__ __forceinline__ uint32_t pack_bf16(const __nv_bfloat16* w, size_t i0, size_t i1) {
	const unsigned short a = *reinterpret_cast<const unsigned short*>(w + i0);
	const unsigned short b = *reinterpret_cast<const unsigned short*>(w + i1);
	return (uint32_t)a | ((uint32_t)b << 16);
}

// A warp works on 32 pixels of a row at a time, as four n-tiles of eight columns
// (or, where they are summed over, two k-steps of sixteen). Column c of n-tile j is
// pixel 4 (c / 2) + 16 (c % 2) + j: lane g then loads its column of all four tiles
// as one float4, the eight g of a channel 128 contiguous bytes, and of a result
// lane t holds pixels 4t .. 4t + 3 and 16 + 4t .. 16 + 4t + 3, two float4. The same
// order makes an accumulator the A operand of the next product (k-step ks holds
// n-tiles 2 ks and 2 ks + 1), so a result's x transform needs no exchange.
constexpr int PX = 32;
__host__ __device__ __forceinline__ int px_of(int c, int j) { return 4 * (c >> 1) + 16 * (c & 1) + j; }

// The twiddle matrices of the x transforms as B fragments, high parts and remainders:
//   forward: E[x][2m + q] = cos / -sin(2 pi m x / T), fe: [T/32][2 k-steps][2 n-tiles][32 lanes]
//   inverse: F[2m + q][x] = cos / -sin(2 pi m x / T), ff: [T/32][4 n-tiles][32 lanes]
__global__ void dft_frag_kernel(const float2* __restrict__ tw, int T, uint4* __restrict__ fe, uint4* __restrict__ ff) {
	const int n = T / PX * 4 * 32;
	for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < 2 * n; e += gridDim.x * blockDim.x) {
		const int f = e % n, lane = f & 31, g = lane >> 2, t = lane & 3, x0 = (f >> 7) * PX;
		float v[4];
		if (e < n) {
			const int nt = (f >> 5) & 1, ks = (f >> 6) & 1;
			const int col = 8 * nt + g, m = col >> 1, q = col & 1;
			const int xs[4] = {px_of(2 * t, 2 * ks), px_of(2 * t + 1, 2 * ks), px_of(2 * t, 2 * ks + 1), px_of(2 * t + 1, 2 * ks + 1)};
#pragma unroll
			for (int k = 0; k < 4; k++) {
				const float2 w = tw[(m * (x0 + xs[k])) & (T - 1)];
				v[k] = q ? -w.y : w.x;
			}
		} else {
			const int x = x0 + px_of(g, (f >> 5) & 3);
			const float2 w0 = tw[(t * x) & (T - 1)], w4 = tw[((t + 4) * x) & (T - 1)];
			v[0] = w0.x;
			v[1] = -w0.y;
			v[2] = w4.x;
			v[3] = -w4.y;
		}
		uint32_t h0, l0, h1, l1;
		split2(v[0], v[1], h0, l0);
		split2(v[2], v[3], h1, l1);
		(e < n ? fe : ff)[f] = make_uint4(h0, h1, l0, l1);
	}
}

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, float a, float b, float c, float d) {
	*reinterpret_cast<float4*>(p) = make_float4(a, b, c, d);
}
// the caller's tensors need not be 16-byte aligned
__device__ __forceinline__ float4 ld4u(const float* p, bool vec) {
	return vec ? ld4(p) : make_float4(p[0], p[1], p[2], p[3]);
}
__device__ __forceinline__ float at(const float4& v, int j) { return j == 0 ? v.x : j == 1 ? v.y : j == 2 ? v.z : v.w; }

// an A fragment kept in shared memory (volatile: read at each use, not held)
__device__ __forceinline__ void ld_frag(uint32_t (&a)[4], const uint4* p) {
	asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
	             : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3])
	             : "r"((unsigned)__cvta_generic_to_shared(p)));
}

// a += c, b += c, rounded to nearest. What a tensor core's sum starts from is not: each of
// its products added to a bias of 1 cost up to 2^-23, so the bias, and in the backward
// pass the channel product, is added to the transform's own sum (4096^2 applied 20.9 ms,
// 21.4 with scalar and 20.5 with paired additions, 20.1 since; a training iteration 5.7 and 5.8, 4.9 since).
__device__ __forceinline__ void add2(float& a, float& b, float c) {
	asm("{\n\t.reg .b64 x, y;\n\tmov.b64 x, {%0, %1};\n\tmov.b64 y, {%2, %2};\n\tadd.rn.f32x2 x, x, y;\n\tmov.b64 {%0, %1}, x;\n\t}"
	    : "+f"(a), "+f"(b)
	    : "f"(c));
}

// d += A B with A = (ah, al) and B = the fragment f split the same way
__device__ __forceinline__ void mma_split(float (&d)[4], const uint32_t (&ah)[4], const uint32_t (&al)[4], const uint4& f) {
	const uint32_t bh[2] = {f.x, f.y}, bl[2] = {f.z, f.w};
	mma_bf16(d, ah, bh);
	mma_bf16(d, ah, bl);
	mma_bf16(d, al, bh);
}

// A fragments of the modes of rows (b, o, y), o = 16 mt + g and + 8: (Re, Im) of
// modes t and t + 4, times their weights
__device__ __forceinline__ void load_modes(const float2* __restrict__ z, long long b, int y, int T, int mt, int g, int t,
                                           float s0, float s4, uint32_t (&ah)[4], uint32_t (&al)[4]) {
#pragma unroll
	for (int h = 0; h < 2; h++) {
		const float2* p = z + ((b * C + 16 * mt + g + 8 * h) * T + y) * MX;
		const float2 z0 = p[t], z4 = p[t + 4];
		split2(s0 * z0.x, s0 * z0.y, ah[h], al[h]);
		split2(s4 * z4.x, s4 * z4.y, ah[2 + h], al[2 + h]);
	}
}

// acc[nt] += the x transform of 32 pixels of 16 channels held as accumulators d[j]
__device__ __forceinline__ void add_dft(float (&acc)[2][4], const float (&d)[4][4], const uint4* __restrict__ fe, int tile,
                                        int lane) {
#pragma unroll
	for (int ks = 0; ks < 2; ks++) {
		uint32_t ah[4], al[4];
#pragma unroll
		for (int h = 0; h < 2; h++) {
			split2(d[2 * ks + h][0], d[2 * ks + h][1], ah[2 * h], al[2 * h]);
			split2(d[2 * ks + h][2], d[2 * ks + h][3], ah[2 * h + 1], al[2 * h + 1]);
		}
#pragma unroll
		for (int nt = 0; nt < 2; nt++) mma_split(acc[nt], ah, al, __ldg(fe + ((tile * 2 + ks) * 2 + nt) * 32 + lane));
	}
}

// the rows' modes from those sums: columns 2t, 2t + 1 of n-tile nt are (Re, Im) of mode 4 nt + t
__device__ __forceinline__ void store_modes(float2* __restrict__ out, const float (&acc)[2][4], long long b, int y, int T,
                                            int mt, int g, int t, const float* __restrict__ scale) {
#pragma unroll
	for (int nt = 0; nt < 2; nt++) {
		const int m = 4 * nt + t;
		const float sc = scale ? scale[m] : 1.f;
		float2* p = out + ((b * C + 16 * mt + g) * T + y) * MX + m;
		p[0] = make_float2(acc[nt][0] * sc, acc[nt][1] * sc);
		p[8LL * T * MX] = make_float2(acc[nt][2] * sc, acc[nt][3] * sc);
	}
}

// x transform of the lifted input: v0 = P x + p is linear, so its modes are P times
// those of x's two fields, plus p T at m = 0. These sums are FP32: every channel takes
// their error times its two weights, so that one of BF16 splits would add up over the
// channels where those of 32 transforms average out (network applied to 2048^2: 8.3e-6
// from 64 bits with split products here, 8.0e-6 with one transform per channel and with
// these; 4096^2 takes 20.9 ms either way).
// One warp per row; pixel 32 i + lane, w = exp(-2 pi i / T):
//   X[m] = sum_lane w^(m lane) sum_i x[32 i + lane] w^(32 m i),
// the inner twiddles the same for every lane.
__global__ void __launch_bounds__(128) lift_dft(const float* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                                                float* __restrict__ out, const float2* __restrict__ tw, long long nrows, int T) {
	__shared__ float Ps[3 * C];
	__shared__ float2 ti[MAXT / 32][MX];
	for (int i = threadIdx.x; i < 3 * C; i += blockDim.x) Ps[i] = wld(w, OFF_P + i);
	for (int i = threadIdx.x; i < T / 32 * MX; i += blockDim.x) ti[i / MX][i % MX] = tw[(32 * (i / MX) * (i % MX)) & (T - 1)];
	__syncthreads();
	const int lane = threadIdx.x & 31;
	float2 tl[MX];
#pragma unroll
	for (int m = 0; m < MX; m++) tl[m] = tw[(m * lane) & (T - 1)];
	const long long npix = (long long)T * T, nw = ((long long)gridDim.x * blockDim.x) >> 5;
	for (long long r = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < nrows; r += nw) {
		const long long b = r / T;
		const int y = (int)(r - b * T);
		const float* p = x + b * 2 * npix + (long long)y * T + lane;
		float a[2 * 2 * MX]; // [field][mode][Re, Im]
#pragma unroll
		for (int k = 0; k < 4 * MX; k++) a[k] = 0.f;
#pragma unroll 4
		for (int i = 0; i < T / 32; i++) {
			const float v[2] = {p[32 * i], p[npix + 32 * i]};
#pragma unroll
			for (int m = 0; m < MX; m++) {
				const float2 c = ti[i][m];
#pragma unroll
				for (int f = 0; f < 2; f++) {
					a[2 * (MX * f + m)] = fmaf(v[f], c.x, a[2 * (MX * f + m)]);
					a[2 * (MX * f + m) + 1] = fmaf(v[f], -c.y, a[2 * (MX * f + m) + 1]);
				}
			}
		}
#pragma unroll
		for (int k = 0; k < 2 * MX; k++) {
			const float2 c = tl[k % MX];
			const float re = a[2 * k], im = a[2 * k + 1];
			a[2 * k] = re * c.x + im * c.y;
			a[2 * k + 1] = im * c.x - re * c.y;
		}
		// over the lanes, halving what a lane keeps: it ends with element `lane`
#pragma unroll
		for (int o = 16; o; o >>= 1)
#pragma unroll
			for (int k = 0; k < o; k++) {
				const bool up = lane & o;
				const float keep = up ? a[o + k] : a[k], send = up ? a[k] : a[o + k];
				a[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
			}
		const float other = __shfl_xor_sync(0xffffffffu, a[0], 16);
		const int e = lane & 15, h = lane >> 4; // (Re, Im) of mode e / 2; this half's channels
		const float x0 = h ? other : a[0], x1 = h ? a[0] : other;
		float* o = out + ((b * C + h) * T + y) * (2 * MX) + e;
#pragma unroll 4
		for (int c = h; c < C; c += 2, o += 2LL * T * (2 * MX))
			*o = Ps[2 * c] * x0 + Ps[2 * c + 1] * x1 + (e == 0 ? Ps[2 * C + c] * (float)T : 0.f);
	}
}
static_assert(4 * MX == 32, "an element of the sums per lane");

// Two-field pixel values of a lane's column for all four n-tiles (channel values of
// the lift's output), v0[c][px] = P[c][0] x0 + P[c][1] x1 + p[c]
struct LiftRow {
	float p0, p1, pc;
	__device__ __forceinline__ void load(const __nv_bfloat16* w, int c) {
		p0 = wld(w, OFF_P + 2 * c);
		p1 = wld(w, OFF_P + 2 * c + 1);
		pc = wld(w, OFF_PB + c);
	}
	__device__ __forceinline__ float4 of(const float4& a, const float4& b) const {
		return make_float4(p0 * a.x + p1 * b.x + pc, p0 * a.y + p1 * b.y + pc, p0 * a.z + p1 * b.z + pc, p0 * a.w + p1 * b.w + pc);
	}
};

// One layer forward, a warp per row (b, y): z = W v + b + K v with K v the inverse x
// transform of the row's mixed modes Bq, v' = gelu(z). FIRST: v is the lift of x.
// Every layer but the last leaves the x transform of v' in A; the last one projects:
// out = x + Q z + q and, with a target, the loss, dy = 2 (out - target) / n and the
// gradients of Q and q. v is read and v' (in training also z) written once, where
// separate kernels for the transforms and the product moved them seven times: 16
// tiles of 512^2 take 302 us a layer (1.07 GB, 0.16 ms at the memory's rate; 848 us
// before). What is left is latency at 16 warps per SM, so registers are kept at 128
// (168 and 12 warps: 406 us) with the weights' fragments in shared memory.
template <bool FIRST, bool LAST, bool TRAIN>
__global__ void __launch_bounds__(128, LAST ? 3 : 4)
    layer_fwd(const float* __restrict__ x, int xvec, const float* v, const float2* __restrict__ Bq,
              const __nv_bfloat16* __restrict__ w, int l, const uint4* __restrict__ fe, const uint4* __restrict__ ff,
              const float* __restrict__ sx, float* z, float* vout, float2* __restrict__ A, float* __restrict__ out,
              const float* __restrict__ target, float* __restrict__ dy, double* __restrict__ loss, float* __restrict__ gr,
              long long nrows, int T, int B) {
	const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
	const long long npix = (long long)T * T;
	__shared__ uint4 sw[4][32]; // the weights' A fragments (in registers they cost a block per SM)
	uint32_t aw[2][2][4];
	float bias[2][2], Qr[2][2][2];
	LiftRow lift[2][4];
#pragma unroll
	for (int mt = 0; mt < 2; mt++) {
#pragma unroll
		for (int h = 0; h < 2; h++) {
			const int o = 16 * mt + g + 8 * h;
			bias[mt][h] = wld(w, off_b(l) + o);
#pragma unroll
			for (int ks = 0; ks < 2; ks++) {
				const size_t at_ = off_W(l) + (size_t)o * C + 16 * ks + 2 * t;
				aw[mt][ks][h] = pack_bf16(w, at_, at_ + 1);
				aw[mt][ks][2 + h] = pack_bf16(w, at_ + 8, at_ + 9);
			}
			if (LAST) {
				Qr[0][mt][h] = wld(w, OFF_Q + o);
				Qr[1][mt][h] = wld(w, OFF_Q + C + o);
			}
		}
	}
	if (FIRST) {
#pragma unroll
		for (int ks = 0; ks < 2; ks++)
#pragma unroll
			for (int k = 0; k < 4; k++) lift[ks][k].load(w, 16 * ks + 2 * t + (k & 1) + 8 * (k >> 1));
	}
	if (threadIdx.x < 32)
#pragma unroll
		for (int k = 0; k < 4; k++) sw[k][lane] = make_uint4(aw[k >> 1][k & 1][0], aw[k >> 1][k & 1][1], aw[k >> 1][k & 1][2], aw[k >> 1][k & 1][3]);
	__syncthreads();
	const float s0 = sx[t], s4 = sx[t + 4];
	const float qb[2] = {LAST ? wld(w, OFF_QB) : 0.f, LAST ? wld(w, OFF_QB + 1) : 0.f};
	float gq[2][2][2], gqb = 0.f;
	double lacc = 0.0;
#pragma unroll
	for (int j = 0; j < 2; j++)
#pragma unroll
		for (int mt = 0; mt < 2; mt++)
#pragma unroll
			for (int h = 0; h < 2; h++) gq[j][mt][h] = 0.f;
	const float inv = 2.f / (float)(2 * (long long)B * npix);

	const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
	for (long long r = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < nrows; r += nw) {
		const long long b = r / T;
		const int y = (int)(r - b * T);
		const long long base = b * C * npix + (long long)y * T, base2 = b * 2 * npix + (long long)y * T;
		uint32_t mh[2][4], ml[2][4];
		float acc[2][2][4];
#pragma unroll
		for (int mt = 0; mt < 2; mt++) {
			load_modes(Bq, b, y, T, mt, g, t, s0, s4, mh[mt], ml[mt]);
#pragma unroll
			for (int nt = 0; nt < 2; nt++)
#pragma unroll
				for (int k = 0; k < 4; k++) acc[mt][nt][k] = 0.f;
		}
		for (int tile = 0; tile < T / PX; tile++) {
			const int pl = tile * PX + px_of(g, 0); // the lane's four columns' pixels
			const int ps = tile * PX + 4 * t;       // the lane's result pixels (and + 16)
			float4 vv[2][4];
			if (FIRST) {
				const float4 x0 = ld4u(x + base2 + pl, xvec), x1 = ld4u(x + base2 + npix + pl, xvec);
#pragma unroll
				for (int ks = 0; ks < 2; ks++)
#pragma unroll
					for (int k = 0; k < 4; k++) vv[ks][k] = lift[ks][k].of(x0, x1);
			} else {
#pragma unroll
				for (int ks = 0; ks < 2; ks++)
#pragma unroll
					for (int k = 0; k < 4; k++) vv[ks][k] = ld4(v + base + (16 * ks + 2 * t + (k & 1) + 8 * (k >> 1)) * npix + pl);
			}
			float d[2][4][4];
#pragma unroll
			for (int j = 0; j < 4; j++) {
				const uint4 f = __ldg(ff + (tile * 4 + j) * 32 + lane);
#pragma unroll
				for (int mt = 0; mt < 2; mt++) {
#pragma unroll
					for (int k = 0; k < 4; k++) d[mt][j][k] = 0.f;
					mma_split(d[mt][j], mh[mt], ml[mt], f);
				}
#pragma unroll
				for (int ks = 0; ks < 2; ks++) {
					uint32_t bh[2], bl[2];
					split2(at(vv[ks][0], j), at(vv[ks][1], j), bh[0], bl[0]);
					split2(at(vv[ks][2], j), at(vv[ks][3], j), bh[1], bl[1]);
#pragma unroll
					for (int mt = 0; mt < 2; mt++) {
						uint32_t aq[4];
						ld_frag(aq, &sw[2 * mt + ks][lane]);
						mma_bf16(d[mt][j], aq, bh);
						mma_bf16(d[mt][j], aq, bl);
					}
				}
			}
			if constexpr (!LAST) {
#pragma unroll
				for (int mt = 0; mt < 2; mt++) {
#pragma unroll
					for (int h = 0; h < 2; h++) {
						const long long o = base + (16 * mt + g + 8 * h) * npix + ps;
#pragma unroll
						for (int j = 0; j < 4; j++) add2(d[mt][j][2 * h], d[mt][j][2 * h + 1], bias[mt][h]);
						if (TRAIN) {
							st4(z + o, d[mt][0][2 * h], d[mt][1][2 * h], d[mt][2][2 * h], d[mt][3][2 * h]);
							st4(z + o + 16, d[mt][0][2 * h + 1], d[mt][1][2 * h + 1], d[mt][2][2 * h + 1], d[mt][3][2 * h + 1]);
						}
#pragma unroll
						for (int j = 0; j < 4; j++) {
							d[mt][j][2 * h] = gelu(d[mt][j][2 * h]);
							d[mt][j][2 * h + 1] = gelu(d[mt][j][2 * h + 1]);
						}
						st4(vout + o, d[mt][0][2 * h], d[mt][1][2 * h], d[mt][2][2 * h], d[mt][3][2 * h]);
						st4(vout + o + 16, d[mt][0][2 * h + 1], d[mt][1][2 * h + 1], d[mt][2][2 * h + 1], d[mt][3][2 * h + 1]);
					}
					add_dft(acc[mt], d[mt], fe, tile, lane);
				}
			} else {
				// Q z: the lane's rows, then over the eight g, halving what a lane keeps: it
				// ends with field (lane >> 4), pixels ps + 16 (bit 3) + 2 (bit 2) + {0, 1}
#pragma unroll
				for (int mt = 0; mt < 2; mt++)
#pragma unroll
					for (int j = 0; j < 4; j++) {
						add2(d[mt][j][0], d[mt][j][1], bias[mt][0]);
						add2(d[mt][j][2], d[mt][j][3], bias[mt][1]);
					}
				float s[2][2][4];
#pragma unroll
				for (int f = 0; f < 2; f++)
#pragma unroll
					for (int c = 0; c < 2; c++)
#pragma unroll
						for (int j = 0; j < 4; j++)
							s[f][c][j] = (Qr[f][0][0] * d[0][j][c] + Qr[f][0][1] * d[0][j][2 + c]) +
							             (Qr[f][1][0] * d[1][j][c] + Qr[f][1][1] * d[1][j][2 + c]);
				const bool b4 = lane & 16, b3 = lane & 8, b2 = lane & 4;
				float u[2][4], q4[4], q2[2];
#pragma unroll
				for (int c = 0; c < 2; c++)
#pragma unroll
					for (int j = 0; j < 4; j++) {
						const float keep = b4 ? s[1][c][j] : s[0][c][j], send = b4 ? s[0][c][j] : s[1][c][j];
						u[c][j] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
					}
#pragma unroll
				for (int j = 0; j < 4; j++) {
					const float keep = b3 ? u[1][j] : u[0][j], send = b3 ? u[0][j] : u[1][j];
					q4[j] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
				}
#pragma unroll
				for (int j = 0; j < 2; j++) {
					const float keep = b2 ? q4[2 + j] : q4[j], send = b2 ? q4[j] : q4[2 + j];
					q2[j] = keep + __shfl_xor_sync(0xffffffffu, send, 4);
				}
				const long long i = base2 + (b4 ? npix : 0) + ps + (b3 ? 16 : 0) + (b2 ? 2 : 0);
				float e[2];
#pragma unroll
				for (int j = 0; j < 2; j++) {
					const float yv = x[i + j] + (q2[j] + (b4 ? qb[1] : qb[0]));
					out[i + j] = yv;
					if (TRAIN) {
						const float er = yv - target[i + j];
						lacc += (double)er * er;
						e[j] = inv * er;
						dy[i + j] = e[j];
						gqb += e[j];
					}
				}
				if constexpr (TRAIN) {
					// every lane's sixteen dy values back, doubling what a lane has
					float d4[4], d8[2][4], dd[2][2][4];
#pragma unroll
					for (int j = 0; j < 2; j++) {
						const float o = __shfl_xor_sync(0xffffffffu, e[j], 4);
						d4[j] = b2 ? o : e[j];
						d4[2 + j] = b2 ? e[j] : o;
					}
#pragma unroll
					for (int j = 0; j < 4; j++) {
						const float o = __shfl_xor_sync(0xffffffffu, d4[j], 8);
						d8[0][j] = b3 ? o : d4[j];
						d8[1][j] = b3 ? d4[j] : o;
					}
#pragma unroll
					for (int c = 0; c < 2; c++)
#pragma unroll
						for (int j = 0; j < 4; j++) {
							const float o = __shfl_xor_sync(0xffffffffu, d8[c][j], 16);
							dd[0][c][j] = b4 ? o : d8[c][j];
							dd[1][c][j] = b4 ? d8[c][j] : o;
						}
#pragma unroll
					for (int f = 0; f < 2; f++)
#pragma unroll
						for (int mt = 0; mt < 2; mt++)
#pragma unroll
							for (int h = 0; h < 2; h++)
#pragma unroll
								for (int c = 0; c < 2; c++)
#pragma unroll
									for (int j = 0; j < 4; j++) gq[f][mt][h] += d[mt][j][2 * h + c] * dd[f][c][j];
				}
			}
		}
		if constexpr (!LAST) {
#pragma unroll
			for (int mt = 0; mt < 2; mt++) store_modes(A, acc[mt], b, y, T, mt, g, t, nullptr);
		}
	}
	if constexpr (LAST && TRAIN) {
		__shared__ float sq[2 * C + 2];
		__shared__ double sl[4];
		for (int i = threadIdx.x; i < 2 * C + 2; i += blockDim.x) sq[i] = 0.f;
		__syncthreads();
#pragma unroll
		for (int f = 0; f < 2; f++)
#pragma unroll
			for (int mt = 0; mt < 2; mt++)
#pragma unroll
				for (int h = 0; h < 2; h++) {
					float a = gq[f][mt][h];
					a += __shfl_xor_sync(0xffffffffu, a, 1);
					a += __shfl_xor_sync(0xffffffffu, a, 2);
					if (t == 0) atomicAdd(&sq[f * C + 16 * mt + g + 8 * h], a);
				}
#pragma unroll
		for (int o = 8; o; o >>= 1) gqb += __shfl_xor_sync(0xffffffffu, gqb, o);
		if ((lane & 15) == 0) atomicAdd(&sq[2 * C + (lane >> 4)], gqb);
		lacc = warp_sum(lacc);
		if (lane == 0) sl[threadIdx.x >> 5] = lacc;
		__syncthreads();
		for (int i = threadIdx.x; i < 2 * C + 2; i += blockDim.x) atomicAdd(gr + OFF_Q + i, sq[i]);
		if (threadIdx.x == 0) atomicAdd(loss, (sl[0] + sl[1] + sl[2] + sl[3]) / (double)(2 * (long long)B * npix));
	}
}
static_assert(OFF_QB == OFF_Q + 2 * C, "q follows Q");

// First half of a layer backward, a warp per row: dz = dout gelu'(z) (the last layer:
// dz = Q^T dy, not stored), written over dout; the x transform of dz, which starts
// the spectral branch's adjoint; dW += dz v^T and db += dz summed over pixels.
template <bool FIRST, bool LAST>
__global__ void __launch_bounds__(128, 4)
    layer_grad(const float* __restrict__ x, int xvec, const float* __restrict__ v, const float* __restrict__ z, float* dz,
               const float* __restrict__ dy, const __nv_bfloat16* __restrict__ w, const uint4* __restrict__ fe,
               const float* __restrict__ sx, float2* __restrict__ A, float* __restrict__ gW, float* __restrict__ gb,
               long long nrows, int T) {
	__shared__ float sW[C * C];
	__shared__ float sb[C];
	// A warp's weight sums, [accumulator][lane]. They leave the tensor core after
	// every 32 pixels: its additions are not rounded to nearest, and sums of whole
	// rows there left the gradient 1.7e-6 from 64 bits at any batch (512^2; now
	// 5e-7 at one tile, 8e-7 at 16). A second set of registers spilled (6.6 ms an
	// iteration, 5.2 to 5.6 this way, 4.6 with the long sums; 4.55 since GELU's derivative needs no clamp).
	__shared__ float sacc[4][32][32];
	float* const mine = &sacc[threadIdx.x >> 5][0][threadIdx.x & 31];
	const unsigned at = (unsigned)__cvta_generic_to_shared(mine);
#pragma unroll
	for (int i = 0; i < 32; i++) mine[32 * i] = 0.f;
	for (int i = threadIdx.x; i < C * C; i += blockDim.x) sW[i] = 0.f;
	if (threadIdx.x < C) sb[threadIdx.x] = 0.f;
	__syncthreads();
	const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
	const long long npix = (long long)T * T;
	float bsum[2][2] = {{0.f, 0.f}, {0.f, 0.f}}, Qr[2][2][2];
	LiftRow lift[4];
#pragma unroll
	for (int mt = 0; mt < 2; mt++) {
		if (LAST) {
#pragma unroll
			for (int h = 0; h < 2; h++) {
				Qr[0][mt][h] = wld(w, OFF_Q + 16 * mt + g + 8 * h);
				Qr[1][mt][h] = wld(w, OFF_Q + C + 16 * mt + g + 8 * h);
			}
		}
	}
	if (FIRST) {
#pragma unroll
		for (int nt = 0; nt < 4; nt++) lift[nt].load(w, 8 * nt + g);
	}
	const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
	for (long long r = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < nrows; r += nw) {
		const long long b = r / T;
		const int y = (int)(r - b * T);
		const long long base = b * C * npix + (long long)y * T, base2 = b * 2 * npix + (long long)y * T;
		float acc[2][2][4];
#pragma unroll
		for (int mt = 0; mt < 2; mt++)
#pragma unroll
			for (int nt = 0; nt < 2; nt++)
#pragma unroll
				for (int k = 0; k < 4; k++) acc[mt][nt][k] = 0.f;
		for (int tile = 0; tile < T / PX; tile++) {
			const int ps = tile * PX + 4 * t;
			// v^T as B fragments: channel 8 nt + g at the lane's pixels
			uint32_t vh[2][4][2], vl[2][4][2];
#pragma unroll
			for (int nt = 0; nt < 4; nt++) {
				float4 a, c;
				if (FIRST) {
					a = lift[nt].of(ld4u(x + base2 + ps, xvec), ld4u(x + base2 + npix + ps, xvec));
					c = lift[nt].of(ld4u(x + base2 + ps + 16, xvec), ld4u(x + base2 + npix + ps + 16, xvec));
				} else {
					a = ld4(v + base + (8 * nt + g) * npix + ps);
					c = ld4(v + base + (8 * nt + g) * npix + ps + 16);
				}
				split2(a.x, c.x, vh[0][nt][0], vl[0][nt][0]);
				split2(a.y, c.y, vh[0][nt][1], vl[0][nt][1]);
				split2(a.z, c.z, vh[1][nt][0], vl[1][nt][0]);
				split2(a.w, c.w, vh[1][nt][1], vl[1][nt][1]);
			}
#pragma unroll
			for (int mt = 0; mt < 2; mt++) {
				float d[4][4]; // dz as the accumulators of four n-tiles
#pragma unroll
				for (int h = 0; h < 2; h++) {
					const long long o = base + (16 * mt + g + 8 * h) * npix + ps;
#pragma unroll
					for (int c = 0; c < 2; c++) {
						float4 q;
						if (LAST) {
							const float4 e0 = ld4(dy + base2 + ps + 16 * c), e1 = ld4(dy + base2 + npix + ps + 16 * c);
							const float a0 = Qr[0][mt][h], a1 = Qr[1][mt][h];
							q = make_float4(a0 * e0.x + a1 * e1.x, a0 * e0.y + a1 * e1.y, a0 * e0.z + a1 * e1.z, a0 * e0.w + a1 * e1.w);
						} else {
							const float4 go = ld4(dz + o + 16 * c), zz = ld4(z + o + 16 * c);
							q = make_float4(go.x * gelu_d(zz.x), go.y * gelu_d(zz.y), go.z * gelu_d(zz.z), go.w * gelu_d(zz.w));
							st4(dz + o + 16 * c, q.x, q.y, q.z, q.w);
						}
						bsum[mt][h] += (q.x + q.y) + (q.z + q.w);
						d[0][2 * h + c] = q.x;
						d[1][2 * h + c] = q.y;
						d[2][2 * h + c] = q.z;
						d[3][2 * h + c] = q.w;
					}
				}
				float dW[4][4] = {};
#pragma unroll
				for (int ks = 0; ks < 2; ks++) {
					uint32_t ah[4], al[4];
#pragma unroll
					for (int h = 0; h < 2; h++) {
						split2(d[2 * ks + h][0], d[2 * ks + h][1], ah[2 * h], al[2 * h]);
						split2(d[2 * ks + h][2], d[2 * ks + h][3], ah[2 * h + 1], al[2 * h + 1]);
					}
#pragma unroll
					for (int nt = 0; nt < 2; nt++) mma_split(acc[mt][nt], ah, al, __ldg(fe + ((tile * 2 + ks) * 2 + nt) * 32 + lane));
#pragma unroll
					for (int nt = 0; nt < 4; nt++) {
						mma_bf16(dW[nt], ah, vh[ks][nt]);
						mma_bf16(dW[nt], ah, vl[ks][nt]);
						mma_bf16(dW[nt], al, vh[ks][nt]);
					}
				}
#pragma unroll
				for (int i = 0; i < 16; i++) {
					// no other thread's and no other access: nothing to order global loads by
					float q;
					asm volatile("ld.shared.f32 %0, [%1];" : "=f"(q) : "r"(at + 128 * (16 * mt + i)));
					q += dW[i >> 2][i & 3];
					asm volatile("st.shared.f32 [%0], %1;" ::"r"(at + 128 * (16 * mt + i)), "f"(q));
				}
			}
		}
#pragma unroll
		for (int mt = 0; mt < 2; mt++) store_modes(A, acc[mt], b, y, T, mt, g, t, sx);
	}
	asm volatile("" ::: "memory"); // mine[] was written behind the compiler's back
#pragma unroll
	for (int mt = 0; mt < 2; mt++) {
#pragma unroll
		for (int nt = 0; nt < 4; nt++) {
			const int o = 16 * mt + g, i = 8 * nt + 2 * t;
			atomicAdd(&sW[o * C + i], mine[32 * (16 * mt + 4 * nt + 0)]);
			atomicAdd(&sW[o * C + i + 1], mine[32 * (16 * mt + 4 * nt + 1)]);
			atomicAdd(&sW[(o + 8) * C + i], mine[32 * (16 * mt + 4 * nt + 2)]);
			atomicAdd(&sW[(o + 8) * C + i + 1], mine[32 * (16 * mt + 4 * nt + 3)]);
		}
		// bias: the four lanes of a group hold disjoint pixels of the same rows
#pragma unroll
		for (int h = 0; h < 2; h++) {
			float q = bsum[mt][h];
			q += __shfl_xor_sync(0xffffffffu, q, 1);
			q += __shfl_xor_sync(0xffffffffu, q, 2);
			if (t == 0) atomicAdd(&sb[16 * mt + g + 8 * h], q);
		}
	}
	__syncthreads();
	for (int i = threadIdx.x; i < C * C; i += blockDim.x) atomicAdd(&gW[i], sW[i]);
	if (threadIdx.x < C) atomicAdd(&gb[threadIdx.x], sb[threadIdx.x]);
}

// Second half, a warp per row: dv = W^T dz + the x transform's adjoint of the mixed
// modes, written over dz. LAST: dz = Q^T dy. FIRST: dv is not stored; dP[c][j] +=
// dv[c] x[j] and dp[c] += dv[c], summed over pixels.
template <bool FIRST, bool LAST>
__global__ void __launch_bounds__(128, 3)
    layer_bwd(const float* __restrict__ x, int xvec, const float* __restrict__ dy, const float2* __restrict__ Aq,
              const __nv_bfloat16* __restrict__ w, int l, const uint4* __restrict__ ff, float* dz, float* __restrict__ gr,
              long long nrows, int T) {
	const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
	const long long npix = (long long)T * T;
	__shared__ uint4 sw[4][32]; // the weights' A fragments (in registers they cost a block per SM)
	uint32_t aw[2][2][4];
	float Qk[2][2][4], gp[3][2][2];
#pragma unroll
	for (int ks = 0; ks < 2; ks++) {
		const int o = 16 * ks + 2 * t;
#pragma unroll
		for (int mt = 0; mt < 2; mt++)
#pragma unroll
			for (int h = 0; h < 2; h++) {
				const size_t col = off_W(l) + 16 * mt + g + 8 * h; // W[o][i] at col + o C
				aw[mt][ks][h] = pack_bf16(w, col + (size_t)o * C, col + (size_t)(o + 1) * C);
				aw[mt][ks][2 + h] = pack_bf16(w, col + (size_t)(o + 8) * C, col + (size_t)(o + 9) * C);
			}
		if (LAST) {
#pragma unroll
			for (int k = 0; k < 4; k++) {
				Qk[0][ks][k] = wld(w, OFF_Q + o + (k & 1) + 8 * (k >> 1));
				Qk[1][ks][k] = wld(w, OFF_Q + C + o + (k & 1) + 8 * (k >> 1));
			}
		}
	}
	if (threadIdx.x < 32)
#pragma unroll
		for (int k = 0; k < 4; k++) sw[k][lane] = make_uint4(aw[k >> 1][k & 1][0], aw[k >> 1][k & 1][1], aw[k >> 1][k & 1][2], aw[k >> 1][k & 1][3]);
	__syncthreads();
#pragma unroll
	for (int j = 0; j < 3; j++)
#pragma unroll
		for (int mt = 0; mt < 2; mt++)
#pragma unroll
			for (int h = 0; h < 2; h++) gp[j][mt][h] = 0.f;
	const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
	for (long long r = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < nrows; r += nw) {
		const long long b = r / T;
		const int y = (int)(r - b * T);
		const long long base = b * C * npix + (long long)y * T, base2 = b * 2 * npix + (long long)y * T;
		uint32_t mh[2][4], ml[2][4];
#pragma unroll
		for (int mt = 0; mt < 2; mt++) load_modes(Aq, b, y, T, mt, g, t, 1.f, 1.f, mh[mt], ml[mt]);
		for (int tile = 0; tile < T / PX; tile++) {
			const int pl = tile * PX + px_of(g, 0), ps = tile * PX + 4 * t;
			float4 vv[2][4];
			if (LAST) {
				const float4 e0 = ld4(dy + base2 + pl), e1 = ld4(dy + base2 + npix + pl);
#pragma unroll
				for (int ks = 0; ks < 2; ks++)
#pragma unroll
					for (int k = 0; k < 4; k++) {
						const float a0 = Qk[0][ks][k], a1 = Qk[1][ks][k];
						vv[ks][k] = make_float4(a0 * e0.x + a1 * e1.x, a0 * e0.y + a1 * e1.y, a0 * e0.z + a1 * e1.z, a0 * e0.w + a1 * e1.w);
					}
			} else {
#pragma unroll
				for (int ks = 0; ks < 2; ks++)
#pragma unroll
					for (int k = 0; k < 4; k++) vv[ks][k] = ld4(dz + base + (16 * ks + 2 * t + (k & 1) + 8 * (k >> 1)) * npix + pl);
			}
			float d[2][4][4];
#pragma unroll
			for (int j = 0; j < 4; j++) {
				const uint4 f = __ldg(ff + (tile * 4 + j) * 32 + lane);
#pragma unroll
				for (int mt = 0; mt < 2; mt++)
#pragma unroll
					for (int k = 0; k < 4; k++) d[mt][j][k] = 0.f;
#pragma unroll
				for (int ks = 0; ks < 2; ks++) {
					uint32_t bh[2], bl[2];
					split2(at(vv[ks][0], j), at(vv[ks][1], j), bh[0], bl[0]);
					split2(at(vv[ks][2], j), at(vv[ks][3], j), bh[1], bl[1]);
#pragma unroll
					for (int mt = 0; mt < 2; mt++) {
						uint32_t aq[4];
						ld_frag(aq, &sw[2 * mt + ks][lane]);
						mma_bf16(d[mt][j], aq, bh);
						mma_bf16(d[mt][j], aq, bl);
					}
				}
#pragma unroll
				for (int mt = 0; mt < 2; mt++) {
					float e[4] = {0.f, 0.f, 0.f, 0.f};
					mma_split(e, mh[mt], ml[mt], f);
#pragma unroll
					for (int k = 0; k < 4; k++) d[mt][j][k] += e[k];
				}
			}
			__syncwarp(); // every lane's loads of this block before its stores over it
#pragma unroll
			for (int c = 0; c < 2; c++) {
				float4 x0, x1;
				if (FIRST) {
					x0 = ld4u(x + base2 + ps + 16 * c, xvec);
					x1 = ld4u(x + base2 + npix + ps + 16 * c, xvec);
				}
#pragma unroll
				for (int mt = 0; mt < 2; mt++)
#pragma unroll
					for (int h = 0; h < 2; h++) {
						const float a0 = d[mt][0][2 * h + c], a1 = d[mt][1][2 * h + c], a2 = d[mt][2][2 * h + c], a3 = d[mt][3][2 * h + c];
						if (FIRST) {
							gp[0][mt][h] += (a0 * x0.x + a1 * x0.y) + (a2 * x0.z + a3 * x0.w);
							gp[1][mt][h] += (a0 * x1.x + a1 * x1.y) + (a2 * x1.z + a3 * x1.w);
							gp[2][mt][h] += (a0 + a1) + (a2 + a3);
						} else {
							st4(dz + base + (16 * mt + g + 8 * h) * npix + ps + 16 * c, a0, a1, a2, a3);
						}
					}
			}
		}
	}
	if constexpr (FIRST) {
		__shared__ float sp[3 * C];
		for (int i = threadIdx.x; i < 3 * C; i += blockDim.x) sp[i] = 0.f;
		__syncthreads();
#pragma unroll
		for (int j = 0; j < 3; j++)
#pragma unroll
			for (int mt = 0; mt < 2; mt++)
#pragma unroll
				for (int h = 0; h < 2; h++) {
					float a = gp[j][mt][h];
					a += __shfl_xor_sync(0xffffffffu, a, 1);
					a += __shfl_xor_sync(0xffffffffu, a, 2);
					const int c = 16 * mt + g + 8 * h;
					if (t == 0) atomicAdd(&sp[j < 2 ? 2 * c + j : 2 * C + c], a);
				}
		__syncthreads();
		for (int i = threadIdx.x; i < 3 * C; i += blockDim.x) atomicAdd(gr + OFF_P + i, sp[i]);
	}
}
static_assert(OFF_PB == OFF_P + 2 * C, "p follows P");

// The truncated transforms along y, per plane of [rows][MX] complex values:
//   forward: out[k][m] = sum_y in[y][m] exp(-2 pi i ky(k) y / T), k < MY
//   inverse: out[y][m] = sum_k in[k][m] exp(+2 pi i ky(k) y / T), y < T
// are GEMMs against fixed twiddle matrices, on the tensor cores with one warp
// per plane. The twiddles are the A operand, their BF16-split fragments
// tabulated once per tile size (dfty_frag_kernel); the plane's values are the
// B operand, split per use, with three products (hi hi, hi lo, lo hi):
//   forward: D[k][2m + q] = sum_{y, c} E[k][2y + c] Z[2y + c][2m + q], (E[k][2y], E[k][2y + 1]) = (cos, sin)(2 pi ky(k) y / T)
//   inverse: D[y][2m + q] = sum_{k, c} F[y][2k + c] Z[2k + c][2m + q], (F[y][2k], F[y][2k + 1]) = (cos, -sin)(2 pi ky(k) y / T)
// with Z[2j][2m] = Re z[j][m], Z[2j + 1][2m] = Im, Z[2j][2m + 1] = Im, Z[2j + 1][2m + 1] = -Re, so that
// the accumulator pair of columns 2t, 2t + 1 is one output's (Re, Im).
static_assert(MY == 16 && MX == 8, "one m16 tile of modes and two n8 tiles of (Re, Im) columns");

// fdy: [T/8 k-steps][32 lanes][hi, lo], fiy: [T/16 m-tiles][2 k-steps][32 lanes][hi, lo];
// each uint4 holds the four A registers (rows g, g + 8 by columns 2t, 2t + 8)
__global__ void dfty_frag_kernel(const float2* __restrict__ tw, int T, uint4* __restrict__ fdy, uint4* __restrict__ fiy) {
	const int nf = T / 8 * 32, ni = T / 16 * 2 * 32;
	for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < nf + ni; e += gridDim.x * blockDim.x) {
		const bool fwd = e < nf;
		const int f = fwd ? e : e - nf;
		const int lane = f & 31, g = lane >> 2, t = lane & 3;
		int rows[2], cols[2];
		if (fwd) {
			const int ks = f >> 5;
			rows[0] = g;
			rows[1] = g + 8;
			cols[0] = 8 * ks + t;
			cols[1] = cols[0] + 4;
		} else {
			const int ks = (f >> 5) & 1, mt = f >> 6;
			rows[0] = 16 * mt + g;
			rows[1] = rows[0] + 8;
			cols[0] = 8 * ks + t;
			cols[1] = cols[0] + 4;
		}
		uint32_t hi[4], lo[4];
#pragma unroll
		for (int r = 0; r < 4; r++) {
			// register r: row rows[r & 1], column pair of cols[r >> 1]
			const int row = rows[r & 1], col = cols[r >> 1];
			const int ky = ky_of(fwd ? row : col, T), y = fwd ? col : row;
			const float2 w = tw[(ky * y) & (T - 1)];
			split2(w.x, fwd ? w.y : -w.y, hi[r], lo[r]);
		}
		uint4* dst = (fwd ? fdy : fiy) + 2 * f;
		dst[0] = make_uint4(hi[0], hi[1], hi[2], hi[3]);
		dst[1] = make_uint4(lo[0], lo[1], lo[2], lo[3]);
	}
}

// the B registers of value z in the output column of parity q: (Re, Im) or (Im, -Re)
__device__ __forceinline__ void zsplit(float2 z, int q, uint32_t& hi, uint32_t& lo) {
	if (q) split2(z.y, -z.x, hi, lo);
	else split2(z.x, z.y, hi, lo);
}

// One block of four warps per plane. Forward: warp w takes the k-steps
// w, w + 4, ... and the warps' partial sums are added in shared memory in a
// fixed order. Inverse: warp w takes the m-tiles w, w + 4, ...
constexpr int DY_WARPS = 4;

__global__ void __launch_bounds__(32 * DY_WARPS) dft_y_fwd(const float2* __restrict__ in, float2* __restrict__ out,
                                                          const uint4* __restrict__ fdy, long long nplanes, int T) {
	__shared__ float red[DY_WARPS][32][8];
	const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3, q = g & 1;
	for (long long plane = blockIdx.x; plane < nplanes; plane += gridDim.x) {
		const float2* pin = in + plane * T * MX;
		float d[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll 4
		for (int ks = wp; ks < T / 8; ks += DY_WARPS) {
			const uint4 fh = __ldg(fdy + (ks * 32 + lane) * 2), fl = __ldg(fdy + (ks * 32 + lane) * 2 + 1);
			const uint32_t ah[4] = {fh.x, fh.y, fh.z, fh.w}, al[4] = {fl.x, fl.y, fl.z, fl.w};
			const int y0 = 8 * ks + t;
#pragma unroll
			for (int nt = 0; nt < 2; nt++) {
				const int m = 4 * nt + (g >> 1);
				uint32_t bh[2], bl[2];
				zsplit(pin[y0 * MX + m], q, bh[0], bl[0]);
				zsplit(pin[(y0 + 4) * MX + m], q, bh[1], bl[1]);
				mma_bf16(d[nt], ah, bh);
				mma_bf16(d[nt], ah, bl);
				mma_bf16(d[nt], al, bh);
			}
		}
		__syncthreads(); // the previous plane's sums have been read
#pragma unroll
		for (int j = 0; j < 8; j++) red[wp][lane][j] = d[j >> 2][j & 3];
		__syncthreads();
		if (wp == 0) {
#pragma unroll
			for (int j = 0; j < 8; j++) d[j >> 2][j & 3] = red[0][lane][j] + red[1][lane][j] + red[2][lane][j] + red[3][lane][j];
			float2* pout = out + plane * MY * MX;
#pragma unroll
			for (int nt = 0; nt < 2; nt++) {
				const int m = 4 * nt + t;
				pout[g * MX + m] = make_float2(d[nt][0], d[nt][1]);
				pout[(g + 8) * MX + m] = make_float2(d[nt][2], d[nt][3]);
			}
		}
	}
}

__global__ void __launch_bounds__(32 * DY_WARPS) dft_y_inv(const float2* __restrict__ in, float2* __restrict__ out,
                                                          const uint4* __restrict__ fiy, long long nplanes, int T) {
	const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3, q = g & 1;
	for (long long plane = blockIdx.x; plane < nplanes; plane += gridDim.x) {
		const float2* pin = in + plane * MY * MX;
		// the whole plane as B fragments: two k-steps (K = 2 MY) by two n-tiles
		uint32_t bh[2][2][2], bl[2][2][2];
#pragma unroll
		for (int ks = 0; ks < 2; ks++)
#pragma unroll
			for (int nt = 0; nt < 2; nt++) {
				const int k0 = 8 * ks + t, m = 4 * nt + (g >> 1);
				zsplit(pin[k0 * MX + m], q, bh[ks][nt][0], bl[ks][nt][0]);
				zsplit(pin[(k0 + 4) * MX + m], q, bh[ks][nt][1], bl[ks][nt][1]);
			}
		float2* pout = out + plane * T * MX;
#pragma unroll 2
		for (int mt = wp; mt < T / 16; mt += DY_WARPS) {
			float d[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
			for (int ks = 0; ks < 2; ks++) {
				const uint4 fh = __ldg(fiy + ((mt * 2 + ks) * 32 + lane) * 2);
				const uint4 fl = __ldg(fiy + ((mt * 2 + ks) * 32 + lane) * 2 + 1);
				const uint32_t ah[4] = {fh.x, fh.y, fh.z, fh.w}, al[4] = {fl.x, fl.y, fl.z, fl.w};
#pragma unroll
				for (int nt = 0; nt < 2; nt++) {
					mma_bf16(d[nt], ah, bh[ks][nt]);
					mma_bf16(d[nt], ah, bl[ks][nt]);
					mma_bf16(d[nt], al, bh[ks][nt]);
				}
			}
			const int y0 = 16 * mt + g;
#pragma unroll
			for (int nt = 0; nt < 2; nt++) {
				const int m = 4 * nt + t;
				pout[y0 * MX + m] = make_float2(d[nt][0], d[nt][1]);
				pout[(y0 + 8) * MX + m] = make_float2(d[nt][2], d[nt][3]);
			}
		}
	}
}

// Mode mixing, per retained mode km:
//   forward: out[b][o][km] = sum_i R[i][o][km] in[b][i][km]
//   adjoint: out[b][i][km] = sum_o conj(R[i][o][km]) in[b][o][km]
// On the tensor cores, one warp per mode and 16 batch rows: D[b][2o + q] =
// sum_{i, c} A[b][2i + c] M[2i + c][2o + q] with A = (Re, Im) of the inputs
// (BF16 high parts and remainders, two products) and M the real 64 x 64 form
// of R or of conj(R)^T, whose entries are the exact BF16 weights:
//   forward: M[2i][2o] = Rr, M[2i+1][2o] = -Ri, M[2i][2o+1] = Ri, M[2i+1][2o+1] = Rr  (of R[i][o])
//   adjoint: M[2o][2i] = Rr, M[2o+1][2i] = Ri, M[2o][2i+1] = -Ri, M[2o+1][2i+1] = Rr
// (M's rows indexed by the step's input channel, its columns by the output).
// The accumulator pair of columns 2t, 2t + 1 is one output's (Re, Im).
__device__ __forceinline__ uint32_t bf16_pair(unsigned short lo, unsigned short hi) { return (uint32_t)lo | ((uint32_t)hi << 16); }

__global__ void __launch_bounds__(128) mix(const float2* __restrict__ in, float2* __restrict__ out,
                                           const __nv_bfloat16* __restrict__ w, int l, int B, int adjoint) {
	const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
	const int mtiles = (B + 15) / 16;
	const unsigned short* Rr = reinterpret_cast<const unsigned short*>(w + off_Rr(l));
	const unsigned short* Ri = reinterpret_cast<const unsigned short*>(w + off_Ri(l));
	const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
	// one warp per (n-tile of eight output columns, mode, 16 batch rows); whole
	// warps take the same items, so the mma.sync lanes stay converged
	for (long long wid = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; wid < (long long)NK * mtiles * 8;
	     wid += nw) {
		const int nt = (int)(wid & 7), km = (int)((wid >> 3) % NK), mt = (int)((wid >> 3) / NK);
		const int b0 = 16 * mt + g, b1 = b0 + 8;
		const int col = 4 * nt + (g >> 1), q = g & 1; // output channel and part of column 8 nt + g
		float d[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
		for (int ks = 0; ks < 4; ks++) {
			const int i0 = 8 * ks + t, i1 = i0 + 4;
			const float2 zero = make_float2(0.f, 0.f);
			const float2 z00 = b0 < B ? in[((long long)b0 * C + i0) * NK + km] : zero;
			const float2 z10 = b1 < B ? in[((long long)b1 * C + i0) * NK + km] : zero;
			const float2 z01 = b0 < B ? in[((long long)b0 * C + i1) * NK + km] : zero;
			const float2 z11 = b1 < B ? in[((long long)b1 * C + i1) * NK + km] : zero;
			uint32_t ah[4], al[4];
			split2(z00.x, z00.y, ah[0], al[0]);
			split2(z10.x, z10.y, ah[1], al[1]);
			split2(z01.x, z01.y, ah[2], al[2]);
			split2(z11.x, z11.y, ah[3], al[3]);
			uint32_t bw[2];
#pragma unroll
			for (int h = 0; h < 2; h++) {
				const int row = 8 * ks + t + 4 * h; // input channel of rows 16 ks + 2t (+8 h), + 1
				const size_t idx = adjoint ? ((size_t)col * C + row) * NK + km : ((size_t)row * C + col) * NK + km;
				const unsigned short rr = Rr[idx], ri = Ri[idx], nri = ri ^ 0x8000u;
				if (!adjoint) bw[h] = q ? bf16_pair(ri, rr) : bf16_pair(rr, nri);
				else bw[h] = q ? bf16_pair(nri, rr) : bf16_pair(rr, ri);
			}
			mma_bf16(d, ah, bw);
			mma_bf16(d, al, bw);
		}
		const int oc = 4 * nt + t;
		if (b0 < B) out[((long long)b0 * C + oc) * NK + km] = make_float2(d[0], d[1]);
		if (b1 < B) out[((long long)b1 * C + oc) * NK + km] = make_float2(d[2], d[3]);
	}
}

// dR[i][o][km] += sum_b dY[b][o][km] conj(X[b][i][km])
__global__ void mix_grad(const float2* __restrict__ X, const float2* __restrict__ dY, float* __restrict__ g, int l, int B) {
	const long long n = (long long)C * C * NK;
	for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
		const int km = (int)(t % NK);
		const int o = (int)((t / NK) % C);
		const int i = (int)(t / ((long long)NK * C));
		float gr = 0.f, gi = 0.f;
		for (int b = 0; b < B; b++) {
			const float2 x = X[((long long)b * C + i) * NK + km];
			const float2 d = dY[((long long)b * C + o) * NK + km];
			gr += d.x * x.x + d.y * x.y;
			gi += d.y * x.x - d.x * x.y;
		}
		g[off_Rr(l) + t] += gr;
		g[off_Ri(l) + t] += gi;
	}
}

__global__ void to_bf16(const float* __restrict__ a, __nv_bfloat16* __restrict__ b, long long n) {
	for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
		b[i] = __float2bfloat16(a[i]);
}

__global__ void adam_kernel(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m,
                            float* __restrict__ v, long long n, float lr, float b1, float b2, float eps, float c1,
                            float c2) {
	for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
		const float gi = g[i];
		const float mi = b1 * m[i] + (1.f - b1) * gi;
		const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
		m[i] = mi;
		v[i] = vi;
		p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
	}
}

// Tiles of a periodic two-field FP64 grid as FP32 network input. Tile j of the
// batch is block (first + j) of the grid's core x core blocks (row-major over
// tiles_x columns) plus halo points on each side, wrapped periodically. One warp
// per row of a tile and field.
__global__ void gather_tiles(const double* __restrict__ f, float* __restrict__ out, int Nx, int Ny, int T, int core,
                             int halo, int tiles_x, int first, int count) {
	const int lane = threadIdx.x & 31, nw = (gridDim.x * blockDim.x) >> 5;
	for (int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < 2 * T * count; r += nw) {
		const int ty = r % T, u = (r / T) & 1, tile = first + r / (2 * T);
		const int by = tile / tiles_x, bx = tile - by * tiles_x;
		int y = (by * core - halo + ty) % Ny, x0 = (bx * core - halo) % Nx;
		if (y < 0) y += Ny;
		if (x0 < 0) x0 += Nx;
		const double* row = f + ((long long)u * Ny + y) * Nx;
		float* o = out + (long long)r * T;
		for (int tx = lane; tx < T; tx += 32) {
			int x = x0 + tx;
			while (x >= Nx) x -= Nx; // at most T / Nx turns
			o[tx] = (float)row[x];
		}
	}
}

// Writes each tile's core block of the network output back to the grid, one warp
// per row of a core and field.
__global__ void scatter_tiles(const float* __restrict__ in, double* __restrict__ f, int Nx, int Ny, int T, int core,
                              int halo, int tiles_x, int first, int count) {
	const int lane = threadIdx.x & 31, nw = (gridDim.x * blockDim.x) >> 5;
	for (int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < 2 * core * count; r += nw) {
		const int cy = r % core, u = (r / core) & 1, j = r / (2 * core), tile = first + j;
		const int by = tile / tiles_x, bx = tile - by * tiles_x;
		const int y = by * core + cy, x0 = bx * core;
		if (y >= Ny) continue;
		const float* i = in + (((long long)j * 2 + u) * T + halo + cy) * T + halo;
		double* row = f + ((long long)u * Ny + y) * Nx + x0;
		for (int cx = lane; cx < core && x0 + cx < Nx; cx += 32) row[cx] = (double)i[cx];
	}
}

// Per-block FP64 partial sums of (out - in) for each of the two fields.
constexpr int MEAN_BLOCKS = 296;
__global__ void diff_partials(const double* __restrict__ in, const double* __restrict__ out, double* __restrict__ part,
                              long long npts) {
	__shared__ double red[2][32];
	for (int u = 0; u < 2; u++) {
		double s = 0.0;
		for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < npts;
		     i += (long long)gridDim.x * blockDim.x)
			s += out[u * npts + i] - in[u * npts + i];
		s = warp_sum(s);
		if ((threadIdx.x & 31) == 0) red[u][threadIdx.x >> 5] = s;
	}
	__syncthreads();
	if (threadIdx.x < 32) {
		for (int u = 0; u < 2; u++) {
			double s = threadIdx.x < (blockDim.x >> 5) ? red[u][threadIdx.x] : 0.0;
			s = warp_sum(s);
			if (threadIdx.x == 0) part[u * gridDim.x + blockIdx.x] = s;
		}
	}
}

// out[u] -= (sum of the partials of u) / npts: gives each field back the
// input's mean (the relaxation conserves it). Fixed summation order.
__global__ void restore_means(double* __restrict__ out, const double* __restrict__ part, int nparts, long long npts) {
	__shared__ double shift[2];
	if (threadIdx.x < 2) {
		double s = 0.0;
		for (int i = 0; i < nparts; i++) s += part[threadIdx.x * nparts + i];
		shift[threadIdx.x] = s / (double)npts;
	}
	__syncthreads();
	for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < 2 * npts;
	     i += (long long)gridDim.x * blockDim.x)
		out[i] -= shift[i >= npts];
}

int grid_for(long long n, int block) {
	long long g = (n + block - 1) / block;
	return (int)(g > 148 * 16 ? 148 * 16 : (g < 1 ? 1 : g));
}


thread_local std::string g_fno_err;

} // namespace

struct pfcg_fno {
	int T = 0, maxB = 0;
	cudaStream_t stream = nullptr;
	float* p = nullptr;          // master weights (FP32)
	__nv_bfloat16* w = nullptr;  // BF16 copy read by the kernels
	float* g = nullptr;          // gradients
	float* am = nullptr;         // Adam moments
	float* av = nullptr;
	long long adam_t = 0;
	float2* tw = nullptr;        // twiddles of the tile size
	uint4* fe = nullptr;         // mma fragments of the truncated x transforms (dft_frag_kernel)
	uint4* ff = nullptr;
	uint4* fdy = nullptr;        // mma fragments of the truncated y transforms (dfty_frag_kernel)
	uint4* fiy = nullptr;
	float* sx = nullptr;         // per-kx weights of the truncated irfft2: (kx ? 2 : 1) / T^2
	float* v[L] = {};            // inputs of layers 1 .. L-1 (layer 0's is the lift of x)
	float* z[L - 1] = {};        // pre-activations (the last layer has no activation)
	float2* A = nullptr;         // [B][C][T][MX] x-transformed rows (and adjoint scratch)
	float2* X[L] = {};           // [B][C][MY][MX] retained modes of each layer input
	float2* Y = nullptr;         // [B][C][MY][MX] mixed modes
	float2* Bq = nullptr;        // [B][C][T][MX] y-inverse rows (and adjoint scratch)
	float* dv = nullptr;         // gradient of a layer's output, pre-activation and input in turn
	float* x = nullptr;          // [B][2][T][T] tile input (apply)
	float* y = nullptr;          // [B][2][T][T] network output
	float* dy = nullptr;
	double* loss = nullptr;
	double* field_tmp = nullptr; // grid-sized scratch for the warm start
	size_t field_tmp_n = 0;
	double* part = nullptr;      // mean partial sums [2][MEAN_BLOCKS]
	long long launches = 0;
	std::string err;
};

namespace {

int ffail(pfcg_fno* f, int code, const std::string& m) {
	if (f) f->err = m;
	g_fno_err = m;
	return code;
}

#define FCK(call)                                                                                                      \
	do {                                                                                                           \
		cudaError_t e_ = (call);                                                                               \
		if (e_ != cudaSuccess) return ffail(f, PFCG_ECUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
	} while (0)

int grid_rows(long long nrows) { return grid_for(nrows * 32, 128); }

// forward pass over a batch of B tiles; with a target also the loss, dy, the
// pre-activations for backward and the projection's gradients (into f->g, cleared here)
int forward(pfcg_fno* f, const float* x, int B, const float* target) {
	const int T = f->T;
	const long long rows = (long long)B * T, planes = (long long)B * C;
	const int vec = (reinterpret_cast<uintptr_t>(x) & 15) == 0;
	cudaStream_t st = f->stream;
	if (target) {
		FCK(cudaMemsetAsync(f->g, 0, sizeof(float) * NPARAM, st));
		FCK(cudaMemsetAsync(f->loss, 0, sizeof(double), st));
	}
	lift_dft<<<grid_rows(rows), 128, 0, st>>>(x, f->w, reinterpret_cast<float*>(f->A), f->tw, rows, T);
	f->launches++;
	for (int l = 0; l < L; l++) {
		dft_y_fwd<<<grid_for(planes * 32 * DY_WARPS, 32 * DY_WARPS), 32 * DY_WARPS, 0, st>>>(f->A, f->X[l], f->fdy, planes, T);
		mix<<<grid_for((long long)NK * ((B + 15) / 16) * 8 * 32, 128), 128, 0, st>>>(f->X[l], f->Y, f->w, l, B, 0);
		dft_y_inv<<<grid_for(planes * 32 * DY_WARPS, 32 * DY_WARPS), 32 * DY_WARPS, 0, st>>>(f->Y, f->Bq, f->fiy, planes, T);
#define PFCG_LAYER(FI, LA, TR)                                                                                        \
	layer_fwd<FI, LA, TR><<<grid_rows(rows), 128, 0, st>>>(x, vec, f->v[l], f->Bq, f->w, l, f->fe, f->ff, f->sx,      \
	                                                       l < L - 1 ? f->z[l] : nullptr, l < L - 1 ? f->v[l + 1] : nullptr, \
	                                                       f->A, f->y, target, f->dy, f->loss, f->g, rows, T, B)
		if (l == 0) {
			if (target) PFCG_LAYER(true, false, true);
			else PFCG_LAYER(true, false, false);
		} else if (l < L - 1) {
			if (target) PFCG_LAYER(false, false, true);
			else PFCG_LAYER(false, false, false);
		} else {
			if (target) PFCG_LAYER(false, true, true);
			else PFCG_LAYER(false, true, false);
		}
#undef PFCG_LAYER
		f->launches += 4;
	}
	FCK(cudaGetLastError());
	return 0;
}

// gradients of every parameter after forward() with a target
int backward(pfcg_fno* f, const float* x, int B) {
	const int T = f->T;
	const long long rows = (long long)B * T, planes = (long long)B * C;
	const int vec = (reinterpret_cast<uintptr_t>(x) & 15) == 0;
	cudaStream_t st = f->stream;
	const int gr = grid_rows(rows);
	for (int l = L - 1; l >= 0; l--) {
		float* gW = f->g + off_W(l);
		float* gb = f->g + off_b(l);
		const float* z = l < L - 1 ? f->z[l] : nullptr;
		if (l == L - 1)
			layer_grad<false, true><<<gr, 128, 0, st>>>(x, vec, f->v[l], z, f->dv, f->dy, f->w, f->fe, f->sx, f->Bq, gW, gb, rows, T);
		else if (l > 0)
			layer_grad<false, false><<<gr, 128, 0, st>>>(x, vec, f->v[l], z, f->dv, f->dy, f->w, f->fe, f->sx, f->Bq, gW, gb, rows, T);
		else
			layer_grad<true, false><<<gr, 128, 0, st>>>(x, vec, nullptr, z, f->dv, f->dy, f->w, f->fe, f->sx, f->Bq, gW, gb, rows, T);
		// spectral branch, in reverse
		dft_y_fwd<<<grid_for(planes * 32 * DY_WARPS, 32 * DY_WARPS), 32 * DY_WARPS, 0, st>>>(f->Bq, f->Y, f->fdy, planes, T);
		mix_grad<<<grid_for((long long)C * C * NK, 256), 256, 0, st>>>(f->X[l], f->Y, f->g, l, B);
		mix<<<grid_for((long long)NK * ((B + 15) / 16) * 8 * 32, 128), 128, 0, st>>>(f->Y, f->Bq, f->w, l, B, 1);
		dft_y_inv<<<grid_for(planes * 32 * DY_WARPS, 32 * DY_WARPS), 32 * DY_WARPS, 0, st>>>(f->Bq, f->A, f->fiy, planes, T);
		if (l == L - 1)
			layer_bwd<false, true><<<gr, 128, 0, st>>>(x, vec, f->dy, f->A, f->w, l, f->ff, f->dv, f->g, rows, T);
		else if (l > 0)
			layer_bwd<false, false><<<gr, 128, 0, st>>>(x, vec, f->dy, f->A, f->w, l, f->ff, f->dv, f->g, rows, T);
		else
			layer_bwd<true, false><<<gr, 128, 0, st>>>(x, vec, f->dy, f->A, f->w, l, f->ff, f->dv, f->g, rows, T);
		f->launches += 6;
	}
	FCK(cudaGetLastError());
	return 0;
}

} // namespace

int fno_apply_device(pfcg_fno* f, const double* d_in, double* d_out, int Nx, int Ny, cudaStream_t st) {
	const int T = f->T, halo = T / 4, core = T - 2 * halo;
	const int tx = (Nx + core - 1) / core, ty = (Ny + core - 1) / core;
	const int ntiles = tx * ty;
	const cudaStream_t own = f->stream;
	cudaEvent_t ev;
	FCK(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
	FCK(cudaEventRecord(ev, st));
	FCK(cudaStreamWaitEvent(own, ev, 0));
	for (int first = 0; first < ntiles; first += f->maxB) {
		const int count = std::min(f->maxB, ntiles - first);
		gather_tiles<<<grid_for(2LL * T * count * 32, 256), 256, 0, own>>>(d_in, f->x, Nx, Ny, T, core, halo, tx, first,
		                                                                  count);
		f->launches++;
		int rc = forward(f, f->x, count, nullptr);
		if (rc) return rc;
		scatter_tiles<<<grid_for(2LL * core * count * 32, 256), 256, 0, own>>>(f->y, d_out, Nx, Ny, T, core, halo, tx,
		                                                                         first, count);
		f->launches++;
	}
	const long long npts = (long long)Nx * Ny;
	diff_partials<<<MEAN_BLOCKS, 256, 0, own>>>(d_in, d_out, f->part, npts);
	restore_means<<<grid_for(2 * npts, 256), 256, 0, own>>>(d_out, f->part, MEAN_BLOCKS, npts);
	f->launches += 2;
	FCK(cudaGetLastError());
	FCK(cudaEventRecord(ev, own));
	FCK(cudaStreamWaitEvent(st, ev, 0));
	FCK(cudaEventDestroy(ev));
	return 0;
}

int fno_scratch_grid(pfcg_fno* f, size_t n, double** out) {
	if (f->field_tmp_n < n) {
		cudaFree(f->field_tmp);
		f->field_tmp = nullptr;
		f->field_tmp_n = 0;
		FCK(cudaMalloc(&f->field_tmp, sizeof(double) * n));
		f->field_tmp_n = n;
	}
	*out = f->field_tmp;
	return 0;
}

const char* fno_error(const pfcg_fno* f) { return f->err.c_str(); }

extern "C" {

size_t pfcg_fno_param_count(void) { return NPARAM; }

int pfcg_fno_create(int tile, int max_batch, pfcg_fno** out) {
	if (!out) return ffail(nullptr, PFCG_EARG, "NULL argument");
	*out = nullptr;
	if (tile < 2 * MY || tile > MAXT || (tile & (tile - 1)) != 0 || max_batch < 1)
		return ffail(nullptr, PFCG_EARG, "tile must be a power of two in [32, 512] and max_batch >= 1");
	pfcg_fno* f = new pfcg_fno();
	f->T = tile;
	f->maxB = max_batch;
	const long long npix = (long long)tile * tile;
	const size_t nv = (size_t)max_batch * C * npix;
	cudaError_t e = cudaStreamCreateWithFlags(&f->stream, cudaStreamNonBlocking);
	std::vector<void**> bufs;
	std::vector<size_t> sizes;
	auto add = [&](void** ptr, size_t bytes) {
		bufs.push_back(ptr);
		sizes.push_back(bytes);
	};
	// the first five (weights, gradients, moments) are cleared below
	add((void**)&f->p, sizeof(float) * NPARAM);
	add((void**)&f->w, sizeof(__nv_bfloat16) * NPARAM);
	add((void**)&f->g, sizeof(float) * NPARAM);
	add((void**)&f->am, sizeof(float) * NPARAM);
	add((void**)&f->av, sizeof(float) * NPARAM);
	add((void**)&f->tw, sizeof(float2) * tile);
	add((void**)&f->fe, sizeof(uint4) * (tile / PX) * 4 * 32);
	add((void**)&f->ff, sizeof(uint4) * (tile / PX) * 4 * 32);
	add((void**)&f->fdy, sizeof(uint4) * (tile / 8) * 32 * 2);
	add((void**)&f->fiy, sizeof(uint4) * (tile / 16) * 2 * 32 * 2);
	add((void**)&f->sx, sizeof(float) * MX);
	for (int l = 1; l < L; l++) add((void**)&f->v[l], sizeof(float) * nv);
	for (int l = 0; l < L - 1; l++) add((void**)&f->z[l], sizeof(float) * nv);
	for (int l = 0; l < L; l++) add((void**)&f->X[l], sizeof(float2) * max_batch * C * NK);
	add((void**)&f->A, sizeof(float2) * max_batch * C * tile * MX);
	add((void**)&f->Y, sizeof(float2) * max_batch * C * NK);
	add((void**)&f->Bq, sizeof(float2) * max_batch * C * tile * MX);
	add((void**)&f->dv, sizeof(float) * nv);
	add((void**)&f->x, sizeof(float) * max_batch * 2 * npix);
	add((void**)&f->y, sizeof(float) * max_batch * 2 * npix);
	add((void**)&f->dy, sizeof(float) * max_batch * 2 * npix);
	add((void**)&f->loss, sizeof(double));
	add((void**)&f->part, sizeof(double) * 2 * MEAN_BLOCKS);
	for (size_t i = 0; i < bufs.size() && e == cudaSuccess; i++) e = cudaMalloc(bufs[i], sizes[i]);
	if (e != cudaSuccess) {
		pfcg_fno_destroy(f);
		return ffail(nullptr, PFCG_ENOMEM, std::string("device allocation: ") + cudaGetErrorString(e));
	}
	float sc[MX];
	for (int m = 0; m < MX; m++) sc[m] = (m == 0 ? 1.f : 2.f) / (float)npix;
	e = cudaMemcpyAsync(f->sx, sc, sizeof(sc), cudaMemcpyHostToDevice, f->stream);
	twiddle_kernel<<<1, 256, 0, f->stream>>>(f->tw, tile);
	dft_frag_kernel<<<(tile * 8 + 255) / 256, 256, 0, f->stream>>>(f->tw, tile, f->fe, f->ff);
	dfty_frag_kernel<<<(tile * 8 + 255) / 256, 256, 0, f->stream>>>(f->tw, tile, f->fdy, f->fiy);
	f->launches += 2;
	for (size_t i = 0; i < 5 && e == cudaSuccess; i++) e = cudaMemsetAsync(*bufs[i], 0, sizes[i], f->stream);
	if (e == cudaSuccess) e = cudaStreamSynchronize(f->stream);
	if (e == cudaSuccess) e = cudaGetLastError();
	if (e != cudaSuccess) {
		pfcg_fno_destroy(f);
		return ffail(nullptr, PFCG_ECUDA, std::string("set-up: ") + cudaGetErrorString(e));
	}
	*out = f;
	return 0;
}

void pfcg_fno_destroy(pfcg_fno* f) {
	if (!f) return;
	if (f->stream) cudaStreamSynchronize(f->stream);
	void* ptrs[] = {f->p, f->w, f->g, f->am, f->av, f->tw, f->sx, f->A, f->Y, f->Bq, f->dv, f->x, f->y, f->dy, f->loss,
	                f->field_tmp, f->part, f->fe, f->ff, f->fdy, f->fiy};
	for (void* q : ptrs) cudaFree(q);
	for (float* q : f->v) cudaFree(q);
	for (float* q : f->z) cudaFree(q);
	for (float2* q : f->X) cudaFree(q);
	if (f->stream) cudaStreamDestroy(f->stream);
	delete f;
}

int pfcg_fno_set_params(pfcg_fno* f, const float* host_params) {
	if (!f || !host_params) return ffail(f, PFCG_EARG, "NULL argument");
	FCK(cudaMemcpyAsync(f->p, host_params, sizeof(float) * NPARAM, cudaMemcpyHostToDevice, f->stream));
	to_bf16<<<grid_for(NPARAM, 256), 256, 0, f->stream>>>(f->p, f->w, NPARAM);
	f->launches++;
	FCK(cudaMemsetAsync(f->am, 0, sizeof(float) * NPARAM, f->stream));
	FCK(cudaMemsetAsync(f->av, 0, sizeof(float) * NPARAM, f->stream));
	f->adam_t = 0;
	FCK(cudaStreamSynchronize(f->stream));
	return 0;
}

int pfcg_fno_get_params(pfcg_fno* f, float* host_params) {
	if (!f || !host_params) return ffail(f, PFCG_EARG, "NULL argument");
	FCK(cudaMemcpyAsync(host_params, f->p, sizeof(float) * NPARAM, cudaMemcpyDeviceToHost, f->stream));
	FCK(cudaStreamSynchronize(f->stream));
	return 0;
}

int pfcg_fno_forward(pfcg_fno* f, const float* d_in, float* d_out, int batch) {
	if (!f || !d_in || !d_out) return ffail(f, PFCG_EARG, "NULL argument");
	if (batch < 1 || batch > f->maxB) return ffail(f, PFCG_EARG, "batch outside [1, max_batch]");
	int rc = forward(f, d_in, batch, nullptr);
	if (rc) return rc;
	FCK(cudaMemcpyAsync(d_out, f->y, sizeof(float) * batch * 2 * f->T * f->T, cudaMemcpyDeviceToDevice, f->stream));
	FCK(cudaStreamSynchronize(f->stream));
	return 0;
}

int pfcg_fno_loss_grad(pfcg_fno* f, const float* d_in, const float* d_target, int batch, double* loss,
                       float* host_grad) {
	if (!f || !d_in || !d_target) return ffail(f, PFCG_EARG, "NULL argument");
	if (batch < 1 || batch > f->maxB) return ffail(f, PFCG_EARG, "batch outside [1, max_batch]");
	int rc = forward(f, d_in, batch, d_target);
	if (!rc) rc = backward(f, d_in, batch);
	if (rc) return rc;
	if (loss) FCK(cudaMemcpyAsync(loss, f->loss, sizeof(double), cudaMemcpyDeviceToHost, f->stream));
	if (host_grad) FCK(cudaMemcpyAsync(host_grad, f->g, sizeof(float) * NPARAM, cudaMemcpyDeviceToHost, f->stream));
	FCK(cudaStreamSynchronize(f->stream));
	return 0;
}

int pfcg_fno_adam_step(pfcg_fno* f, float lr, float beta1, float beta2, float eps) {
	if (!f) return ffail(f, PFCG_EARG, "NULL argument");
	f->adam_t++;
	const float c1 = 1.f - std::pow(beta1, (float)f->adam_t), c2 = 1.f - std::pow(beta2, (float)f->adam_t);
	adam_kernel<<<grid_for(NPARAM, 256), 256, 0, f->stream>>>(f->p, f->g, f->am, f->av, NPARAM, lr, beta1, beta2, eps,
	                                                           c1, c2);
	to_bf16<<<grid_for(NPARAM, 256), 256, 0, f->stream>>>(f->p, f->w, NPARAM);
	f->launches += 2;
	FCK(cudaGetLastError());
	return 0;
}

int pfcg_fno_apply(pfcg_fno* f, const double* d_in, double* d_out, int Nx, int Ny, void* stream) {
	if (!f || !d_in || !d_out) return ffail(f, PFCG_EARG, "NULL argument");
	if (d_in == d_out) return ffail(f, PFCG_EARG, "input and output grids must be distinct");
	if (Nx < 1 || Ny < 1) return ffail(f, PFCG_EARG, "empty grid");
	cudaStream_t st = (cudaStream_t)stream;
	int rc = fno_apply_device(f, d_in, d_out, Nx, Ny, st);
	if (rc) return rc;
	FCK(cudaStreamSynchronize(st));
	return 0;
}

int pfcg_fno_stream(const pfcg_fno* f, void** stream) {
	if (!f || !stream) return PFCG_EARG;
	*stream = (void*)f->stream;
	return 0;
}

int pfcg_fno_launch_count(const pfcg_fno* f, long long* count) {
	if (!f || !count) return PFCG_EARG;
	*count = f->launches;
	return 0;
}

const char* pfcg_fno_last_error(const pfcg_fno* f) { return f ? f->err.c_str() : g_fno_err.c_str(); }

} // extern "C"
