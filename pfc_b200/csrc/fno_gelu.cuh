// GELU and its derivative for the warm-start network (fno.cu).
#pragma once

namespace pfcg {

// The normal distribution's lower tail at -u and the density's exponential, u = |z|:
// Phi(-u) = exp(-u^2 / 2) R(u), and R(u) = t Q(t) with t = 1 / (1 + 0.21 u) and Q of
// degree 8, fitted here by iteratively reweighted least squares to 1.4e-8 relative over
// u < 13.5, beyond which both are zero in FP32. GELU from it is within 2.4e-7 of FP64 on
// [-9, 9] (rms 4.7e-8), from erff 4.5e-7 (6.3e-8), in 17 instructions and two
// special-function ones instead of about 22; the derivative shares both parts. GELU was
// half of a layer's instructions.
// The special values are those of 0.5 z (1 + erf(z / sqrt 2)): GELU(inf) = inf, for which u
// is clamped where the tail is zero, and GELU(-inf) = NaN, so that a network that has
// overflowed cannot look finite; the derivative is NaN at both, and without the clamp
// (training iteration 4.8 ms, 5.7 with it in the derivative as well).
struct Tail {
	float u, phi, e;
	__device__ __forceinline__ Tail(float z, bool clamp) {
		float t;
		u = clamp ? fminf(fabsf(z), 20.f) : fabsf(z);
		asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(t) : "f"(fmaf(0.21f, u, 1.f)));
		asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(-0.72134752f * u * u));
		float q = -0.07203336f;
		q = fmaf(q, t, 0.28545034f);
		q = fmaf(q, t, -0.33418325f);
		q = fmaf(q, t, 0.35402617f);
		q = fmaf(q, t, -0.097240396f);
		q = fmaf(q, t, 0.1263528f);
		q = fmaf(q, t, 0.068790667f);
		q = fmaf(q, t, 0.085129313f);
		q = fmaf(q, t, 0.083707705f);
		phi = q * t * e;
	}
};
__device__ __forceinline__ float gelu(float z) {
	const Tail p(z, true);
	const float h = 0.5f * z, r = h + fabsf(h); // max(z, 0); NaN at -inf
	return fmaf(-p.u, p.phi, r);
}
__device__ __forceinline__ float gelu_d(float z) {
	const Tail p(z, false);
	return fmaf(z * 0.39894228040143268f, p.e, z < 0.f ? p.phi : 1.f - p.phi);
}

} // namespace pfcg
