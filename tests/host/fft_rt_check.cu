// Host-side check of the run-time transform plans (pfc_b200/csrc/fft_rt.cuh,
// their __host__ __device__ code compiled for the CPU). For every even 7-smooth
// length from 8 to 8192 and both precisions: a plan exists exactly where the
// pass rule of include/pfc_b200.h admits the length, its radices multiply to the
// length, the reciprocal divisions are exact over every index used, the strided
// addresses equal the padded index of the element they stand for, and the
// transform that the passes compute in order equals a direct one (spot checks
// of four outputs against FP64 sums). Prints a summary and exits non-zero on
// any failure.
#include "../../pfc_b200/csrc/fft_rt.cuh"

#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <vector>

using namespace pfcg;

static long failures = 0, lengths = 0, refused = 0;

// the length rule: N/r <= 512 * floor(16/r) for the radices of N's factors
static bool admitted(int n) {
	int m = n, k2 = 0;
	while (m % 2 == 0) { m /= 2; k2++; }
	bool f[3] = {m % 3 == 0, m % 5 == 0, m % 7 == 0};
	const int rad[3] = {3, 5, 7};
	auto ok = [&](int r) { return (n / r + 16 / r - 1) / (16 / r) <= 512; };
	if (k2 >= 4 && !ok(16)) return false;
	if (k2 % 4 && !ok(1 << (k2 % 4))) return false;
	for (int i = 0; i < 3; i++)
		if (f[i] && !ok(rad[i])) return false;
	return true;
}

template <int R, typename T> static void run_pass(std::vector<cplx<T>>& buf, const FftPlan& pl, const RtPass& q, const std::vector<cplx<T>>& tw) {
	std::vector<cplx<T>> out(buf.size());
	for (int j = 0; j < q.nr; j++) {
		cplx<T> v[R];
		for (int r = 0; r < R; r++) {
			const int at = rt_pad(j, pl.sh) + r * q.sin;
			if (at != rt_pad(j + r * q.nr, pl.sh)) { failures++; return; }
			v[r] = buf[at];
		}
		int jm, d;
		rt_place(R, q.ns, q.mns, j, jm, d);
		const int jd = j / q.ns;
		if (jm != j % q.ns || d != jd * q.ns * R + jm) { failures++; return; }
		rt_butterfly<R, T>(v, tw.data() + q.two + jm, q.ns, q.ns > 1);
		for (int r = 0; r < R; r++) {
			const int at = rt_pad(d, pl.sh) + r * q.sout + (R == 16 && r >= 8 ? q.sx : 0);
			if (at != rt_pad(d + r * q.ns, pl.sh) || at >= pl.ld) { failures++; return; }
			out[at] = v[r];
		}
	}
	buf.swap(out);
}

template <typename T> static void check(int n, int max_radix) {
	const bool fp64 = sizeof(T) == 8;
	FftPlan pl;
	const bool have = rt_make_plan(n, fp64, 512, max_radix, &pl);
	if (have != admitted(n) && max_radix == 16) {
		failures++;
		std::printf("length %d: plan %d, rule %d\n", n, have, admitted(n));
	}
	if (!have) { refused++; return; }
	lengths++;
	long prod = 1;
	for (int s = 0; s < pl.npass; s++) {
		const RtPass& q = pl.p[s];
		if (q.ns != prod || q.nr != n / q.r) failures++;
		prod *= q.r;
		// four sequences' worth of butterflies, as the largest row tile has
		for (int b = 0; b < 8 * q.nr && b < 16384; b++)
			if (rt_div(b, q.mnr) != b / q.nr) { failures++; break; }
	}
	for (int e = 0; e < 8 * n; e++)
		if (rt_div(e, pl.mn) != e / n || rt_div(e, pl.mnh) != e / (n / 2)) { failures++; break; }
	if (prod != n || pl.npass > RT_MAXP || rt_plan_threads(pl, 1) > 512) failures++;
	std::vector<cplx<T>> tw(pl.ntw + 1);
	if (pl.ntw >= n) failures++; // the caller's table holds n entries
	for (int i = 0; i < pl.ntw; i++) {
		int num, den;
		rt_twiddle_of(pl, fp64, i, &num, &den);
		tw[i] = mk<T>((T)std::cos(-2.0 * M_PI * num / den), (T)std::sin(-2.0 * M_PI * num / den));
	}
	std::vector<cplx<T>> buf(pl.ld), x(n);
	for (int i = 0; i < n; i++) {
		x[i] = mk<T>((T)std::sin(1.3 * i + 0.2), (T)std::cos(0.7 * i * (i % 97) + 1.0));
		buf[rt_pad(i, pl.sh)] = x[i];
	}
	for (int s = 0; s < pl.npass; s++) {
		const RtPass& q = pl.p[s];
		switch (q.r) {
		case 16: run_pass<16, T>(buf, pl, q, tw); break;
		case 15: run_pass<15, T>(buf, pl, q, tw); break;
		case 14: run_pass<14, T>(buf, pl, q, tw); break;
		case 12: run_pass<12, T>(buf, pl, q, tw); break;
		case 10: run_pass<10, T>(buf, pl, q, tw); break;
		case 9: run_pass<9, T>(buf, pl, q, tw); break;
		case 8: run_pass<8, T>(buf, pl, q, tw); break;
		case 7: run_pass<7, T>(buf, pl, q, tw); break;
		case 6: run_pass<6, T>(buf, pl, q, tw); break;
		case 5: run_pass<5, T>(buf, pl, q, tw); break;
		case 4: run_pass<4, T>(buf, pl, q, tw); break;
		case 3: run_pass<3, T>(buf, pl, q, tw); break;
		case 2: run_pass<2, T>(buf, pl, q, tw); break;
		default: failures++;
		}
	}
	// each stage multiplies the values by about sqrt(radix) and adds its roundings
	const double tol = (fp64 ? 2.3e-16 : 1.2e-7) * 8 * pl.npass * std::sqrt((double)n) + (fp64 ? 1e-16 * n : 0);
	const int ks[4] = {0, 1, n / 2 + 3 < n ? n / 2 + 3 : 2, n - 1};
	for (int c = 0; c < 4; c++) {
		double re = 0, im = 0;
		for (int i = 0; i < n; i++) {
			const double a = -2.0 * M_PI * (double)((long)i * ks[c] % n) / n;
			re += (double)x[i].x * std::cos(a) - (double)x[i].y * std::sin(a);
			im += (double)x[i].x * std::sin(a) + (double)x[i].y * std::cos(a);
		}
		const cplx<T> g = buf[rt_pad(ks[c], pl.sh)];
		const double err = std::hypot(g.x - re, g.y - im);
		if (err > tol) {
			failures++;
			std::printf("length %d output %d: error %.2e above %.2e\n", n, ks[c], err, tol);
		}
	}
}

int main(int argc, char** argv) {
	const int show = argc > 1 ? std::atoi(argv[1]) : 0;
	if (show) {
		for (int f = 0; f < 2; f++) {
			FftPlan pl;
			if (!rt_make_plan(show, f, 512, argc > 2 ? std::atoi(argv[2]) : 16, &pl)) continue;
			std::printf("%s sh %d ld %d ntw %d:", f ? "fp64" : "fp32", pl.sh, pl.ld, pl.ntw);
			for (int s = 0; s < pl.npass; s++) std::printf(" %d", pl.p[s].r);
			std::printf("\n");
		}
		return 0;
	}
	for (int n = 8; n <= 8192; n += 2) {
		int m = n;
		for (int f : {2, 3, 5, 7})
			while (m % f == 0) m /= f;
		if (m != 1) continue;
		check<float>(n, 16);
		check<double>(n, 16);
	}
	std::printf("%ld plans, %ld refused, %ld failures\n", lengths, refused, failures);
	return failures ? 1 : 0;
}
