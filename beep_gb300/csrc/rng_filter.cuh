// The FP64 form's keyed Poisson and binomial draws (rng_fp64.cuh) at FP32 cost.
//
// GB300 issues one FP64 warp instruction per SM every 16 cycles, and an FP64
// draw is a few hundred of them: the samplers kept the FP64 pipe of the plain
// form 82% busy.  A draw is an integer, though, and every comparison that
// decides it is between numbers that are rarely close.  These functions
// evaluate the same recipe (same Philox counters and words, same accept and
// reject regions) in FP32, each comparison with a bound on how far the FP32
// value and the FP64 form's own rounded value can be apart; a draw with a
// comparison inside its bound is redone by the FP64 function.  The result is
// the FP64 function's in every case.  Words of the stream are compared as the
// 32-bit integers they are; a count's integer part is split off the FP64 mean
// exactly, so the bounds do not grow with the mean's magnitude.
//
// Bounds, with e = 2^-24 (conversions round to nearest; expf and log1pf within
// 2 ulp, __fdividef within 2 ulp, __logf as documented):
//   inversion     |F32_k - F64_k| <= 5e-7 + 4e-7 mean + 4e-8 k: the argument of exp
//                 carries mean*e, a term 4 roundings (4e each, so 4e * sum j p_j <= 4e mean),
//                 an addition to F < 1 half an ulp; u's own rounding is in the constant.
//                 Binomial: 1e-6 + 1.3e-6 nq + 4e-8 k (7 roundings per term, and n times
//                 the rounding of 1 - q in FP64).
//   PTRS / BTRS k  the offset (2a/us + b) U is a sum of positive terms: 1e-6 relative,
//                 bounded by 1.5e-6 (2e-6) of it plus 2e-6 for the fraction of the mean.
//   vr            2e-6 absolute
//   acceptance    1e-4 + 2e-6 |d| (4e-6 |d|) + 1e-6 |rhs|, d = mean - (k+1) or k - m, with
//                 the density written without cancellation (as the fast form's), its log Gamma
//                 remainders within 5e-6 (stirling_rem_f32).
// tests/test_filtered_draws.py puts 1e6 draws at the places where a decision turns.
// Redone draws: 1 in 11,000 at means of 1 to 10, 1 in 3,000 at 10 to 1000, 1 in 1,000 up to 1e5,
// 1 in 130 up to 1e7.  Per draw and SM: 26 -> 1.1 ns at mean 1, 255 -> 5.4 ns at 20, 137 -> 11 ns
// at 1e5 (2.5e8 draws over means 1e-6 to 1e9, and as many binomials, equal to the FP64 ones).
#pragma once

#include <cstdint>

#include "rng_fp64.cuh"

namespace beep {

// 1/k (k = 1..64, at [k-1]) and log k! (k < 16): shared memory of the CTA
struct __align__(16) FilterTab {
	float rcp[64];
	float lnfact[16];
};

__device__ __forceinline__ void filter_tab_fill(FilterTab &t, int tid, int nth)
{
	for (int k = tid; k < 64; k += nth) t.rcp[k] = __fdiv_rn(1.f, (float)(k + 1));
	for (int k = tid; k < 16; k += nth) {
		float f = 0.f;
		for (int j = 2; j <= k; j++) f += logf((float)j);
		t.lnfact[k] = f;
	}
}

// FP32 of a positive finite double below 2^127, rounded to nearest (0 below 2^-126), on the integer pipe
__device__ __forceinline__ float f32_of_pos(double x)
{
	const uint32_t hi = (uint32_t)__double2hiint(x), lo = (uint32_t)__double2loint(x);
	if (hi < 0x38100000u) return 0.f;
	return __uint_as_float((((hi - 0x38000000u) << 3) | (lo >> 29)) + ((lo >> 28) & 1u));
}

// x in [0, 2^31): integer part (exact) and fraction
__device__ __forceinline__ int32_t split_pos(double x, float &frac)
{
	const uint32_t hi = (uint32_t)__double2hiint(x), lo = (uint32_t)__double2loint(x);
	const int e = (int)(hi >> 20) - 1023;
	if (e < 0) {
		frac = f32_of_pos(x);
		return 0;
	}
	const uint64_t mant = ((uint64_t)((hi & 0xfffffu) | 0x100000u) << 32) | lo;
	frac = __uint2float_rn((uint32_t)((mant << (12 + e)) >> 32)) * 2.3283064365386963e-10f;
	return (int32_t)(mant >> (52 - e));
}

__device__ __forceinline__ float u01_f32(uint32_t w)
{
	return fmaf(__uint2float_rn(w), 2.3283064365386963e-10f, 1.1641532182693481e-10f);
}

// u - 0.5 of a word, to 32-bit relative accuracy also near 0
__device__ __forceinline__ float u_minus_half_f32(uint32_t w)
{
	return fmaf(__int2float_rn((int32_t)(w ^ 0x80000000u)), 2.3283064365386963e-10f, 1.1641532182693481e-10f);
}

// us = 0.5 - |u - 0.5| of a word, as the word w' with us = (w' + 1/2) 2^-32
__device__ __forceinline__ uint32_t us_word(uint32_t w) { return (int32_t)w < 0 ? ~w : w; }
constexpr uint32_t kUs07 = 300647711u;    // us >= 0.07   <=>  w' >= this
constexpr uint32_t kUs013 = 55834574u;    // us < 0.013   <=>  w' <= this

// Search of the CDF for u from F = p at k = 0, terms p * next(k); -2 when a comparison is
// closer than bound0 + bound1 k or the search runs on (u in the far tail).  Four terms per
// pass: one branch and one vector load of 1/k for the four.
template <typename Next>
__device__ __forceinline__ int32_t search_cdf(float u, float p, float bound0, float bound1, const FilterTab &t, Next next)
{
	float F0 = p;
	if (u <= F0) return F0 - u > bound0 ? 0 : -2;
	for (int32_t k = 0; k < 56; k += 4) {
		const float4 r = *reinterpret_cast<const float4 *>(t.rcp + k);
		const float p1 = next(p, k) * r.x, F1 = F0 + p1;
		const float p2 = next(p1, k + 1) * r.y, F2 = F1 + p2;
		const float p3 = next(p2, k + 2) * r.z, F3 = F2 + p3;
		const float p4 = next(p3, k + 3) * r.w, F4 = F3 + p4;
		if (u <= F4) {
			const float near = fminf(fminf(fminf(fabsf(u - F0), fabsf(u - F1)), fminf(fabsf(u - F2), fabsf(u - F3))), F4 - u);
			if (!(near > fmaf(bound1, (float)k + 4.f, bound0))) return -2;
			return k + 1 + (u > F1) + (u > F2) + (u > F3);
		}
		p = p4;
		F0 = F4;
	}
	return -2;
}

// poisson_fp64's draw (mean > 0).  Beyond 1e9, which only the difference from a negative current mean
// reaches, by the FP64 function: the integer part is kept in 32 bits here.
__device__ __forceinline__ int32_t poisson_filtered(double mean, uint32_t k0, uint32_t k1, uint32_t col, uint32_t tr,
                                                    uint32_t sett, uint32_t stream, uint32_t limit, const FilterTab &t)
{
	const float mf = f32_of_pos(mean);
	if (__double_as_longlong(mean) < 0x4024000000000000ll) {           // mean < 10
		const U4 r = philox10(U4{col, sett, stream, (PURPOSE_INV << 24) | (tr >> 2)}, k0, k1);
		const float u = u01_f32(word_of(r, tr & 3u));
		const int32_t k = search_cdf(u, expf(-mf), fmaf(4e-7f, mf, 5e-7f), 4e-8f, t,
		                             [mf](float p, int32_t) { return p * mf; });
		return k >= 0 ? k : poisson_fp64(mean, k0, k1, col, tr, sett, stream, limit);
	}
	if (__double_as_longlong(mean) > __double_as_longlong(1e9)) return poisson_fp64(mean, k0, k1, col, tr, sett, stream, limit);
	float frac;
	const int32_t whole = split_pos(mean, frac);
	const float b = fmaf(2.53f, __fsqrt_rn(mf), 0.931f);
	const float a = fmaf(0.02483f, b, -0.059f);
	const float vr = 0.9277f - __fdividef(3.6224f, b - 2.0f);
	for (uint32_t it = 0; it < limit; it++) {
		const U4 r = philox10(U4{col, sett, stream, (PURPOSE_PTRS << 24) | (tr << 16) | it}, k0, k1);
		const uint32_t w = us_word(r.x);
		if (w <= kUs013 && r.y > w) continue;                            // us < 0.013 and V > us
		const float us = u01_f32(w), U = u_minus_half_f32(r.x), V = u01_f32(r.y);
		const float off = (__fdividef(2.0f * a, us) + b) * U;
		const float x = frac + 0.43f + off, fl = floorf(x), xf = x - fl;
		const float bk = fmaf(1.5e-6f, fabsf(off), 2e-6f);
		if (!(fabsf(off) < 4e6f) || xf < bk || xf > 1.f - bk) break;       // k not certain
		const int32_t j = (int32_t)fl, k = whole + j;
		if (w >= kUs07) {
			if (V < vr - 2e-6f) return k;
			if (!(V > vr + 2e-6f)) break;
		}
		if (k < 0) continue;
		const float lhs = __logf(__fdividef(V * (1.1239f + __fdividef(1.1328f, b - 3.4f)), __fdividef(a, us * us) + b));
		float rhs, d = 0.f;
		if (k < 10) rhs = fmaf((float)k, __logf(mf), -mf) - t.lnfact[k];
		else {
			const float n = (float)(k + 1), in = __fdividef(1.f, n), in2 = in * in;
			d = frac - (float)(j + 1);                                     // mean - n
			const float z = d * in;
			const float corr = in * (0.083333333f - in2 * (0.0027777778f - in2 * 0.00079365079f));
			rhs = (float)k * (log1pf(z) - z) - z - 0.5f * __logf(n) - 0.91893853f - corr;
		}
		const float gap = lhs - rhs, bound = 1e-4f + 2e-6f * fabsf(d) + 1e-6f * fabsf(rhs);
		if (gap < -bound) return k;
		if (!(gap > bound)) break;
	}
	return poisson_fp64(mean, k0, k1, col, tr, sett, stream, limit);   // an uncertain comparison (or `limit` rejections)
}

// log Gamma(z) - ((z - 1/2) log z - z + log(2 pi)/2) of an integer z: three terms of the series, off
// by less than the first one omitted, 1 / (1680 z^7) <= 5e-6, from z = 2 on; at z = 1 (a candidate of
// 0 or of n) they would be 2.9e-4 off, so the value itself stands there, 1 - log(2 pi)/2
__device__ __forceinline__ float stirling_rem_f32(float z)
{
	const float iz = __fdividef(1.f, z), iz2 = iz * iz;
	return z < 1.5f ? 0.081061467f : iz * (0.083333333f - iz2 * (0.0027777778f - iz2 * 0.00079365079f));
}

// binomial_fp64's draw
__device__ __forceinline__ int32_t binomial_filtered(double p, int32_t n, uint32_t k0, uint32_t k1, uint32_t col,
                                                     uint32_t tr, uint32_t sett, uint32_t stream, uint32_t limit,
                                                     const FilterTab &t)
{
	if (n <= 0 || !(p > 0.0)) return 0;
	if (p >= 1.0) return n;
	const bool flip = p > 0.5;
	const double q = flip ? 1.0 - p : p;
	const double nd = (double)n, nq = nd * q;
	const float qf = f32_of_pos(q), qc = 1.f - qf, nqf = f32_of_pos(nq);
	int32_t k = -2;
	if (nq < 10.0) {
		const U4 r = philox10(U4{col, sett, stream, (PURPOSE_THIN << 24) | (tr >> 2)}, k0, k1);
		const float u = u01_f32(word_of(r, tr & 3u));
		const float ratio = __fdiv_rn(qf, qc);
		k = search_cdf(u, expf((float)n * log1pf(-qf)), fmaf(1.3e-6f, nqf, 1e-6f), 4e-8f, t,
		               [ratio, n](float f, int32_t j) { return f * ratio * (float)max(n - j, 0); });
	} else {
		float frac;
		const int32_t whole = split_pos(nq, frac);
		const float spq = __fsqrt_rn(nqf * qc);
		const float b = fmaf(2.53f, spq, 1.15f);
		const float a = fmaf(0.0248f, b, -0.0873f) + 0.01f * qf;
		const float vr = 0.92f - __fdividef(4.2f, b);
		for (uint32_t it = 0; it < limit; it++) {
			const U4 r = philox10(U4{col, sett, stream, (PURPOSE_BTRS << 24) | (tr << 16) | it}, k0, k1);
			const uint32_t w = us_word(r.x);
			const float us = u01_f32(w), U = u_minus_half_f32(r.x), V = u01_f32(r.y);
			const float off = (__fdividef(2.f * a, us) + b) * U;
			const float x = frac + 0.5f + off, fl = floorf(x), xf = x - fl;
			const float bk = fmaf(2e-6f, fabsf(off), 2e-6f);
			if (!(fabsf(off) < 4e6f) || xf < bk || xf > 1.f - bk) break;   // k not certain
			const int32_t kd = whole + (int32_t)fl;
			if (kd < 0 || kd > n) continue;
			if (w >= kUs07) {
				if (V < vr - 2e-6f) { k = kd; break; }
				if (!(V > vr + 2e-6f)) break;
			}
			float mfrac;
			const int32_t m = split_pos((nd + 1.0) * q, mfrac);
			const float alpha = (2.83f + __fdividef(5.1f, b)) * spq;
			const float lhs = __logf(__fdividef(V * alpha, __fdividef(a, us * us) + b));
			const float d = (float)(kd - m), m1 = (float)m + 1.f, nm1 = (float)(n - m) + 1.f;
			const float k1f = (float)kd + 1.f, nk1 = (float)(n - kd) + 1.f;
			const float rhs = -(m1 - 0.5f) * log1pf(d / m1) - (nm1 - 0.5f) * log1pf(-d / nm1) +
			                  d * __logf(nk1 * qf / (k1f * qc)) + stirling_rem_f32(m1) + stirling_rem_f32(nm1) -
			                  stirling_rem_f32(k1f) - stirling_rem_f32(nk1);
			const float gap = lhs - rhs, bound = 1e-4f + 4e-6f * fabsf(d) + 1e-6f * fabsf(rhs);
			if (gap < -bound) { k = kd; break; }
			if (!(gap > bound)) break;
		}
	}
	if (k < 0) return binomial_fp64(p, n, k0, k1, col, tr, sett, stream, limit);
	return flip ? n - k : k;
}

}  // namespace beep
