// beep_abcsmc_weights: ABC-SMC importance weights of a generation
// (ABCSMC::calculate_particle_weight, src/abcsmc.cc:260-271, with
// MVN::probability, src/mvn.cc:185-196, and normalise_particle_weights,
// src/abcsmc.cc:275-283):
//   w_i = exp(logprior_i) / sum_j w_j^last exp(-0.5 (d/size)^T M^-1 (d/size)),
//   d = theta_i - theta_j over the inferred parameters; then w /= mean(w).
//
// The quadratic form is evaluated as a sum of squares: with the Cholesky
// factor L of M^-1 / size^2 (= L L^T, FP64 on the host) every particle is
// mapped to z = L^T (theta - mean of the last generation), and
// q_ij = |z_i - z_j|^2 -- no cancellation between positive and negative
// terms of the form, whatever the correlations (centring removes any large
// common offset).  A matrix that is not positive definite (the reference
// inverts whatever sample covariance it has, singular or not) is used as
// given: q_ij = d^T A d on the centred parameters, as the reference does.
// Each new particle's sum  sum_j w_j exp(-q_ij / 2)  is accumulated as a
// running log-sum-exp -- the largest exponent so far and the compensated sum
// of exp(x_j - max) -- so it cannot underflow.
//   pass 1  FP32 differences and sums, one thread per new particle;
//   pass 2  FP64, for the new particles whose nearest previous particles are
//           far (largest term below exp(-10) of the heaviest previous
//           weight): there the FP32 rounding of q (a few 1e-8 of q) would
//           reach the 1e-6 level in exp(-q/2).
// The log sums, the prior factor and the normalisation (relative to the
// largest weight, so nothing overflows) are FP64.  Where the reference's FP64
// sum underflows to zero (its weight is then infinite) this one stays finite.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "capi_internal.h"

namespace beep {
namespace {

constexpr int kAbcThreads = 32;      // new particles per CTA
constexpr int kAbcTile = 256;        // last-generation particles staged per pass
constexpr int kAbcGroup = 8;         // terms in flight per thread
constexpr int kFarThreads = 256;     // threads of the FP64 pass, per new particle
constexpr int kMaxVar = 16;
constexpr double kFarExponent = 10.0;

// q of a difference d: |d|^2 (whitened coordinates) or d^T A d (A row-major nvar x nvar)
template <bool WHITE, typename R>
__device__ __forceinline__ R quad_form(const R *d, const R *A, int nvar)
{
	R q = 0;
	if (WHITE) {
#pragma unroll
		for (int v = 0; v < kMaxVar; v++)
			if (v < nvar) q = fma(d[v], d[v], q);
	} else {
#pragma unroll
		for (int v1 = 0; v1 < kMaxVar; v1++) {
			if (v1 < nvar) {
				R r = 0;
#pragma unroll
				for (int v2 = 0; v2 < kMaxVar; v2++)
					if (v2 < nvar) r = fma(A[v1 * nvar + v2], d[v2], r);
				q = fma(d[v1], r, q);
			}
		}
	}
	return q;
}

// Pass 1.  A new particle's terms enter its running log-sum-exp one after another (the
// running maximum and the compensated sum depend on their order), so a thread owns a new
// particle and the bound is the latency of its chain of sums: four dependent additions per
// term.  What feeds the chain is taken off it -- kAbcGroup terms' forms and exponentials are
// in flight at once, a previous particle (its coordinates and log weight, padded to 16 bytes)
// loads as one or a few vectors, and only a group that raises the maximum (a handful per
// particle) or holds a weight of zero goes term by term.  CTAs of one warp put a warp on
// every scheduler from 608 x 32 new particles.  16384 x 16384, 3 parameters: 3.73 ms as 64
// CTAs of 256 threads, one term at a time with predicated loops over 16 parameters;
// 0.56 ms now (71 cycles per term and warp, 29 instructions).
// NV: the parameters, or 0 for a count only known at run time.
template <bool WHITE, int NV>
__global__ void __launch_bounds__(kAbcThreads) abc_logsums_f32(int nvar_, int nnew, const float *z_new, int nlast,
                                                               const float *z_last, const float *logw_last,
                                                               const float *A, double *logsum_out, float *max_out)
{
	constexpr int kV = NV > 0 ? NV : kMaxVar, kStride = (kV + 1 + 3) & ~3;
	__shared__ float4 s_zw[kAbcTile * kStride / 4];      // per previous particle: coordinates, log weight
	__shared__ float s_A[kMaxVar * kMaxVar];
	const int nvar = NV > 0 ? NV : nvar_;
	const int i = blockIdx.x * kAbcThreads + threadIdx.x;
	float *zw = reinterpret_cast<float *>(s_zw);
	if (!WHITE)
		for (int k = threadIdx.x; k < nvar * nvar; k += kAbcThreads) s_A[k] = A[k];
	float x[kV];
#pragma unroll
	for (int v = 0; v < kV; v++) x[v] = (i < nnew && v < nvar) ? z_new[(size_t)i * nvar + v] : 0.f;
	float mx = -INFINITY, s = 0.f, cmp = 0.f;      // running max exponent; compensated sum of exp(x_j - mx)
	auto exponent = [&](int j) {
		float d[kMaxVar], q4[kStride];
#pragma unroll
		for (int k = 0; k < kStride / 4; k++) *reinterpret_cast<float4 *>(q4 + 4 * k) = s_zw[j * (kStride / 4) + k];
#pragma unroll
		for (int v = 0; v < kMaxVar; v++) d[v] = v < kV && v < nvar ? x[v < kV ? v : 0] - q4[v < kV ? v : 0] : 0.f;
		return q4[kV] - 0.5f * quad_form<WHITE>(d, s_A, nvar);
	};
	auto add = [&](float term) {
		const float y = term - cmp;                  // Kahan
		const float t = s + y;
		cmp = (t - s) - y;
		s = t;
	};
	auto one = [&](float xe) {
		if (xe == -INFINITY) return;                 // a previous particle of weight zero
		if (xe > mx) {                               // new largest exponent: rescale the sum
			const float f = expf(mx - xe);
			s *= f;
			cmp *= f;
			mx = xe;
		}
		add(expf(xe - mx));
	};
	for (int j0 = 0; j0 < nlast; j0 += kAbcTile) {
		const int nj = min(kAbcTile, nlast - j0);
		__syncthreads();
		for (int k = threadIdx.x; k < nj * nvar; k += kAbcThreads) zw[k / nvar * kStride + k % nvar] = z_last[(size_t)j0 * nvar + k];
		for (int k = threadIdx.x; k < nj; k += kAbcThreads) zw[k * kStride + kV] = logw_last[j0 + k];
		__syncthreads();
		if (i >= nnew) continue;
		// the next group's exponents are formed beside this group's chain
		const int ng = nj / kAbcGroup;
		float xe[kAbcGroup], xn[kAbcGroup];
		auto form = [&](float *to, int g) {
#pragma unroll
			for (int u = 0; u < kAbcGroup; u++) to[u] = exponent(g * kAbcGroup + u);
		};
		if (ng > 0) form(xn, 0);
		for (int g = 0; g < ng; g++) {
			const int gn = min(g + 1, ng - 1);
			float hi = xn[0], lo = xn[0];
#pragma unroll
			for (int u = 0; u < kAbcGroup; u++) {
				xe[u] = xn[u];
				hi = fmaxf(hi, xn[u]);
				lo = fminf(lo, xn[u]);
			}
			if (hi <= mx && lo > -INFINITY) {
				float ex[kAbcGroup];
#pragma unroll
				for (int u = 0; u < kAbcGroup; u++) ex[u] = expf(xe[u] - mx);
				form(xn, gn);
#pragma unroll
				for (int u = 0; u < kAbcGroup; u++) add(ex[u]);
			} else {
				form(xn, gn);
#pragma unroll 1
				for (int u = 0; u < kAbcGroup; u++) {
					float v = xe[0];
#pragma unroll
					for (int w = 1; w < kAbcGroup; w++) v = u == w ? xe[w] : v;
					one(v);
				}
			}
		}
		int j = ng * kAbcGroup;
		for (; j < nj; j++) one(exponent(j));
	}
	if (i < nnew) {
		logsum_out[i] = (double)mx + log((double)s - (double)cmp);
		max_out[i] = mx;
	}
}

// Pass 2: FP64 log sums of the listed new particles, a CTA each (the FP64 pipe issues one
// warp instruction per 64 cycles and scheduler: one thread per particle took 26 ms for any
// number of them at 16384 previous particles)
template <bool WHITE>
__global__ void __launch_bounds__(kFarThreads) abc_logsums_f64(int nvar, const int *far_idx, const double *z_new,
                                                               int nlast, const double *z_last,
                                                               const double *logw_last, const double *A,
                                                               double *logsum_out)
{
	__shared__ double s_m[kFarThreads], s_s[kFarThreads];
	const int i = far_idx[blockIdx.x], tid = threadIdx.x;
	double x[kMaxVar];
#pragma unroll
	for (int v = 0; v < kMaxVar; v++) x[v] = v < nvar ? z_new[(size_t)i * nvar + v] : 0.0;
	double mx = -INFINITY, s = 0.0;
	for (int j = tid; j < nlast; j += kFarThreads) {
		const double lw = logw_last[j];
		if (lw == -INFINITY) continue;
		double d[kMaxVar];
#pragma unroll
		for (int v = 0; v < kMaxVar; v++) d[v] = v < nvar ? x[v] - z_last[(size_t)j * nvar + v] : 0.0;
		const double xe = lw - 0.5 * quad_form<WHITE>(d, A, nvar);
		if (xe > mx) {
			s *= exp(mx - xe);
			mx = xe;
		}
		s += exp(xe - mx);
	}
	s_m[tid] = mx;
	s_s[tid] = s;
	for (int o = kFarThreads / 2; o > 0; o >>= 1) {
		__syncthreads();
		if (tid >= o) continue;
		const double m2 = s_m[tid + o], s2 = s_s[tid + o];
		if (m2 > s_m[tid]) {
			s_s[tid] = s_s[tid] * exp(s_m[tid] - m2) + s2;
			s_m[tid] = m2;
		} else if (m2 > -INFINITY) {
			s_s[tid] += s2 * exp(m2 - s_m[tid]);
		} else {
			s_s[tid] += s2;                            // no term, or NaN
		}
	}
	if (tid == 0) logsum_out[i] = s_m[0] + log(s_s[0]);
}

using LogSums32 = void (*)(int, int, const float *, int, const float *, const float *, const float *, double *, float *);

template <bool WHITE>
LogSums32 pick_logsums(int nvar)
{
	switch (nvar) {
	case 1: return abc_logsums_f32<WHITE, 1>;
	case 2: return abc_logsums_f32<WHITE, 2>;
	case 3: return abc_logsums_f32<WHITE, 3>;
	case 4: return abc_logsums_f32<WHITE, 4>;
	case 5: return abc_logsums_f32<WHITE, 5>;
	case 6: return abc_logsums_f32<WHITE, 6>;
	case 7: return abc_logsums_f32<WHITE, 7>;
	default: return abc_logsums_f32<WHITE, 0>;
	}
}

// L with A = L L^T (A symmetric positive definite, row-major n x n); false otherwise
bool cholesky(int n, const std::vector<double> &A, std::vector<double> &L)
{
	L.assign((size_t)n * n, 0.0);
	for (int i = 0; i < n; i++)
		for (int j = 0; j <= i; j++) {
			double s = A[(size_t)i * n + j];
			for (int k = 0; k < j; k++) s -= L[(size_t)i * n + k] * L[(size_t)j * n + k];
			if (i == j) {
				if (!(s > 0.0)) return false;
				L[(size_t)i * n + i] = std::sqrt(s);
			} else {
				L[(size_t)i * n + j] = s / L[(size_t)j * n + j];
			}
		}
	return true;
}

}  // namespace
}  // namespace beep

using namespace beep;

extern "C" BEEP_API beep_status beep_abcsmc_weights(int32_t nvar, int32_t nnew, const double *theta_new,
                                                    const double *logprior_new, int32_t nlast,
                                                    const double *theta_last, const double *w_last,
                                                    const double *inv_cov, double size, int32_t normalise,
                                                    double *w_out)
{
	if (nvar <= 0 || nvar > kMaxVar || nnew <= 0 || nlast <= 0 || !theta_new || !logprior_new || !theta_last ||
	    !w_last || !inv_cov || !w_out || !(size > 0))
		return fail(BEEP_BAD_INPUT, "abcsmc weights: bad arguments (nvar must be 1..16, size > 0)");
	int dev = 0;
	CUDA_TRY(cudaGetDevice(&dev));
	// (d/size)^T M^-1 (d/size) = |L^T d|^2 with L L^T = M^-1 / size^2
	std::vector<double> Am((size_t)nvar * nvar), Lc;
	for (int i = 0; i < nvar; i++)
		for (int j = 0; j < nvar; j++)   // the symmetric part (the form only sees it)
			Am[(size_t)i * nvar + j] = 0.5 * (inv_cov[i * nvar + j] + inv_cov[j * nvar + i]) / (size * size);
	const bool white = cholesky(nvar, Am, Lc);
	if (!white) {                                  // the form as given, on centred parameters
		Lc.assign((size_t)nvar * nvar, 0.0);
		for (int v = 0; v < nvar; v++) Lc[(size_t)v * nvar + v] = 1.0;
	}
	std::vector<float> Af(Am.begin(), Am.end());
	std::vector<double> mean(nvar, 0.0);
	for (int j = 0; j < nlast; j++)
		for (int v = 0; v < nvar; v++) mean[v] += theta_last[(size_t)j * nvar + v];
	for (int v = 0; v < nvar; v++) mean[v] /= nlast;
	auto whiten = [&](const double *th, int n, std::vector<double> &z64, std::vector<float> &z32) {
		z64.assign((size_t)n * nvar, 0.0);
		z32.resize((size_t)n * nvar);
		for (int i = 0; i < n; i++)
			for (int k = 0; k < nvar; k++) {
				double s = 0.0;
				for (int v = k; v < nvar; v++) s += Lc[(size_t)v * nvar + k] * (th[(size_t)i * nvar + v] - mean[v]);
				z64[(size_t)i * nvar + k] = s;
				z32[(size_t)i * nvar + k] = (float)s;
			}
	};
	std::vector<double> zn64, zl64;
	std::vector<float> zn32, zl32;
	whiten(theta_new, nnew, zn64, zn32);
	whiten(theta_last, nlast, zl64, zl32);
	std::vector<double> lw64(nlast);
	std::vector<float> lw32(nlast);
	double lwmax = -INFINITY;
	for (int k = 0; k < nlast; k++) {
		if (!(w_last[k] >= 0.0)) return fail(BEEP_BAD_INPUT, "abcsmc weights: negative or NaN previous weight");
		lw64[k] = w_last[k] > 0.0 ? std::log(w_last[k]) : -INFINITY;
		lw32[k] = (float)lw64[k];
		lwmax = std::max(lwmax, lw64[k]);
	}
	if (!(lwmax > -INFINITY)) return fail(BEEP_BAD_INPUT, "abcsmc weights: every previous weight is zero");
	Layout L;
	const size_t o_zn = L.add(4 * zn32.size()), o_zl = L.add(4 * zl32.size()), o_wl = L.add(4 * (size_t)nlast),
	             o_s = L.add(8 * (size_t)nnew), o_mx = L.add(4 * (size_t)nnew), o_zn64 = L.add(8 * zn64.size()),
	             o_zl64 = L.add(8 * zl64.size()), o_wl64 = L.add(8 * (size_t)nlast), o_far = L.add(4 * (size_t)nnew),
	             o_A = L.add(4 * Af.size()), o_A64 = L.add(8 * Am.size());
	DevBuf buf;
	CUDA_TRY(buf.reserve(L.size));
	char *d = (char *)buf.ptr;
	std::vector<double> logsums(nnew);
	std::vector<float> mx(nnew);
	std::vector<int> far;
	cudaError_t e = cudaMemcpy(d + o_zn, zn32.data(), 4 * zn32.size(), cudaMemcpyHostToDevice);
	if (e == cudaSuccess) e = cudaMemcpy(d + o_zl, zl32.data(), 4 * zl32.size(), cudaMemcpyHostToDevice);
	if (e == cudaSuccess) e = cudaMemcpy(d + o_wl, lw32.data(), 4 * (size_t)nlast, cudaMemcpyHostToDevice);
	if (e == cudaSuccess) e = cudaMemcpy(d + o_A, Af.data(), 4 * Af.size(), cudaMemcpyHostToDevice);
	if (e == cudaSuccess) e = cudaMemcpy(d + o_A64, Am.data(), 8 * Am.size(), cudaMemcpyHostToDevice);
	if (e == cudaSuccess) {
		const LogSums32 k32 = white ? pick_logsums<true>(nvar) : pick_logsums<false>(nvar);
		k32<<<(nnew + kAbcThreads - 1) / kAbcThreads, kAbcThreads>>>(
		    nvar, nnew, (const float *)(d + o_zn), nlast, (const float *)(d + o_zl), (const float *)(d + o_wl),
		    (const float *)(d + o_A), (double *)(d + o_s), (float *)(d + o_mx));
		e = cudaGetLastError();
	}
	if (e == cudaSuccess) e = cudaMemcpy(mx.data(), d + o_mx, 4 * (size_t)nnew, cudaMemcpyDeviceToHost);
	if (e == cudaSuccess) {
		for (int i = 0; i < nnew; i++)
			if (!((double)mx[i] >= lwmax - kFarExponent)) far.push_back(i);   // also NaN: recomputed, then checked
		if (!far.empty()) {
			e = cudaMemcpy(d + o_zn64, zn64.data(), 8 * zn64.size(), cudaMemcpyHostToDevice);
			if (e == cudaSuccess) e = cudaMemcpy(d + o_zl64, zl64.data(), 8 * zl64.size(), cudaMemcpyHostToDevice);
			if (e == cudaSuccess) e = cudaMemcpy(d + o_wl64, lw64.data(), 8 * (size_t)nlast, cudaMemcpyHostToDevice);
			if (e == cudaSuccess) e = cudaMemcpy(d + o_far, far.data(), 4 * far.size(), cudaMemcpyHostToDevice);
			if (e == cudaSuccess) {
				auto k64 = white ? abc_logsums_f64<true> : abc_logsums_f64<false>;
				k64<<<(int)far.size(), kFarThreads>>>(
				    nvar, (const int *)(d + o_far), (const double *)(d + o_zn64), nlast,
				    (const double *)(d + o_zl64), (const double *)(d + o_wl64), (const double *)(d + o_A64),
				    (double *)(d + o_s));
				e = cudaGetLastError();
			}
		}
	}
	if (e == cudaSuccess) e = cudaMemcpy(logsums.data(), d + o_s, 8 * (size_t)nnew, cudaMemcpyDeviceToHost);
	buf.release();
	if (e != cudaSuccess) return fail(BEEP_DEVICE_ERROR, std::string("abcsmc weights: ") + cudaGetErrorString(e));
	std::vector<double> logw(nnew);
	double lmax = -INFINITY;
	for (int i = 0; i < nnew; i++) {
		if (logsums[i] != logsums[i]) return fail(BEEP_NAN_RATE, "abcsmc weights: NaN kernel sum (non-finite parameters?)");
		logw[i] = logprior_new[i] - logsums[i];
		lmax = std::max(lmax, logw[i]);
	}
	if (!normalise) {
		for (int i = 0; i < nnew; i++) w_out[i] = std::exp(logw[i]);
	} else {
		// ABCSMC::normalise_particle_weights, w /= mean(w), formed relative to the
		// largest weight so that no weight overflows on the way
		if (!(lmax > -INFINITY)) return fail(BEEP_BAD_INPUT, "abcsmc weights: every new particle has prior weight zero");
		double wsum = 0.0;
		for (int i = 0; i < nnew; i++) {
			w_out[i] = std::exp(logw[i] - lmax);
			wsum += w_out[i];
		}
		wsum /= nnew;
		for (int i = 0; i < nnew; i++) w_out[i] /= wsum;
	}
	return BEEP_OK;
}
