// Single trials of the FP64 samplers and of their FP32-decided forms (rng_filter.cuh) on
// given Philox words: as host C++ (with the approximate intrinsics replaced by IEEE
// operations, off by their documented error to either side) and, under nvcc, on the GPU.
// The test compiles it against copies of the two headers in which philox10 returns the key
// as a draw's first words, and for a second trial words on the other side of the density's
// peak that are accepted, so that a draw's words are arguments and a rejection shows.
#include <cmath>
#include <cstdint>
#include <cstring>

#ifndef __CUDACC__
#include <algorithm>
#define __device__
#define __forceinline__ inline
#define __noinline__
#define __align__(n) alignas(n)
using std::max;
using std::min;
struct float4 { float x, y, z, w; };
static int g_off;                     // bit 0, 1: quotients, logarithms above (else below); bit 2: exact
static double off_by(double x, int bit, double err) { return g_off & 4 ? x : x + (g_off & bit ? err : -err); }
static inline float __fdividef(float a, float b) { const double q = (double)a / b; return (float)off_by(q, 1, std::fabs(q) * 2.4e-7); }
static inline float logf_off(float x)
{
	const double l = std::log((double)x);
	return (float)off_by(l, 2, x >= 0.5f && x <= 2.f ? 3.6e-7 : 3.6e-7 * std::fabs(l));
}
#define __logf logf_off              // (the C library has a __logf of its own)
static inline float __fdiv_rn(float a, float b) { return a / b; }
static inline float __fsqrt_rn(float a) { return std::sqrt(a); }
static inline uint32_t __umulhi(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }
static inline double __longlong_as_double(long long v) { double d; memcpy(&d, &v, 8); return d; }
static inline long long __double_as_longlong(double d) { long long v; memcpy(&v, &d, 8); return v; }
static inline int __double2hiint(double d) { return (int)(__double_as_longlong(d) >> 32); }
static inline int __double2loint(double d) { return (int)__double_as_longlong(d); }
static inline float __uint_as_float(uint32_t v) { float f; memcpy(&f, &v, 4); return f; }
static inline float __uint2float_rn(uint32_t v) { return (float)v; }
static inline float __int2float_rn(int32_t v) { return (float)v; }
#endif

#include "rng_filter.cuh"

using namespace beep;

// one draw: Poisson of mean `par` (n < 0) or binomial (par, n), first words (x, y)
struct Trial {
	double par;
	int32_t n;
	uint32_t x, y;
	int32_t fp64;                       // the FP64 sampler's draw in two trials
};

// (limit 1: -1 where the first trial is rejected)
static __device__ int32_t trial_fp64(double par, int32_t n, uint32_t x, uint32_t y, uint32_t limit = 1)
{
	return n < 0 ? poisson_fp64(par, x, y, 0, 0, 0, 0, limit) : binomial_fp64(par, n, x, y, 0, 0, 0, 0, limit);
}

static __device__ int32_t trial_filtered(double par, int32_t n, uint32_t x, uint32_t y, const FilterTab &t)
{
	return n < 0 ? poisson_filtered(par, x, y, 0, 0, 0, 0, 2, t) : binomial_filtered(par, n, x, y, 0, 0, 0, 0, 2, t);
}

#ifndef __CUDACC__

namespace {

struct Out {
	Trial *buf;
	int64_t cap, len;
	void put(double par, int32_t n, int64_t x, int64_t y)
	{
		if (x < 0 || y < 0 || x > 0xffffffffll || y > 0xffffffffll || len >= cap) return;
		buf[len++] = Trial{par, n, (uint32_t)x, (uint32_t)y, trial_fp64(par, n, (uint32_t)x, (uint32_t)y, 2)};
	}
};

// the first word w in [0, 2^32] for which at(w) holds, at monotone
template <typename F>
int64_t first_word(F at)
{
	int64_t lo = 0, hi = 1ll << 32;
	while (lo < hi) {
		const int64_t mid = (lo + hi) >> 1;
		if (at((uint32_t)mid)) hi = mid;
		else lo = mid + 1;
	}
	return lo;
}

}  // namespace

extern "C" {

// Trials around every place where a decision of the sampler turns, for the counts in want: the
// words between one count and the next, and for words within each count the V at which the
// trial turns from accepted to rejected; each place at distances 0, 1, 2, 4, ... words.
int64_t boundary_trials(double par, int32_t n, const int32_t *want, int nwant, Trial *buf, int64_t cap)
{
	Out o{buf, cap, 0};
	const double mean = n < 0 ? par : n * std::min(par, 1.0 - par);
	const bool flip = n >= 0 && par > 0.5;
	auto around = [&](int64_t w, int bits, auto put) {
		put(w);
		for (int b = 0; b < bits; b++) {
			put(w - (1ll << b));
			put(w + (1ll << b));
		}
	};
	for (int i = 0; i < nwant; i++) {
		const int32_t k = want[i];
		if (mean < 10.0) {                  // inversion: one word decides
			const int64_t w = first_word([&](uint32_t x) {
				const int32_t r = trial_fp64(par, n, x, 0);
				return (flip ? n - r : r) >= k;
			});
			around(w, 12, [&](int64_t x) { o.put(par, n, x, 0); });
			continue;
		}
		// (at V = 2^-33 a candidate in range is accepted unless its tail is cut: the rejected
		// candidates are those below the range for small words, above it for large ones)
		auto reaches = [&](uint32_t x, int32_t kk) {
			int32_t r = trial_fp64(par, n, x, 0);
			if (r < 0) return x >= 0x80000000u;
			return (flip ? n - r : r) >= kk;
		};
		const int64_t a = first_word([&](uint32_t x) { return reaches(x, k); });
		const int64_t b = first_word([&](uint32_t x) { return reaches(x, k + 1); });
		for (int64_t e : {a, b}) around(e, 20, [&](int64_t x) { o.put(par, n, x, 0); o.put(par, n, x, 0x40000000); });
		if (b <= a) continue;
		for (int j = 0; j <= 8; j++) {
			const int64_t x = a + (b - 1 - a) * j / 8;
			const int64_t v = first_word([&](uint32_t y) { return trial_fp64(par, n, (uint32_t)x, y) < 0; });
			around(v, 30, [&](int64_t y) { o.put(par, n, x, y); });
		}
	}
	return o.len;
}

// the FP64 sampler's draws of the trials' words
void fp64_host(Trial *t, int64_t len)
{
	for (int64_t k = 0; k < len; k++) t[k].fp64 = trial_fp64(t[k].par, t[k].n, t[k].x, t[k].y, 2);
}

// the filtered samplers' results on the host, the approximate operations off by `off`
void filtered_host(const Trial *t, int64_t len, int off, int32_t *out)
{
	g_off = off;
	FilterTab tab;
	filter_tab_fill(tab, 0, 1);
	for (int64_t k = 0; k < len; k++) out[k] = trial_filtered(t[k].par, t[k].n, t[k].x, t[k].y, tab);
}

}  // extern "C"

#else

static __global__ void filtered_kernel(const Trial *t, long long len, int32_t *out)
{
	__shared__ FilterTab tab;
	filter_tab_fill(tab, threadIdx.x, blockDim.x);
	__syncthreads();
	const long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x;
	if (k < len) out[k] = trial_filtered(t[k].par, t[k].n, t[k].x, t[k].y, tab);
}

extern "C" int filtered_gpu(const Trial *t, long long len, int32_t *out)
{
	Trial *dt = nullptr;
	int32_t *dout = nullptr;
	cudaError_t e = cudaMalloc(&dt, sizeof(Trial) * len);
	if (e == cudaSuccess) e = cudaMalloc(&dout, 4 * len);
	if (e == cudaSuccess) e = cudaMemcpy(dt, t, sizeof(Trial) * len, cudaMemcpyHostToDevice);
	if (e == cudaSuccess) {
		filtered_kernel<<<(unsigned)((len + 255) / 256), 256>>>(dt, len, dout);
		e = cudaGetLastError();
	}
	if (e == cudaSuccess) e = cudaMemcpy(out, dout, 4 * len, cudaMemcpyDeviceToHost);
	cudaFree(dt);
	cudaFree(dout);
	return (int)e;
}

#endif
