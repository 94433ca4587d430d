// Plain FP64 form of the tau-leap + observation log-likelihood.
//
// One CTA advances one particle over steps [ti, tf).  Every FP64 value the
// reference computes is computed with the same operations in the same order
// (this file is compiled with --fmad=false), so transition counts and
// populations are bit-identical to the reference driven by the same keyed
// variates.  Per step the CTA runs five phases separated by barriers:
//   A  dinf[st][c][a]     set_I_from_pop / update_I_from_transnum   src/state.cc:178-290
//   B  Imap, Idiag         the same functions' scatter, as a gather  src/state.cc:209-216
//   C  NMI[st][c][a]       get_NMI (+ strain shift of S)             src/state.cc:392-401,547-578
//   D  transition counts   set_transmean + poisson draws             src/state.cc:380-456,608-631
//   E  observation sums    get_obs_value_section                    src/obsmodel.cc:74-109
//      and pop[sett+1]     update_pop                               src/state.cc:460-485
// Models with demographic changes first apply State::democat_change_pop_adjust
// (src/state.cc:339-376) to pop[sett] at the start of each step; their
// populations are FP64 (the kernel's PopT = double instantiation), as in the
// reference, whose populations are doubles throughout.
// The log-likelihood of the scored observations is reduced at the end with
// compensated (Neumaier) sums; the reference sums naively in index order
// (src/obsmodel.cc:28), so the two agree to rounding (1e-12 relative).
//
// The same kernel advances MBP chains (src/mbp.cc:252-330), whose two states
// per chain (Mbp::initial, Mbp::propose) are full trajectories in HBM:
//   mode 1  a new state in the slot that is not current: every cell coupled
//           to the current state (n' = n + Poisson(m'-m), n, or
//           Binomial(n, m'/m)) unless it is a SIMU cell; Imap' either
//           recomputed (INF_UPDATE) or Imap + dImap with dImap built from
//           the count differences (INF_DIF_UPDATE, src/state.cc:109-123).
//           Initialisation (State::simulate) is this mode with every cell SIMU.
//   mode 3  State::initialise_from_particle (src/state.cc:294-322): the counts
//           already in the slot that is not current are kept; Imap
//           (set_Imap), the means (set_transmean) and L are recomputed.
//   mode 2  State::likelihood (src/state.cc:812-826) of the current state
//           with the means recomputed under this batch's tables on the fixed
//           state (Mbp::parameter_proposal, src/mbp.cc:460-478).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <type_traits>

#include "beep_internal.h"
#include "rng_filter.cuh"
#include "rng_fp64.cuh"

namespace beep {
namespace {

constexpr int kMaxThreads = 512;

__device__ double normal_lp(double x, double mean, double var)
{
	return -0.5 * log(2 * 3.14159265358979323846 * var) - (x - mean) * (x - mean) / (2 * var);
}

__device__ double poisson_lp(int i, double lam)
{
	if (lam == 0) return i == 0 ? 0 : -1000000000.0;
	if (i < 0) return -1000000000.0;
	return i * log(lam) - lam - lgamma((double)(i + 1));
}

__device__ double negbin_lp(unsigned int val, double m, double shape)
{
	return lgamma(shape + val) - lgamma((double)val + 1) - lgamma(shape) + shape * log(shape / (shape + m)) +
	       val * log(m / (shape + m));
}

// ObservationModel::obs_prob, src/obsmodel.cc:245-305
__device__ double obs_prob(double value, int kind, double val, int model, double sd, double shape, double thresh)
{
	if (value < 0) value = 0;
	if (kind == BEEP_OBSVAL_UNKNOWN) return 0;
	if (kind == BEEP_OBSVAL_THRESH) {
		if (model == BEEP_OBS_NORMAL || model == BEEP_OBS_NORMAL_PERCENT) {
			if (value < thresh) return normal_lp(thresh, thresh, sd * sd);
			return normal_lp(thresh, value, sd * sd);
		}
		double lam = value < 1 ? 1 : value;
		double sum = 0.0;
		for (double v = 0; v <= thresh; v++)
			sum += exp(model == BEEP_OBS_POISSON ? poisson_lp((int)v, lam) : negbin_lp((unsigned)v, lam, shape));
		return log(sum);
	}
	if (model == BEEP_OBS_NORMAL || model == BEEP_OBS_NORMAL_PERCENT) return normal_lp(val, value, sd * sd);
	double lam = value < 1 ? 1 : value;
	if (model == BEEP_OBS_POISSON) return poisson_lp((int)(val + 0.5), lam);
	return negbin_lp((unsigned)(int)(val + 0.5), lam, shape);
}

__device__ __forceinline__ void set_status(int32_t *st, int v)
{
	atomicCAS(st, 0, v);
}

// State::democat_change_pop_adjust (src/state.cc:339-376) of one particle's
// pop[sett]: per change, each value's population summed over the change's
// areas, groups and compartments (in that order, one thread per value), the
// shares' gap to the step's fractions, and every (area, group, compartment)
// row shifted by gap x the row's total.  The rows are disjoint (areas and dp
// are unique within a change), so they are updated in parallel.
__device__ void democat_adjust(const ModelDev &m, double *pop, int sett, int tid, int nth)
{
	__shared__ double s_cat[kMaxDccValues], s_gap[kMaxDccValues];
	const int C = m.C, DP = m.DP;
	for (int k = 0; k < m.ndcc; k++) {
		const int nv = m.dcc_nval[k], a0 = m.dcc_area_ptr[k], a1 = m.dcc_area_ptr[k + 1];
		const int *dpg = m.dcc_dp + m.dcc_dp_ptr[k];
		const int ng = (m.dcc_dp_ptr[k + 1] - m.dcc_dp_ptr[k]) / nv;
		if (tid < nv) {
			double s = 0.0;
			for (int j = a0; j < a1; j++) {
				const double *pc = pop + (size_t)m.dcc_area[j] * C * DP;
				for (int g = 0; g < ng; g++) {
					const int dp = dpg[g * nv + tid];
					for (int co = 0; co < C; co++) s += pc[(size_t)co * DP + dp];
				}
			}
			s_cat[tid] = s;
		}
		__syncthreads();
		if (tid == 0) {
			const double *fr = m.dcc_frac + m.dcc_frac_ptr[k] + (size_t)sett * nv;
			double tot = 0.0;
			for (int f = 0; f < nv; f++) tot += s_cat[f];
			for (int f = 0; f < nv; f++) s_gap[f] = fr[f] - s_cat[f] / tot;
		}
		__syncthreads();
		const int nrow = (a1 - a0) * ng * C;
		for (int idx = tid; idx < nrow; idx += nth) {
			const int co = idx % C, g = (idx / C) % ng, c = m.dcc_area[a0 + idx / (C * ng)];
			double *pc = pop + ((size_t)c * C + co) * DP;
			const int *dps = dpg + g * nv;
			double sum = 0.0;
			for (int f = 0; f < nv; f++) sum += pc[dps[f]];
			for (int f = 0; f < nv; f++) pc[dps[f]] += s_gap[f] * sum;
		}
		__syncthreads();
	}
}

// n / d for the kernel's index splits: one multiply where every n in [0, nmax] allows it
struct Div {
	uint32_t d, mul;
	__device__ __forceinline__ Div(int div, size_t nmax) : d((uint32_t)div), mul(0u)
	{
		if (d > 1 && (unsigned long long)nmax * d < 0x100000000ull) mul = 0xffffffffu / d + 1u;
	}
	__device__ __forceinline__ int quot(int n) const
	{
		return d == 1 ? n : mul ? (int)__umulhi((uint32_t)n, mul) : (int)((uint32_t)n / d);
	}
};

// FP64 values tested on the integer pipe
__device__ __forceinline__ bool is_zero(double x) { return (__double_as_longlong(x) << 1) == 0; }
__device__ __forceinline__ bool is_nan(double x)
{
	return (unsigned long long)(__double_as_longlong(x) & 0x7fffffffffffffffll) > 0x7ff0000000000000ull;
}

// Integer-valued infectious-count changes (integer infectivities: the counts' sums are integers)
// are kept as a normalised 32-bit magnitude and {sign, bits}, so that their products with the
// mixing matrix come from the integer pipe: 20 instructions beside the sum's 64 cycles on the
// FP64 pipe instead of 64 more on it.  {0, 0} is zero; a magnitude without its top bit marks a
// value kept as a double.
__device__ __forceinline__ uint2 encode_int(long long v)
{
	const unsigned long long a = (unsigned long long)(v < 0 ? -v : v);
	if (a == 0) return make_uint2(0u, 0u);
	if (a >> 32) return make_uint2(1u, 0u);
	const uint32_t x = (uint32_t)a;
	const int z = __clz((int)x);
	return make_uint2(x << z, (v < 0 ? 0x80000000u : 0u) | (uint32_t)(32 - z));
}

// The IEEE product, rounded to nearest even, of an encoded integer and a normal double of
// exponent -500 to 500: 53 x 32 bits, the top 53 kept
__device__ __forceinline__ double mul_int(uint2 d, double v)
{
	const uint32_t vh = (uint32_t)__double2hiint(v), vl = (uint32_t)__double2loint(v);
	const uint64_t lo = (uint64_t)vl * d.x;
	const uint64_t t = (uint64_t)((vh & 0xfffffu) | 0x100000u) * d.x + (lo >> 32);   // the product / 2^32
	const uint32_t w = (uint32_t)lo;
	const bool top = (t >> 52) != 0;
	uint64_t mant = top ? t : (t << 1) | (w >> 31);
	const uint32_t rest = top ? w : w << 1;
	mant += rest > 0x80000000u || (rest == 0x80000000u && (mant & 1u)) ? 1u : 0u;
	const uint32_t e = ((vh >> 20) & 0x7ffu) + (d.y & 63u) - (top ? 1u : 2u);       // (the mantissa's top bit adds one)
	return __longlong_as_double((long long)((((uint64_t)e << 52) + mant) | ((uint64_t)((vh ^ d.y) & 0x80000000u) << 32)));
}

// What the kernel keeps in shared memory: level 2 the particle's arrays and the tables, level 1
// the tables (a larger model's arrays stay in its global work region), level 0 nothing.
// The step's tables are double-buffered: a step's are loaded during the previous step's draws.
struct PlainSmem {
	size_t pop, tn, imap, idiag, dinf, x, rate, sus, infdif, bea, eta, N, diag, fac, from, to, age, adp, brow, eref, dint, idi, total;
	__host__ __device__ PlainSmem(const ModelDev &m, int pop_bytes, int level)
	{
		size_t off = 0;
		const bool state = level == 2;
		auto take = [&](size_t n) { const size_t o = off; off += level == 0 ? 0 : (n + 15) & ~(size_t)15; return o; };
		const size_t ncol = (size_t)m.A * m.DP, ag = (size_t)m.NS * m.A * m.G, sa = (size_t)m.NS * m.A;
		pop = take(state ? 2 * (size_t)pop_bytes * m.C * ncol : 0);
		tn = take(state ? 4 * (size_t)m.T * ncol : 0);
		imap = take(state ? 8 * ag : 0);
		idiag = take(state ? 8 * ag : 0);
		dinf = take(state ? 8 * ag : 0);
		x = take(state ? 8 * ag : 0);
		rate = take(8 * (size_t)m.T * m.DP);
		sus = take(8 * (size_t)m.DP);
		infdif = take(8 * (size_t)m.T);
		bea = take(16 * sa);
		eta = take(16 * sa);
		N = take(16 * (size_t)m.G * m.G);
		diag = take(8 * (size_t)m.A);
		fac = take(8 * (size_t)m.A);
		from = take(4 * (size_t)m.T);
		to = take(4 * (size_t)m.T);
		age = take(4 * (size_t)m.DPS);
		adp = take(4 * (size_t)m.G);
		brow = take(4 * sa);
		eref = take(4 * sa);
		dint = take(8 * ag);
		idi = take(4 * (size_t)m.T);
		total = off;
	}
};

// One CTA per particle.  Bound: latency of a step's dependent phases for small models; the
// FP64 pipe (one warp instruction per 16 cycles and SM) for large ones, where the
// area-mixing sums remain: an addition per (source, target, age), its product formed on the
// integer pipe where the counts are integers (187 particles of 77x5 over 180 steps: 138 ms with
// everything on the FP64 pipe, 16.8 ms before the products left it, 12.3 ms now).  The rest
// was taken off that pipe: the draws are decided in FP32 (rng_filter.cuh), comparisons and
// zero tests are done on the bits, a target's NMI terms are formed once instead of once
// per age, unit observation factors sum their integer counts as integers.
// PopT: int32_t, or double for models with demographic changes.
template <typename PopT>
__global__ void __launch_bounds__(kMaxThreads) sim_plain_kernel(const ModelDev m, const BatchDev b, const int level, const int sms)
{
	constexpr bool kPop64 = sizeof(PopT) == 8;
	extern __shared__ __align__(16) unsigned char smem_raw[];
	__shared__ FilterTab ftab;
	const uint32_t lim = b.sampler_limit ? b.sampler_limit : 65536u;   // sampler rejection iterations
	const int p = blockIdx.x;
	if (p >= b.P) return;
	// CTAs that share an SM start their threads two schedulers apart: the small models' FP64 work
	// is one warp's, and two of them on one scheduler took turns on its pipe
	const int nth = blockDim.x, tid = (threadIdx.x + 64 * ((p / sms) & 1)) & (nth - 1);
	const int A = m.A, G = m.G, DP = m.DP, NS = m.NS, DPS = m.DPS, C = m.C, T = m.T, ncol = A * DP, GG = G * G;
	const size_t popsz = (size_t)C * ncol, tnsz = (size_t)T * ncol;
	const int agsz = NS * A * G, NSA = NS * A;
	const int nsteps = b.tf - b.ti;
	const GroupDir dir = b.dirs[b.group_of ? b.group_of[p] : 0];
	const uint32_t stream = b.stream_of ? b.stream_of[p] : (uint32_t)p;
	const uint32_t k0 = b.key_of ? b.key_of[p].x : b.k0, k1 = b.key_of ? b.key_of[p].y : b.k1;   // the particle's key
	const double *fp = b.fpool;
	const int32_t *ip = b.ipool;
	const double *infectivity = fp + dir.infectivity, *beta_rows = fp + dir.beta_rows, *areafactor = fp + dir.areafactor;
	const double *Ntime = fp + dir.Ntime, *geo = fp + dir.geo_spline, *efoi_spline = fp + dir.efoi_spline;
	const double *efoi_age = fp + dir.efoi_agedist, *obs_spline = fp + dir.obs_spline;
	const double *efoi_mult = dir.efoi_mult >= 0 ? fp + dir.efoi_mult : nullptr;
	const double *tm_mult = dir.tm_mult >= 0 ? fp + dir.tm_mult : nullptr;

	// MBP chains: slot of the current state and of the state being written
	const int mode = b.mode;
	const int cs_i = mode ? b.cur[p] : 0, cs_p = 1 - cs_i;
	const bool dif = mode == 1 && b.inf_dif && !b.simu_all;
	const bool writes = mode == 1 || mode == 3;          // the non-current slot receives a state
	auto chs = [&](int slot, int s) { return ((size_t)slot * b.P + p) * m.S + s; };
	double Lsum = 0.0, Lcmp = 0.0;   // mode 2: compensated partial sum of this thread

	const bool smem_state = level == 2, smem_tabs = level >= 1;
	const PlainSmem lay(m, (int)sizeof(PopT), level);
	PopT *pop_cur = smem_state ? (PopT *)(smem_raw + lay.pop) : (PopT *)b.pop_a + (size_t)p * popsz;
	PopT *pop_nxt = smem_state ? pop_cur + popsz : (PopT *)b.pop_b + (size_t)p * popsz;
	double *Imap = smem_state ? (double *)(smem_raw + lay.imap) : b.Imap + (size_t)p * agsz;
	double *Idiag = smem_state ? (double *)(smem_raw + lay.idiag) : b.Idiag + (size_t)p * agsz;
	double *dinf = smem_state ? (double *)(smem_raw + lay.dinf) : b.dinf + (size_t)p * agsz;
	double *X = smem_state ? (double *)(smem_raw + lay.x) : b.NMI + (size_t)p * agsz;   // NMI terms (NMI for one age)
	double *acc = b.obs_acc + (size_t)p * b.nscored;
	double *bea = (double *)(smem_raw + lay.bea), *eta = (double *)(smem_raw + lay.eta), *Nm = (double *)(smem_raw + lay.N);
	int32_t *adp = (int32_t *)(smem_raw + lay.adp);      // the dp of each age, where each has one
	const bool one_dp = smem_tabs && m.dp_age_unique;
	int32_t *status = b.status + p;

	const int src = b.pop_of ? b.pop_of[p] : p;
	for (size_t k = tid; k < popsz; k += nth)
		pop_cur[k] = b.ti == 0 ? (PopT)m.pop_init[k] : ((const PopT *)b.pop_in)[(size_t)src * popsz + k];
	for (int k = tid; k < b.nscored; k += nth) acc[k] = 0.0;
	// tables in shared memory (level >= 1) or where they are
	auto table = [&](size_t off, const auto *src, int n) {
		if (!smem_tabs) return src;
		auto *dst = (std::remove_const_t<std::remove_pointer_t<decltype(src)>> *)(smem_raw + off);
		for (int k = tid; k < n; k += nth) dst[k] = src[k];
		return (decltype(src))dst;
	};
	const double *rate = table(lay.rate, fp + dir.transrate, T * DP), *sus = table(lay.sus, fp + dir.susceptibility, DP);
	const double *infdif = table(lay.infdif, fp + dir.infdif, T);
	const double *diag = table(lay.diag, m.M_diag, A), *afac = table(lay.fac, m.M_factor, A);
	const int32_t *from = table(lay.from, m.trans_from, T), *to = table(lay.to, m.trans_to, T);
	const int32_t *age = table(lay.age, m.dp_age, DPS);
	const int32_t *brow = table(lay.brow, ip + dir.beta_row_of, NSA), *eref = table(lay.eref, ip + dir.efoi_ref, NSA);
	uint2 *dint = (uint2 *)(smem_raw + lay.dint);
	int32_t *idi = (int32_t *)(smem_raw + lay.idi);
	__shared__ int s_soft;
	if (tid == 0) {
		// integer infectivities (and a mixing matrix of ordinary values): dinf as integers
		bool whole = smem_tabs && m.mix_regular;
		for (int tr = 0; tr < T && whole; tr++) {
			const double x = fp[dir.infdif + tr];
			whole = fabs(x) <= 1024.0 && x == floor(x);
			idi[tr] = (int32_t)x;
		}
		for (int co = 0; co < C && whole; co++) whole = fabs(infectivity[co]) <= 1024.0 && infectivity[co] == floor(infectivity[co]);
		s_soft = whole;
	}
	if (one_dp)
		for (int dp = tid; dp < DPS; dp += nth) adp[m.dp_age[dp]] = dp;
	filter_tab_fill(ftab, tid, nth);
	__syncthreads();

	const bool soft = s_soft != 0;
	const Div divDP(DP, tnsz + popsz), divG(G, agsz), divA(A, NSA), divDPS(DPS, (size_t)A * DPS);
	// a step's tables of (strain, area) i: beta * areafactor, external force per capita (loaded, and
	// combined once the loads have landed)
	auto slice_load = [&](int s, int i, double &be, double &af, double &et, double &em) {
		const int st = divA.quot(i), c = i - st * A;
		be = beta_rows[(size_t)brow[i] * m.S + s];
		af = areafactor[(size_t)(s / m.div_per_time) * A + c];
		et = efoi_spline[(size_t)eref[i] * m.S + s];
		if (efoi_mult) em = efoi_mult[((size_t)s * A + c) * NS + st];
	};
	auto slice_value = [&](double be, double af, double et, double em, double &b_out, double &e_out) {
		b_out = be * af;
		et = is_zero(et) ? m.efoi_zero : et / m.popsize;
		if (efoi_mult) et *= em;
		e_out = et;
	};
	auto slice = [&](int s, int i, double &be, double &et) {
		double q0, q1, q2, q3 = 1.0;
		slice_load(s, i, q0, q1, q2, q3);
		slice_value(q0, q1, q2, q3, be, et);
	};
	for (int i = tid; smem_tabs && i < NSA; i += nth) slice(b.ti, i, bea[i], eta[i]);
	for (int i = tid; smem_tabs && i < GG; i += nth) Nm[i] = Ntime[(size_t)b.ti * GG + i];

	// draws of a step: (transition, column), the columns of a transition padded to whole warps
	// where that costs no further pass of the CTA (a warp then draws from similar means)
	const int pad = (ncol + 31) & ~31;
	const int cols = (T * pad + nth - 1) / nth <= ((int)tnsz + nth - 1) / nth ? pad : ncol;
	const Div divCol(cols, (size_t)T * cols);
	// dinf per (strain, source area, age) of the next step's maps, from the step's counts
	const int tinf = (tid + 32) & (nth - 1);             // (the last warp first: see below)
	auto dinf_of_counts = [&](const int32_t *cnt, const int32_t *base) {
		for (int idx = tinf; idx < agsz; idx += nth) {
			const int sc = divG.quot(idx), a = idx - sc * G, st = divA.quot(sc), c = sc - st * A;
			const int dp0 = one_dp ? adp[a] : 0, dp1 = one_dp ? dp0 + 1 : DPS;
			if (soft) {
				long long s = 0;
				for (int tr = 0; tr < T; tr++) {
					const int di = idi[tr];
					if (di == 0) continue;
					for (int dp = dp0; dp < dp1; dp++) {
						if (age[dp] != a) continue;
						const int cl = (c * T + tr) * DP + st * DPS + dp;
						s += (long long)di * (base ? cnt[cl] - base[cl] : cnt[cl]);
					}
				}
				const uint2 q = encode_int(s);
				dint[idx] = q;
				if (q.x == 1u) dinf[idx] = (double)s;
				continue;
			}
			double s = 0.0;
			for (int tr = 0; tr < T; tr++) {
				const double di = infdif[tr];
				if (is_zero(di)) continue;
				for (int dp = dp0; dp < dp1; dp++) {
					if (age[dp] != a) continue;
					const int cl = (c * T + tr) * DP + st * DPS + dp;
					const int num = base ? cnt[cl] - base[cl] : cnt[cl];
					if (num != 0) s += di * (double)num;
				}
			}
			dinf[idx] = s;
		}
	};

	const int itr = m.infection_trans;
	const int inf_from = m.trans_from[itr];
	// Loads whose latency a small model's step would wait for are issued a phase or a step ahead,
	// by the threads that draw last: the tables of the next step by the last warps (tslice), the
	// observations from three quarters of the CTA on (tobs), the next infectious changes by the
	// last warp first (tinf).
	const int tslice = nth - 1 - tid, tobs = (tid + nth / 4) & (nth - 1);
	const bool few = agsz <= nth / 4;
	int buf = 0;
	int s0 = b.step_ptr[0], s1 = b.step_ptr[1], s2 = b.step_ptr[min(2, nsteps)];   // this step's observations and the next's
	int opos = s0 + tobs < s1 ? b.step_obs[s0 + tobs] : 0;   // this thread's first observation
	double d_next = geo[b.ti];
	for (int sett = b.ti; sett < b.tf; sett++) {
		// the step's counts: in shared memory, or the output or chain array itself (ext)
		int32_t *ext = mode ? b.ch_tn + chs(writes ? cs_p : cs_i, sett) * tnsz
		           : b.tn_traj ? b.tn_traj + ((size_t)p * nsteps + (sett - b.ti)) * tnsz : nullptr;
		int32_t *tn = smem_state ? (int32_t *)(smem_raw + lay.tn) : ext ? ext : b.tn + (size_t)p * tnsz;
		const bool copy = smem_state && ext;
		const double *be = bea + buf * NSA, *et = eta + buf * NSA;
		const double *N = smem_tabs ? Nm + buf * GG : Ntime + (size_t)sett * GG;
		const int sn = sett + 1 < b.tf ? sett + 1 : sett;
		const double d = d_next, omd = 1 - d;
		d_next = geo[sn];
		const bool scoring = mode != 2;
		const int s3 = b.step_ptr[min(sett + 3 - b.ti, nsteps)];
		const int oidx = scoring && s0 + tobs < s1 ? b.scored[opos] : -1;
		// the current state's cell of this thread's first draw (MBP chains)
		int32_t first_n = 0;
		double first_r = 0.0;
		if (mode == 1 && !b.simu_all && tid < T * cols) {
			const int tr = divCol.quot(tid), col = tid - tr * cols;
			if (col < ncol) {
				const int c = divDP.quot(col);
				const size_t ci = chs(cs_i, sett) * tnsz + ((size_t)c * T + tr) * DP + (col - c * DP);
				first_n = b.ch_tn[ci];
				first_r = b.ch_mean[ci];
			}
		}

		if constexpr (kPop64) {
			if (m.ndcc > 0) democat_adjust(m, pop_cur, sett, tid, nth);   // pop[sett] before its step
		}
		if (sett == b.ti && mode != 2 && !dif) {
			// the start populations' infectious counts
			for (int idx = tid; idx < agsz; idx += nth) {
				const int sc = divG.quot(idx), a = idx - sc * G, st = divA.quot(sc), c = sc - st * A;
				double s = 0.0;
				for (int co = 0; co < C; co++) {
					const double inf = infectivity[co];
					if (inf != 0) {
						for (int dp = 0; dp < DPS; dp++) {
							if (age[dp] != a) continue;
							const double pv = (double)pop_cur[((size_t)c * C + co) * DP + st * DPS + dp];
							if (pv != 0) s += inf * pv;
						}
					}
				}
				dinf[idx] = s;
				if (soft) dint[idx] = is_zero(s) ? make_uint2(0u, 0u) : make_uint2(1u, 0u);
			}
			__syncthreads();
		}

		// ---- B: Imap/Idiag per (strain, target area, age), sources in ascending order, and
		// the target's NMI term (INF_DIF_UPDATE: the running sums are dImap/dIdiag and the
		// state's maps are the current state's plus them); strain shift of the susceptibles
		for (int idx = tid; idx < agsz; idx += nth) {
			const int sc = divG.quot(idx), a = idx - sc * G, st = divA.quot(sc), t = sc - st * A;
			double imv, idv;                               // the state's maps
			const size_t io = mode ? chs(cs_i, sett) * agsz + idx : 0;
			const double im_i = dif || mode == 2 ? b.ch_Imap[io] : 0.0, id_i = dif || mode == 2 ? b.ch_Idiag[io] : 0.0;
			if (mode == 2) {
				imv = im_i;
				idv = id_i;
			} else {
				const double *dst = dinf + (size_t)st * A * G + a;
				double im = sett == b.ti ? 0.0 : Imap[idx];
				double id = sett == b.ti ? 0.0 : Idiag[idx];
				const int j1 = m.csc_ptr[t + 1];
				if (dif && sett == b.ti) {
				} else if (soft) {
					const uint2 *dq = dint + (size_t)st * A * G + a;
					const uint2 q = dq[t * G];
					if (q.x != 0u) id += q.x == 1u ? dst[t * G] * diag[t] : mul_int(q, diag[t]);
					// few elements: four products at once (independent), then their additions in order;
					// many: the warps hide each other, and zero counts are passed by (77 areas x 5 ages:
					// 13.8 ms with four at once against 12.3 ms; 10 x 3: 4.6 against 4.9 ms)
					int j = m.csc_ptr[t];
					for (; few && j + 4 <= j1; j += 4) {
						uint2 qs[4];
						double v[4];
						bool wide = false;
#pragma unroll
						for (int u = 0; u < 4; u++) {
							qs[u] = dq[m.csc_src[j + u] * G];
							v[u] = m.csc_val[j + u];
							wide |= qs[u].x == 1u;
						}
						if (!wide) {
#pragma unroll
							for (int u = 0; u < 4; u++) v[u] = mul_int(qs[u], v[u]);
						} else {
#pragma unroll 1
							for (int u = 0; u < 4; u++) {
								const uint2 q1 = u == 0 ? qs[0] : u == 1 ? qs[1] : u == 2 ? qs[2] : qs[3];
								const double v1 = u == 0 ? v[0] : u == 1 ? v[1] : u == 2 ? v[2] : v[3];
								const double pr = q1.x == 1u ? dst[m.csc_src[j + u] * G] * v1 : mul_int(q1, v1);
								if (u == 0) v[0] = pr;
								else if (u == 1) v[1] = pr;
								else if (u == 2) v[2] = pr;
								else v[3] = pr;
							}
						}
#pragma unroll
						for (int u = 0; u < 4; u++)
							if (qs[u].x != 0u) im += v[u];
					}
#pragma unroll 4
					for (; j < j1; j++) {
						const int src = m.csc_src[j] * G;
						const double v = m.csc_val[j];
						const uint2 qs = dq[src];
						if (qs.x != 0u) im += qs.x == 1u ? dst[src] * v : mul_int(qs, v);
					}
				} else {
					const double dself = dst[t * G];
					if (!is_zero(dself)) id += dself * diag[t];
#pragma unroll 4
					for (int j = m.csc_ptr[t]; j < j1; j++) {
						const double ds = dst[m.csc_src[j] * G], v = m.csc_val[j];
						if (!is_zero(ds)) im += ds * v;
					}
				}
				Imap[idx] = im;
				Idiag[idx] = id;
				imv = dif ? im_i + im : im;
				idv = dif ? id_i + id : id;
				if (writes) {
					const size_t ow = chs(cs_p, sett) * agsz + idx;
					b.ch_Imap[ow] = imv;
					b.ch_Idiag[ow] = idv;
				}
			}
			const double fac = afac[t];
			if (G == 1) {
				const double val = idv * (d + fac * omd) + imv * d;
				X[idx] = val < 0 ? 0 : val;
			} else {
				X[idx] = (idv + imv) * d + fac * idv * omd;
			}
		}
		if (NS > 1) {
			for (int idx = tid; idx < A * DPS; idx += nth) {
				const int c = divDPS.quot(idx), dp = idx - c * DPS;
				PopT *sp = pop_cur + ((size_t)c * C + inf_from) * DP;
				double sum = 0.0;
				for (int st = 1; st < NS; st++) {
					sum += (double)sp[DPS * st + dp];
					sp[DPS * st + dp] = 0;
				}
				if constexpr (kPop64) sp[dp] += sum;
				else sp[dp] = (int32_t)((double)sp[dp] + sum);
			}
		}
		__syncthreads();

		// ---- D: transition means and counts per (transition, column); the next step's tables
		// and this thread's next observation are loaded on the way
		double nb = 0.0, na = 0.0, ne = 0.0, nm = 1.0, nN = 0.0;
		if (smem_tabs && tslice < NSA) slice_load(sn, tslice, nb, na, ne, nm);
		if (smem_tabs && tslice < GG) nN = Ntime[(size_t)sn * GG + tslice];
		int oq0 = 0, oq1 = 0, ospl = -1;
		double ofac = 0.0, oacc = 0.0;
		if (oidx >= 0) {
			oq0 = m.obs_cell_ptr[oidx];
			oq1 = m.obs_cell_ptr[oidx + 1];
			ospl = m.obs_spline[oidx];
			ofac = m.obs_factor[oidx];
			oacc = acc[opos];
		}
		const int npos = scoring && s1 + tobs < s2 ? b.step_obs[s1 + tobs] : 0;
		for (int item = tid; item < T * cols; item += nth) {
			const int tr = divCol.quot(item), col = item - tr * cols;
			if (col >= ncol) continue;
			const int c = divDP.quot(col), dp = col - c * DP;
			const size_t cell = ((size_t)c * T + tr) * DP + dp;
			double mean = 0.0;
			if (tr == itr) {
				const int st = dp / DPS, dpl = dp - st * DPS;
				const PopT popu = pop_cur[((size_t)c * C + inf_from) * DP + dpl];
				if (!(popu <= 0)) {                // (a NaN population's rate is NaN)
					const int sc = st * A + c, a = age[dpl];
					double nmi;
					if (G == 1) nmi = X[sc];
					else {
						nmi = 0.0;
						for (int aa = 0; aa < G; aa++) nmi += N[a * G + aa] * X[sc * G + aa];
						if (nmi < 0) nmi = 0;
					}
					double bsc, esc;
					if (smem_tabs) { bsc = be[sc]; esc = et[sc]; }
					else slice(sett, sc, bsc, esc);
					const double ext_foi = esc * efoi_age[(size_t)eref[sc] * G + a];
					mean = m.dt * (double)popu * sus[dp] * (bsc * nmi + ext_foi);
				}
			} else {
				const PopT popu = pop_cur[((size_t)c * C + from[tr]) * DP + dp];
				if (!(popu <= 0)) mean = m.dt * (double)popu * rate[tr * DP + dp];
			}
			if (tm_mult) mean *= tm_mult[(size_t)sett * tnsz + cell];   // prediction modifications
			const bool bad = is_nan(mean);
			if (bad) set_status(status, BEEP_NAN_RATE);
			int32_t n = 0;
			if (mode >= 2) {                    // the given counts stay
				n = ext[cell];
				if (mode == 2) {                  // State::likelihood term of the fixed count
					double lp;
					// (no logarithm for a zero count, log n! from the table: the same values)
					if (n == 0 && (unsigned long long)__double_as_longlong(mean) < 0x7ff0000000000000ull) lp = -mean;
					else if (n <= 0 || n >= b.nlgam || is_zero(mean)) lp = poisson_lp(n, mean);
					else lp = n * log(mean) - mean - b.lgam[n];
					const double t = Lsum + lp;
					const bool big = (__double_as_longlong(Lsum) & 0x7fffffffffffffffll) >= (__double_as_longlong(lp) & 0x7fffffffffffffffll);
					Lcmp += ((big ? Lsum : lp) - t) + (big ? lp : Lsum);
					Lsum = t;
				} else {
					b.ch_mean[chs(cs_p, sett) * tnsz + cell] = mean;
				}
				if (copy) tn[cell] = n;
				continue;
			}
			if (!bad && !is_zero(mean)) {
				if (__double_as_longlong(mean) > __double_as_longlong(1000000000.0)) set_status(status, BEEP_COUNT_OVERFLOW);
				else {
					// integers equal to the FP64 samplers' (rng_filter.cuh)
					double draw = mean;
					int32_t n0 = 0;
					bool thin = false;
					double ri = 0.0;
					if (mode != 0 && !b.simu_all && !(b.simu && b.simu[((size_t)p * m.S + sett) * A + c])) {
						// coupled to the current state (src/mbp.cc:293-305)
						const size_t ci = chs(cs_i, sett) * tnsz + cell;
						n0 = item == tid ? first_n : b.ch_tn[ci];
						ri = item == tid ? first_r : b.ch_mean[ci];
						draw = mean - ri;
						thin = !(mean >= ri);           // (a NaN current mean draws as the binomial of NaN: 0)
					}
					if (thin) n = binomial_filtered(mean / ri, n0, k0, k1, (uint32_t)col, (uint32_t)tr, (uint32_t)sett, stream, lim, ftab);
					else {
						if (draw > 0.0) n = poisson_filtered(draw, k0, k1, (uint32_t)col, (uint32_t)tr, (uint32_t)sett, stream, lim, ftab);
						if (n >= 0) n += n0;
					}
					if (n < 0) { set_status(status, BEEP_TIMEOUT); n = 0; }
				}
			}
			if (mode == 1) b.ch_mean[chs(cs_p, sett) * tnsz + cell] = mean;
			tn[cell] = n;
			if (copy) ext[cell] = n;
		}
		if (smem_tabs) {
			double *tb = bea + (buf ^ 1) * NSA, *te = eta + (buf ^ 1) * NSA, *tN = Nm + (buf ^ 1) * GG;
			if (tslice < NSA) slice_value(nb, na, ne, nm, tb[tslice], te[tslice]);
			if (tslice < GG) tN[tslice] = nN;
			for (int i = tslice + nth; i < NSA; i += nth) slice(sn, i, tb[i], te[i]);
			for (int i = tslice + nth; i < GG; i += nth) tN[i] = Ntime[(size_t)sn * GG + i];
		}
		int oc[4];                                           // its first cells
#pragma unroll
		for (int i = 0; i < 4; i++) oc[i] = oq0 + i < oq1 ? m.obs_cells[oq0 + i] : 0;
		__syncthreads();

		// ---- E: observation sums (one thread per active observation, cells in reference order)
		for (int k = scoring ? s0 + tobs : s1; k < s1; k += nth) {
			const bool head = k == s0 + tobs;
			int q0 = oq0, q1 = oq1, spl = ospl, pos = opos;
			double fac = ofac, v = oacc;
			if (!head) {
				pos = b.step_obs[k];
				const int o = b.scored[pos];
				q0 = m.obs_cell_ptr[o];
				q1 = m.obs_cell_ptr[o + 1];
				spl = m.obs_spline[o];
				fac = m.obs_factor[o];
				v = acc[pos];
			}
			if (!kPop64 && spl < 0 && __double_as_longlong(fac) == __double_as_longlong(1.0)) {
				// a unit factor: the counts' sum is an integer, exact in either arithmetic
				long long sum = 0;
				int q = q0;
				if (head) {
#pragma unroll
					for (int i = 0; i < 4; i++)
						if (q0 + i < q1) sum += oc[i] >= 0 ? (long long)tn[oc[i]] : (long long)pop_cur[-1 - oc[i]];
					q = q0 + 4;
				}
				for (; q < q1; q++) {
					const int cell = m.obs_cells[q];
					sum += cell >= 0 ? (long long)tn[cell] : (long long)pop_cur[-1 - cell];
				}
				if (sum != 0) v += (double)sum;
			} else {
				for (int q = q0; q < q1; q++) {
					const int cell = m.obs_cells[q];
					if (cell >= 0) {
						const double num = (double)tn[cell];
						if (num != 0) {
							if (spl < 0) v += fac * num;
							else v += fac * num * obs_spline[(size_t)spl * m.S + sett];
						}
					} else {
						v += fac * (double)pop_cur[-1 - cell];
					}
				}
			}
			acc[pos] = v;
		}
		opos = npos;
		s0 = s1;
		s1 = s2;
		s2 = s3;
		// update_pop into the other buffer, a column per thread and compartment
		for (int k = tid; k < (int)popsz; k += nth) {
			const int cc = divDP.quot(k), dp = k - cc * DP, c = cc / C, co = cc - c * C;
			const int32_t *tc = tn + (size_t)c * T * DP + dp;
			if constexpr (kPop64) {
				// FP64 populations: the flows in transition order, as update_pop applies them
				double v = pop_cur[k];
				for (int tr = 0; tr < T; tr++) {
					const int32_t n = tc[tr * DP];
					if (n != 0) {
						if (from[tr] == co) v -= (double)n;
						if (to[tr] == co) v += (double)n;
					}
				}
				pop_nxt[k] = v;
			} else {
				long long v = pop_cur[k];
				for (int tr = 0; tr < T; tr++) {
					const long long n = tc[tr * DP];
					if (from[tr] == co) v -= n;
					if (to[tr] == co) v += n;
				}
				if (v > 2147483647ll || v < -2147483648ll) { set_status(status, BEEP_COUNT_OVERFLOW); v = 0; }
				pop_nxt[k] = (int32_t)v;
			}
			if (b.pop_traj) ((PopT *)b.pop_traj)[((size_t)p * nsteps + (sett - b.ti)) * popsz + k] = pop_cur[k];
		}
		// ---- A of the next step: dinf from this step's counts (INF_DIF_UPDATE: their differences)
		if (sett + 1 < b.tf && mode != 2) dinf_of_counts(tn, dif ? b.ch_tn + chs(cs_i, sett) * tnsz : nullptr);
		__syncthreads();
		PopT *sw = pop_cur; pop_cur = pop_nxt; pop_nxt = sw;
		buf ^= 1;
	}

	if (b.pop_out)
		for (size_t k = tid; k < popsz; k += nth) ((PopT *)b.pop_out)[(size_t)p * popsz + k] = pop_cur[k];

	__shared__ double part_s[kMaxThreads], part_c[kMaxThreads];
	if (mode == 2) {
		// the threads' compensated partial sums, combined in thread order
		part_s[tid] = Lsum;
		part_c[tid] = Lcmp;
		__syncthreads();
		if (tid == 0) {
			double S = 0.0, Cc = 0.0;
			for (int k = 0; k < nth; k++) {
				const double x = part_s[k];
				const double t = S + x;
				Cc += fabs(S) >= fabs(x) ? (S - t) + x : (x - t) + S;
				S = t;
				Cc += part_c[k];
			}
			b.Li[p] = S + Cc;
		}
	} else if (b.L) {
		// each thread sums a contiguous run of scored observations (Neumaier), then the
		// partials are combined in thread order by thread 0
		const int per = (b.nscored + nth - 1) / nth;
		const int k0 = tid * per, k1 = min(b.nscored, k0 + per);
		double s = 0.0, cmp = 0.0;
		for (int k = k0; k < k1; k++) {
			const int o = b.scored[k];
			const double lp = obs_prob(acc[k], m.obs_kind[o], m.obs_value[o], m.obs_model[o], m.obs_sd[o],
			                           m.obs_shape[o], m.obs_thresh[o]);
			const double t = s + lp;
			cmp += fabs(s) >= fabs(lp) ? (s - t) + lp : (lp - t) + s;
			s = t;
		}
		part_s[tid] = s;
		part_c[tid] = cmp;
		__syncthreads();
		if (tid == 0) {
			double S = 0.0, Cc = 0.0;
			for (int k = 0; k < nth; k++) {
				const double x = part_s[k];
				const double t = S + x;
				Cc += fabs(S) >= fabs(x) ? (S - t) + x : (x - t) + S;
				S = t;
				Cc += part_c[k];
			}
			const double L = S + Cc;
			if (L != L) set_status(status, BEEP_NAN_RATE);
			b.L[p] = L;
		}
	}
}

}  // namespace

namespace {

__global__ void __launch_bounds__(256) lgamma_table(double *t, int n)
{
	const int k = blockIdx.x * 256 + threadIdx.x;
	if (k < n) t[k] = lgamma((double)(k + 1));
}

template <typename PopT>
int launch_pop(const ModelDev &m, const BatchDev &b, cudaStream_t st)
{
	// the particle's arrays in shared memory where two CTAs per SM still fit (they leave the
	// chain of global loads between a step's phases); 512 threads per CTA when each SM holds
	// one particle anyway and a step has that many draws
	const size_t most = 104 * 1024;
	int level = 2;
	while (level > 0 && PlainSmem(m, (int)sizeof(PopT), level).total > most) level--;
	const size_t smem = PlainSmem(m, (int)sizeof(PopT), level).total;
	int dev = 0, sms = 0;
	cudaError_t e = cudaGetDevice(&dev);
	if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
	if (e == cudaSuccess) e = allow_dynamic_smem(sim_plain_kernel<PopT>, smem);
	if (e != cudaSuccess) return (int)e;
	const int nth = b.P <= sms && m.T * m.A * m.DP > 256 ? 512 : 256;
	sim_plain_kernel<PopT><<<b.P, nth, smem, st>>>(m, b, level, std::max(1, sms));
	return (int)cudaGetLastError();
}

}  // namespace

int launch_lgamma_table(double *t, int n, void *stream)
{
	lgamma_table<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(t, n);
	return (int)cudaGetLastError();
}

int launch_sim_plain(const ModelDev &m, const BatchDev &b, void *stream)
{
	if (b.P == 0) return 0;
	return m.ndcc > 0 ? launch_pop<double>(m, b, (cudaStream_t)stream) : launch_pop<int32_t>(m, b, (cudaStream_t)stream);
}

}  // namespace beep
