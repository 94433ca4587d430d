// beep_pf_loglik: the bootstrap particle filter of PMCMC on the device
// (PMCMC::obs_prob + bootstrap, src/pmcmc.cc:180-268; Mpi::end_sec_swap,
// src/mpi.cc:215-327).
//
// Per filter section, on the model's stream with no host round trip:
//   1. the simulation kernel (plain or fast form) advances every particle slot
//      from its carried population and writes the section log-likelihood L;
//   2. pf_bootstrap (one CTA) forms w = exp(invT (L - Lmax)), the cumulative
//      sums in slot order, the section's term invT Lmax + log(sum w / N), and the
//      ancestors: N uniforms (word 0 of Philox({j, section, stream, RESAMPLE})),
//      each located in the cumulative sums, then the reference's placement
//      (a selected particle keeps its own slot, the other slots take the
//      surplus selections last-in first-out);
//   3. the next section's kernel starts each slot from its ancestor's population
//      (BatchDev::pop_of).
// With a lineage request every section also writes its slots' transition
// counts, and the sampled particle's trajectory is assembled by walking the
// ancestors back (Mpi::particle_sample, src/mpi.cc:331-389).
// The cumulative sums are sequential in slot order and the placement gives the
// reference's slots, so the ancestors match it exactly (the FP64 weights of the
// plain form agree with the reference's to the last bits).
// The host stages a section's tables while the sections before it run.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "capi_internal.h"
#include "rng_fp64.cuh"

namespace beep {
namespace {

constexpr int kBootThreads = 1024;
constexpr int kBootSmemN = 8192;   // particles whose arrays fit shared memory

// Doubles >= 0 compare as their bits (the FP64 pipe takes 64 cycles per warp comparison)
__device__ __forceinline__ bool above(double x, double y) { return __double_as_longlong(x) > __double_as_longlong(y); }

// One CTA of up to 1024 threads (the particles, rounded up to warps).  Bound: the cumulative
// sums, N dependent FP64 additions of 64 cycles in the reference's order; the rest runs beside
// or around that chain in parallel -- the maximum and the search on the integer pipe, the
// placement as a scan: a selected particle keeps its slot, and the r-th free slot takes the
// r-th last of the draws that found their particle taken, which is what the reference's
// last-in first-out placement does one slot after another.  256 particles: 41.1 us with the
// placement on one thread and a 1024-thread tree for the maximum, 20.9 us now.  The arrays
// are in shared memory up to kBootSmemN particles (20 N bytes), in global scratch beyond.
__global__ void __launch_bounds__(kBootThreads) pf_bootstrap(const double *L, int N, double invT, uint32_t k0,
                                                            uint32_t k1, uint32_t rstream, int sec, double *wsum_g,
                                                            int32_t *sel_g, int32_t *first_g, int32_t *extra_g,
                                                            double *ob_sec, int32_t *anc, int32_t *status)
{
	extern __shared__ __align__(16) unsigned char boot_smem[];
	__shared__ long long s_max[kBootThreads / 32];
	__shared__ int32_t s_cnt[kBootThreads / 32];
	const bool sm = N <= kBootSmemN;
	double *wsum = sm ? (double *)boot_smem : wsum_g;
	int32_t *sel = sm ? (int32_t *)(boot_smem + 8 * (size_t)N) : sel_g;
	int32_t *first = sm ? sel + N : first_g;         // first draw that selected each particle
	int32_t *extra = sm ? first + N : extra_g;       // draws whose particle was taken, in draw order
	const int tid = threadIdx.x, nth = blockDim.x, lane = tid & 31, warp = tid >> 5, nwarp = nth >> 5;
	// the largest L, at least -LARGE (src/pmcmc.cc:223), as a 64-bit key in the doubles' order; NaN is passed by
	auto key = [](double x) { const long long v = __double_as_longlong(x); return v ^ ((v >> 63) & 0x7fffffffffffffffll); };
	long long mk = key(-1000000000.0);
	for (int p = tid; p < N; p += nth) {
		const double x = L[p];
		const long long v = __double_as_longlong(x);
		if ((unsigned long long)(v & 0x7fffffffffffffffll) <= 0x7ff0000000000000ull) mk = max(mk, key(x));
		first[p] = 0x7fffffff;
	}
	for (int o = 16; o > 0; o >>= 1) mk = max(mk, __shfl_xor_sync(0xffffffffu, mk, o));
	if (lane == 0) s_max[warp] = mk;
	__syncthreads();
	for (int k = 0; k < nwarp; k++) mk = max(mk, s_max[k]);
	const double Lmax = __longlong_as_double(mk ^ ((mk >> 63) & 0x7fffffffffffffffll));
	for (int p = tid; p < N; p += nth) wsum[p] = exp(invT * (L[p] - Lmax));
	__syncthreads();
	if (tid == 0) {
		double sum = 0.0;
#pragma unroll 8
		for (int p = 0; p < N; p++) {
			sum += wsum[p];
			wsum[p] = sum;
		}
	}
	__syncthreads();
	const double sum = wsum[N - 1];
	if (tid == nth - 1) ob_sec[sec] = invT * Lmax + log(sum / N);
	for (int j = tid; j < N; j += nth) {
		const U4 r = philox10(U4{(uint32_t)j, (uint32_t)sec, rstream, PURPOSE_RESAMPLE << 24}, k0, k1);
		const double z = u01_d(r.x) * sum;
		int lo = 0, hi = N;                          // first slot with wsum >= z
		if (z == z) {
			while (lo < hi) {
				const int mid = (lo + hi) >> 1;
				if (above(z, wsum[mid])) lo = mid + 1;
				else hi = mid;
			}
		}
		if (lo == N) { atomicCAS(status, 0, BEEP_NAN_RATE); lo = N - 1; }
		sel[j] = lo;
		atomicMin(first + lo, j);
	}
	__syncthreads();
	// ranks among the flagged of 0..N-1, in order, nth at a time
	auto rank = [&](bool flag, int32_t &base) {
		const unsigned vote = __ballot_sync(0xffffffffu, flag);
		if (lane == 0) s_cnt[warp] = __popc(vote);
		__syncthreads();
		int32_t r = base + __popc(vote & ((1u << lane) - 1u)), all = 0;
		for (int k = 0; k < nwarp; k++) {
			const int32_t c = s_cnt[k];
			if (k < warp) r += c;
			all += c;
		}
		base += all;
		__syncthreads();
		return r;
	};
	int32_t ne = 0, nf = 0;
	for (int j0 = 0; j0 < N; j0 += nth) {
		const int j = j0 + tid;
		const bool flag = j < N && first[sel[j]] != j;
		const int32_t r = rank(flag, ne);
		if (flag) extra[r] = sel[j];
	}
	__syncthreads();
	for (int p0 = 0; p0 < N; p0 += nth) {
		const int p = p0 + tid;
		const bool flag = p < N && first[p] == 0x7fffffff;
		const int32_t r = rank(flag, nf);
		if (p < N) anc[p] = flag ? extra[ne - 1 - r] : p;
	}
}

}  // namespace
}  // namespace beep

using namespace beep;

beep_status beep::pf_loglik(beep_model *m, const beep_pf_request *r, const std::function<void()> &ready)
{
	if (!m || !r || !r->tables) return fail(BEEP_BAD_INPUT, "null argument");
	const int N = r->nparticle, ns = r->nsection;
	if (N <= 0 || ns <= 0 || !r->section_ti || !r->section_tf || !r->loglik_out)
		return fail(BEEP_BAD_INPUT, "nparticle, sections and loglik_out are required");
	if (r->section_ti[0] != 0 || r->section_tf[ns - 1] != m->S)
		return fail(BEEP_BAD_INPUT, "sections must cover [0, ndivision)");
	for (int k = 0; k < ns; k++) {
		if (r->section_tf[k] <= r->section_ti[k]) return fail(BEEP_BAD_INPUT, "empty section");
		if (k > 0 && r->section_ti[k] != r->section_tf[k - 1]) return fail(BEEP_BAD_INPUT, "sections must be contiguous");
	}
	std::lock_guard<std::mutex> lock(m->mu);
	CUDA_TRY(cudaSetDevice(m->device));
	// populations as 32-bit words: one per population, or two (FP64 populations of a
	// model with demographic changes)
	const size_t popsz = (size_t)m->A * m->C * m->DP * (m->pop64 ? 2 : 1);
	cudaStream_t st = m->stream;

	// one prepared batch per section, kept on the model for later calls of the same
	// shape (then only the tables are staged again and the keys changed)
	const bool lineage = r->lineage_transnum_out != nullptr;
	beep_model::PfCache &pc = m->pf;
	auto drop_cache = [&]() {
		for (auto *x : pc.q) beep_batch_destroy(x);
		pc.q.clear();
		pc.N = 0;
		pc.form = -1;
	};
	const bool same = pc.N == N && pc.form == r->form && pc.lineage == lineage && (int)pc.q.size() == ns &&
	                  std::equal(pc.ti.begin(), pc.ti.end(), r->section_ti) &&
	                  std::equal(pc.tf.begin(), pc.tf.end(), r->section_tf);
	if (!same) {
		drop_cache();
		pc.q.assign(ns, nullptr);
		for (int k = 0; k < ns; k++) {
			beep_sim_batch b{};
			b.nparticle = N; b.ngroup = 1; b.groups = r->tables; b.seed = r->seed;
			b.ti = r->section_ti[k]; b.tf = r->section_tf[k];
			b.form = r->form;
			beep_status s = batch_create_internal(m, &b, true, &pc.q[k], lineage);
			if (s != BEEP_OK) { std::string e = beep_last_error(); drop_cache(); return fail(s, e); }
		}
		pc.N = N;
		pc.form = r->form;
		pc.lineage = lineage;
		pc.ti.assign(r->section_ti, r->section_ti + ns);
		pc.tf.assign(r->section_tf, r->section_tf + ns);
	}
	std::vector<beep_batch *> &q = pc.q;
	const size_t tnsz = (size_t)m->A * m->T * m->DP;
	Layout L;
	const size_t o_tn = L.add(lineage ? 4 * tnsz * (size_t)m->S * N : 0);
	const size_t o_pa = L.add(4 * popsz * N), o_pb = L.add(4 * popsz * N), o_L = L.add(8 * (size_t)ns * N),
	             o_ws = L.add(8 * (size_t)N), o_sel = L.add(4 * (size_t)N), o_fi = L.add(4 * (size_t)N),
	             o_ex = L.add(4 * (size_t)N), o_ob = L.add(8 * (size_t)ns), o_anc = L.add(4 * (size_t)ns * N),
	             o_pst = L.add(4 * ((size_t)ns * N + 1));
	if (pc.work.cap < L.size) pc.work.release(m->pool.get());   // (nothing is in flight between calls)
	cudaError_t e = pc.work.reserve(L.size, m->pool.get());
	if (e != cudaSuccess) { drop_cache(); return fail(BEEP_OOM, std::string("particle filter buffers: ") + cudaGetErrorString(e)); }
	if (ready) ready();
	char *d = (char *)pc.work.ptr;
	int32_t *pops[2] = {(int32_t *)(d + o_pa), (int32_t *)(d + o_pb)};   // the sections' final populations, in turn
	double *Lall = (double *)(d + o_L), *obsec = (double *)(d + o_ob);
	// the sections' per-particle statuses and, after them, the resampling's
	int32_t *anc = (int32_t *)(d + o_anc), *secst = (int32_t *)(d + o_pst), *pst = secst + (size_t)ns * N;
	beep_status status = BEEP_OK;
	std::string err;
	auto bail = [&](beep_status s, const std::string &msg) { status = s; err = msg; };
	if (cudaMemsetAsync(secst, 0, 4 * ((size_t)ns * N + 1), st) != cudaSuccess) bail(BEEP_DEVICE_ERROR, "memset");
	const size_t boot_smem = N <= kBootSmemN ? 20 * (size_t)N : 0;
	const int boot_threads = std::min(kBootThreads, (N + 31) / 32 * 32);
	if (status == BEEP_OK && allow_dynamic_smem(pf_bootstrap, boot_smem) != cudaSuccess)
		bail(BEEP_DEVICE_ERROR, "bootstrap shared memory");
	for (int k = 0; k < ns && status == BEEP_OK; k++) {
		beep_batch *b = q[k];
		if (same) {                              // prepared by an earlier call: this call's tables and key
			b->b.groups = r->tables;
			b->b.seed = r->seed;
			b->bd.k0 = (uint32_t)r->seed;
			b->bd.k1 = (uint32_t)(r->seed >> 32);
			// (every call waits for its copies before it returns: the staging buffer is free)
			const beep_status s = batch_stage_idle(b);
			if (s != BEEP_OK) { bail(s, beep_last_error()); break; }
		}
		if (beep_batch_upload(b) != BEEP_OK) { bail(BEEP_DEVICE_ERROR, beep_last_error()); break; }
		b->bd.pop_in = k > 0 ? pops[(k - 1) & 1] : nullptr;
		b->bd.pop_of = k > 0 ? anc + (size_t)(k - 1) * N : nullptr;
		b->bd.pop_out = pops[k & 1];
		b->bd.L = Lall + (size_t)k * N;
		b->bd.status = secst + (size_t)k * N;
		// section k's counts of every slot: [slot][step - ti][cell] at N * ti cells in
		if (lineage) b->bd.tn_traj = (int32_t *)(d + o_tn) + (size_t)N * r->section_ti[k] * tnsz;
		if (batch_launch_kernels(b) != BEEP_OK) { bail(BEEP_DEVICE_ERROR, beep_last_error()); break; }
		pf_bootstrap<<<1, boot_threads, boot_smem, st>>>(Lall + (size_t)k * N, N, r->invT, (uint32_t)r->seed,
		                                                 (uint32_t)(r->seed >> 32), r->resample_stream, k,
		                                                 (double *)(d + o_ws), (int32_t *)(d + o_sel),
		                                                 (int32_t *)(d + o_fi), (int32_t *)(d + o_ex), obsec,
		                                                 anc + (size_t)k * N, pst);
		if (cudaGetLastError() != cudaSuccess) bail(BEEP_DEVICE_ERROR, "bootstrap launch");
	}
	std::vector<double> ob(ns);
	std::vector<int32_t> ps((size_t)ns * N);
	int32_t bst = 0;
	if (status == BEEP_OK) {
		e = cudaMemcpyAsync(ob.data(), obsec, 8 * (size_t)ns, cudaMemcpyDeviceToHost, st);
		if (e == cudaSuccess) e = cudaMemcpyAsync(ps.data(), secst, 4 * (size_t)ns * N, cudaMemcpyDeviceToHost, st);
		if (e == cudaSuccess) e = cudaMemcpyAsync(&bst, pst, 4, cudaMemcpyDeviceToHost, st);
		if (e == cudaSuccess && r->L_out) e = cudaMemcpyAsync(r->L_out, Lall, 8 * (size_t)ns * N, cudaMemcpyDeviceToHost, st);
		if (e == cudaSuccess && r->ancestors_out)
			e = cudaMemcpyAsync(r->ancestors_out, anc, 4 * (size_t)ns * N, cudaMemcpyDeviceToHost, st);
		if (e == cudaSuccess) e = cudaStreamSynchronize(st);
		if (e != cudaSuccess) bail(BEEP_DEVICE_ERROR, cudaGetErrorString(e));
	}
	// per-particle statuses of the simulation launches
	for (int k = 0; k < ns && status == BEEP_OK; k++)
		for (int p = 0; p < N; p++)
			if (ps[(size_t)k * N + p] != 0) {
				bail((beep_status)ps[(size_t)k * N + p], "section " + std::to_string(k) + " particle " + std::to_string(p));
				break;
			}
	if (status == BEEP_OK && bst != 0) bail((beep_status)bst, "resampling found no particle (non-finite weights)");
	if (status == BEEP_OK && lineage) {
		// Mpi::particle_sample: start from the particle the last resampling put in slot
		// 0 and walk the ancestors back, copying each section from the slot its
		// ancestor held then
		std::vector<int32_t> a((size_t)ns * N);
		e = cudaMemcpy(a.data(), anc, 4 * (size_t)ns * N, cudaMemcpyDeviceToHost);
		int32_t pcur = a[(size_t)(ns - 1) * N + 0];
		for (int k = ns - 1; k >= 0 && e == cudaSuccess; k--) {
			const int ti = r->section_ti[k], nst = r->section_tf[k] - ti;
			const int32_t *src = (int32_t *)(d + o_tn) + ((size_t)N * ti + (size_t)pcur * nst) * tnsz;
			e = cudaMemcpy(r->lineage_transnum_out + (size_t)ti * tnsz, src, 4 * (size_t)nst * tnsz, cudaMemcpyDeviceToHost);
			if (k > 0) pcur = a[(size_t)(k - 1) * N + pcur];
		}
		if (e != cudaSuccess) bail(BEEP_DEVICE_ERROR, std::string("lineage copy: ") + cudaGetErrorString(e));
	}
	cudaStreamSynchronize(st);
	if (status != BEEP_OK) {
		drop_cache();
		return fail(status, err);
	}
	double total = 0.0;
	for (int k = 0; k < ns; k++) total += ob[k];
	*r->loglik_out = total;
	if (r->loglik_section_out) memcpy(r->loglik_section_out, ob.data(), 8 * (size_t)ns);
	return BEEP_OK;
}

size_t beep::pf_device_bytes(const beep_model *m)
{
	size_t n = m->pf.work.cap;
	for (const beep_batch *q : m->pf.q) n += batch_device_bytes(q);
	return n;
}

extern "C" BEEP_API beep_status beep_pf_loglik(beep_model *m, const beep_pf_request *r) { return pf_loglik(m, r, nullptr); }
