// Host-side definitions shared by the C-ABI translation units: error text,
// growable device/host buffers, buffer layouts and the model handle.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <functional>
#include <memory>
#include <mutex>
#include <string>
#include <vector>

#include "beep_internal.h"

namespace beep {

// Records the message returned by beep_last_error() on this thread.
beep_status fail(beep_status s, const std::string &msg);

#define CUDA_TRY(expr)                                                                         \
	do {                                                                                       \
		cudaError_t e_ = (expr);                                                               \
		if (e_ != cudaSuccess)                                                                 \
			return ::beep::fail(e_ == cudaErrorMemoryAllocation ? BEEP_OOM : BEEP_DEVICE_ERROR, \
			                    std::string(#expr) + ": " + cudaGetErrorString(e_));           \
	} while (0)

inline size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

// Device and pinned buffers of destroyed batches and models, kept for the next ones: an
// allocation, and above all a release, of either kind costs 0.1 to 1 ms and waits for the
// whole device.  What pools keep never makes an allocation fail: one that does is tried again
// with every pool of the process emptied (driver_alloc).  A pool belongs to a model (its batches come and go, one per beep_simulate)
// or to a server (models and batches per request); it keeps at most `limit` bytes of each kind
// and goes with its last owner.  Buffers are given back only when no work that uses them is
// left in flight.  Safe from several threads.
class BufPool {
public:
	explicit BufPool(size_t limit) : limit_(limit)
	{
		std::lock_guard<std::mutex> lk(all().mu);
		all().pools.push_back(this);
	}
	~BufPool()
	{
		{
			std::lock_guard<std::mutex> lk(all().mu);
			all().pools.erase(std::find(all().pools.begin(), all().pools.end(), this));
		}
		trim(0);
	}
	BufPool(const BufPool &) = delete;
	BufPool &operator=(const BufPool &) = delete;
	cudaError_t take(bool host, size_t n, void **ptr, size_t *cap)
	{
		// sizes in steps of 1/8 of their power of two, so that batches of near sizes share buffers;
		// at most 2 MiB, the driver's own granularity, so that a batch fits where its bytes do
		size_t step = 4096;
		while (step * 16 < n && step < (size_t)2 << 20) step *= 2;
		n = align_up(n, step);
		{
			std::lock_guard<std::mutex> lk(mu_);
			std::vector<Buf> &v = spare_[host];
			size_t best = v.size();
			for (size_t k = 0; k < v.size(); k++)
				if (v[k].cap >= n && v[k].cap / 4 <= n && (best == v.size() || v[k].cap < v[best].cap)) best = k;
			if (best < v.size()) {
				*ptr = v[best].ptr;
				*cap = v[best].cap;
				bytes_[host] -= v[best].cap;
				v.erase(v.begin() + best);
				return cudaSuccess;
			}
		}
		const cudaError_t e = driver_alloc(host, n, ptr);
		*cap = e == cudaSuccess ? n : 0;
		return e;
	}
	// Memory from the driver; where there is none left, every pool gives its spare buffers back
	// first.
	static cudaError_t driver_alloc(bool host, size_t n, void **ptr)
	{
		cudaError_t e = host ? cudaMallocHost(ptr, n) : cudaMalloc(ptr, n);
		if (e == cudaErrorMemoryAllocation) {
			cudaGetLastError();
			{
				std::lock_guard<std::mutex> lk(all().mu);
				for (BufPool *p : all().pools) p->trim(0);
			}
			e = host ? cudaMallocHost(ptr, n) : cudaMalloc(ptr, n);
			if (e == cudaErrorMemoryAllocation) cudaGetLastError();   // (the caller's to report, not a later launch's)
		}
		if (e != cudaSuccess) *ptr = nullptr;
		return e;
	}
	void give(bool host, void *ptr, size_t cap)
	{
		{
			std::lock_guard<std::mutex> lk(mu_);
			if (bytes_[host] + cap <= limit_ && spare_[host].size() < 256) {
				spare_[host].push_back(Buf{ptr, cap});
				bytes_[host] += cap;
				return;
			}
		}
		drop(host, ptr);
	}
	// releases spare buffers, the oldest first, until at most `keep` bytes of each kind are left
	void trim(size_t keep)
	{
		for (int host = 0; host < 2; host++)
			for (;;) {
				void *p = nullptr;
				{
					std::lock_guard<std::mutex> lk(mu_);
					if (bytes_[host] <= keep || spare_[host].empty()) break;
					p = spare_[host].front().ptr;
					bytes_[host] -= spare_[host].front().cap;
					spare_[host].erase(spare_[host].begin());
				}
				drop(host != 0, p);
			}
	}
	size_t device_bytes()
	{
		std::lock_guard<std::mutex> lk(mu_);
		return bytes_[0];
	}

private:
	// the pools of the process (never destroyed: a pool may outlive the library's statics)
	struct All {
		std::mutex mu;
		std::vector<BufPool *> pools;
	};
	static All &all()
	{
		static All *a = new All;
		return *a;
	}
	struct Buf {
		void *ptr;
		size_t cap;
	};
	static void drop(bool host, void *p)
	{
		if (host) cudaFreeHost(p);
		else cudaFree(p);
	}
	std::mutex mu_;
	std::vector<Buf> spare_[2];          // [0] device, [1] pinned host
	size_t bytes_[2] = {0, 0}, limit_;
};

// A buffer that only grows, from a pool or from the driver.  (What it held when it grows goes
// back to the driver, which waits for the work that may still read it.)
template <bool HOST>
struct GrowBuf {
	void *ptr = nullptr;
	size_t cap = 0;
	cudaError_t reserve(size_t n, BufPool *pool = nullptr)
	{
		if (n <= cap) return cudaSuccess;
		release();
		if (pool) return pool->take(HOST, n, &ptr, &cap);
		const cudaError_t e = BufPool::driver_alloc(HOST, n, &ptr);
		if (e == cudaSuccess) cap = n;
		return e;
	}
	void release(BufPool *pool = nullptr)
	{
		if (ptr && pool) pool->give(HOST, ptr, cap);
		else if (ptr && HOST) cudaFreeHost(ptr);
		else if (ptr) cudaFree(ptr);
		ptr = nullptr;
		cap = 0;
	}
};
using DevBuf = GrowBuf<false>;
using HostBuf = GrowBuf<true>;
constexpr size_t kModelPoolBytes = (size_t)256 << 20;   // spare bytes a model keeps, of each kind

// Sequential layout of named regions inside one buffer (256-byte aligned).
struct Layout {
	size_t size = 0;
	size_t add(size_t bytes)
	{
		size_t off = align_up(size, 256);
		size = off + bytes;
		return off;
	}
};

// Scored observations of a step range and the steps each is active in
// (positions into `scored`), as the kernels consume them.
struct ObsLists {
	std::vector<int32_t> scored, step_ptr, step_obs;
};
void build_obs_lists(const int32_t *sett_i, const int32_t *sett_f, int nobs, int ti, int tf, ObsLists &out);

}  // namespace beep

struct beep_model {
	int device = 0;
	int sms = 152;                // SMs of the device
	cudaStream_t stream = nullptr;
	beep::ModelDev dev{};
	std::shared_ptr<beep::BufPool> pool;   // its batches' buffers
	beep::DevBuf model_mem;
	// host copies used to prepare batches
	int32_t A, G, DP, NS, C, T, S, period, dpt, nobs;
	std::vector<int32_t> obs_sett_i, obs_sett_f, obs_spline, trans_from_h, trans_to_h, obs_cell_ptr_h, obs_cells_f_h,
	    obs_cells_full_h;
	std::vector<float> obs_factor_f_h;
	int32_t max_obs_spline = -1;
	bool pop64 = false;           // demographic changes: populations are FP64 (plain form only)
	int32_t tuned_foi = 0;        // fast-form FOI path chosen by beep_autotune (0: none)
	int32_t tuned_ctas = 0;       // fast-form particles per SM chosen by beep_autotune (0: none)
	// beep_pf_loglik's prepared section batches and buffers, kept while later calls
	// have the same particles, sections, form and lineage request (PMCMC calls it
	// once per proposal with new tables only)
	struct PfCache {
		int32_t N = 0, form = -1;
		bool lineage = false;
		std::vector<int32_t> ti, tf;
		std::vector<beep_batch *> q;
		beep::DevBuf work;
	} pf;
	std::mutex mu;
};

// A prepared batch: the caller's host arrays (kept by pointer), pinned staging,
// device inputs, work and outputs, and the kernel's view of them.
struct beep_batch {
	bool device_io = false;   // pop_in / L / pop_out are device buffers set by an internal caller
	beep_model *m = nullptr;
	beep_sim_batch b{};
	beep::HostBuf in_host, out_host;
	beep::DevBuf in_dev, work_dev, out_dev;
	size_t in_size = 0, out_size = 0;
	size_t o_f = 0, u_st = 0, u_L = 0, u_po = 0, u_tn = 0, u_pt = 0;
	std::vector<beep::GroupDir> dirs;
	std::vector<uint2> keys;           // per-particle Philox keys (requests packed into one batch), or empty
	std::vector<int32_t> scored, step_ptr, step_obs, slot_of, tasks;
	beep::BatchDev bd{};
	cudaEvent_t ev0 = nullptr, ev1 = nullptr;
	bool pending = false;
	bool state_global = false;   // fast form keeps particle state in global memory
	std::vector<cudaEvent_t> ev_split;   // beep_batch_time_split: around each step's product kernel
	// CUDA graph of upload + status reset + kernel + download (beep_batch_run_graph)
	cudaGraph_t graph = nullptr;
	cudaGraphExec_t graph_exec = nullptr;
	size_t graph_in_size = 0;
	beep::BatchDev graph_bd{};   // the arguments it was captured with
	int32_t nefoi_layout = 0;    // external-force tables the fast form's shared-memory layout holds
};


namespace beep {
// beep_model_create with the model's and its batches' buffers from a pool shared with others.
beep_status model_create_internal(const beep_model_desc *d, std::shared_ptr<BufPool> pool, beep_model **out);
// beep_batch_create for internal callers whose start populations and outputs
// live on the device (device_io: pop_in is not read from the host and the
// caller sets bd.pop_in / bd.L / bd.pop_out before each launch).
// With device_traj the kernels write every step's transition counts to a
// device buffer the caller sets in bd.tn_traj ([P][tf-ti][A][T][DP]) before
// each launch.
// allow_tc = false keeps the fast form's force of infection on FP32 SIMT;
// allow_ctas = false keeps it at one particle per SM.
// keys (may be null): one Philox key per particle, for batches that pack the
// particles of requests with different seeds.
beep_status batch_create_internal(beep_model *m, const beep_sim_batch *b, bool device_io, beep_batch **out,
                                  bool device_traj = false, bool allow_tc = true, bool allow_ctas = true,
                                  const std::vector<uint2> *keys = nullptr);
// beep_batch_stage for a caller whose copies from the staging buffer have completed (no wait).
beep_status batch_stage_idle(beep_batch *q);
// beep_batch_launch for a caller that has cleared bd.status itself.
beep_status batch_launch_kernels(beep_batch *q);
// beep_batch_download in two halves: the device->host copy enqueued on the
// model's stream, and (once that copy completed) the status check and the
// copy into the caller's arrays.
beep_status batch_download_enqueue(beep_batch *q);
beep_status batch_download_finish(beep_batch *q);
// beep_pf_loglik; ready (may be null) is called once its device buffers are in place, before
// the sections are launched.
beep_status pf_loglik(beep_model *m, const beep_pf_request *r, const std::function<void()> &ready);
// Device bytes held by a model / a batch / a model's filter.
size_t model_device_bytes(const beep_model *m);
size_t batch_device_bytes(const beep_batch *q);
size_t pf_device_bytes(const beep_model *m);
}  // namespace beep
