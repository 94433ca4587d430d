// The buffer pools (capi_internal.h) over a driver of a given capacity, for the tests: the four
// calls they make, counted.
#include "capi_internal.h"

#include <cstdlib>
#include <map>
#include <thread>

namespace {
struct Driver {
	std::mutex mu;
	size_t capacity[2] = {0, 0}, used[2] = {0, 0};
	std::map<void *, std::pair<int, size_t>> live;
	int errors = 0;
	cudaError_t last = cudaSuccess;
	cudaError_t alloc(int host, void **p, size_t n)
	{
		std::lock_guard<std::mutex> lk(mu);
		if (used[host] + n > capacity[host]) return last = cudaErrorMemoryAllocation;
		used[host] += n;
		*p = malloc(1);
		live[*p] = {host, n};
		return cudaSuccess;
	}
	cudaError_t free_(int host, void *p)
	{
		std::lock_guard<std::mutex> lk(mu);
		auto it = live.find(p);
		if (it == live.end() || it->second.first != host) {   // released twice, or as the other kind
			errors++;
			return cudaErrorInvalidValue;
		}
		used[host] -= it->second.second;
		live.erase(it);
		free(p);
		return cudaSuccess;
	}
} drv;

void reset(size_t device, size_t host)
{
	for (auto &kv : drv.live) free(kv.first);            // (of a case that ended early)
	drv.live.clear();
	drv.used[0] = drv.used[1] = 0;
	drv.capacity[0] = device;
	drv.capacity[1] = host;
	drv.errors = 0;
	drv.last = cudaSuccess;
}

using namespace beep;
constexpr size_t kMB = (size_t)1 << 20;

#define EXPECT(c)                                                                                                      \
	do {                                                                                                                 \
		if (!(c)) return __LINE__;                                                                                         \
	} while (0)
}  // namespace

extern "C" {

cudaError_t cudaMalloc(void **p, size_t n) { return drv.alloc(0, p, n); }
cudaError_t cudaMallocHost(void **p, size_t n) { return drv.alloc(1, p, n); }
cudaError_t cudaFree(void *p) { return drv.free_(0, p); }
cudaError_t cudaFreeHost(void *p) { return drv.free_(1, p); }
cudaError_t cudaGetLastError()
{
	const cudaError_t e = drv.last;
	drv.last = cudaSuccess;
	return e;
}

// each returns 0, or the line of the first expectation that does not hold

int spare_of_other_pools_is_given_up()
{
	reset(100 * kMB, 100 * kMB);
	{
		BufPool a(64 * kMB), b(64 * kMB);
		DevBuf x, y;
		HostBuf h;
		EXPECT(x.reserve(40 * kMB, &a) == cudaSuccess && y.reserve(40 * kMB, &b) == cudaSuccess);
		EXPECT(h.reserve(60 * kMB, &a) == cudaSuccess);
		x.release(&a);
		h.release(&a);
		EXPECT(drv.used[0] == 80 * kMB && drv.used[1] == 60 * kMB);       // kept by a
		DevBuf z;                                                         // chains, weights: no pool
		EXPECT(z.reserve(50 * kMB) == cudaSuccess && drv.used[0] == 90 * kMB);
		z.release();
		HostBuf g;                                                        // another pool's request
		EXPECT(g.reserve(90 * kMB, &b) == cudaSuccess);
		g.release(&b);
		y.release(&b);
		EXPECT(x.reserve(90 * kMB, &a) == cudaSuccess);
		x.release(&a);
	}
	EXPECT(drv.used[0] == 0 && drv.used[1] == 0 && drv.errors == 0);
	return 0;
}

int a_failed_allocation_leaves_nothing_behind()
{
	reset(100 * kMB, 0);
	BufPool a(64 * kMB);
	DevBuf x;
	EXPECT(x.reserve(60 * kMB, &a) == cudaSuccess);
	DevBuf y, z;
	EXPECT(y.reserve(60 * kMB, &a) == cudaErrorMemoryAllocation && !y.ptr && y.cap == 0);
	EXPECT(drv.last == cudaSuccess);                                    // no error left for a later launch
	EXPECT(z.reserve(60 * kMB) == cudaErrorMemoryAllocation && !z.ptr && drv.last == cudaSuccess);
	x.release(&a);
	EXPECT(y.reserve(60 * kMB) == cudaSuccess);
	y.release();
	EXPECT(drv.used[0] == 0 && drv.errors == 0);
	return 0;
}

int a_pool_keeps_its_limit_and_trims_the_oldest()
{
	reset((size_t)4096 * kMB, (size_t)4096 * kMB);
	BufPool a(256 * kMB);
	DevBuf x[4];
	const size_t n[4] = {100 * kMB, 120 * kMB, 80 * kMB, 300 * kMB};
	for (int k = 0; k < 4; k++) EXPECT(x[k].reserve(n[k], &a) == cudaSuccess && x[k].cap >= n[k] && x[k].cap <= n[k] + n[k] / 8 + 4096);
	const size_t c0 = x[0].cap, c1 = x[1].cap;
	for (auto &b : x) b.release(&a);
	EXPECT(a.device_bytes() == c0 + c1 && drv.used[0] == c0 + c1);      // the third and fourth went to the driver
	a.trim(c1);
	EXPECT(a.device_bytes() == c1);
	EXPECT(x[0].reserve(20 * kMB, &a) == cudaSuccess && a.device_bytes() == c1);   // too large a spare for 20 MB
	EXPECT(x[1].reserve(110 * kMB, &a) == cudaSuccess && x[1].cap == c1 && a.device_bytes() == 0);
	x[0].release(&a);
	x[1].release(&a);
	a.trim(0);
	EXPECT(drv.used[0] == 0 && drv.errors == 0);
	return 0;
}

int large_buffers_take_what_they_ask_for()
{
	reset((size_t)270000 * kMB, (size_t)100000 * kMB);
	{
		BufPool a(256 * kMB), server((size_t)200000 * kMB);
		for (BufPool *pool : {&a, &server})
			for (size_t n : {(size_t)270000 * kMB, (size_t)131073 * kMB, (size_t)33 * kMB + 1, (size_t)5 * kMB + 7}) {
				DevBuf x;
				EXPECT(x.reserve(n, pool) == cudaSuccess && x.cap - n < 2 * kMB);
				x.release();
			}
		HostBuf h;
		EXPECT(h.reserve((size_t)100000 * kMB, &a) == cudaSuccess);
		h.release();
	}
	EXPECT(drv.used[0] == 0 && drv.used[1] == 0 && drv.errors == 0);
	return 0;
}

int threads_share_pools_of_a_full_device()
{
	reset(64 * kMB, 64 * kMB);
	{
		BufPool shared(32 * kMB);
		std::vector<std::thread> th;
		for (int t = 0; t < 8; t++)
			th.emplace_back([&shared, t] {
				for (int k = 0; k < 400; k++) {
					BufPool own(4 * kMB);
					BufPool *pool = k % 3 ? &shared : &own;
					DevBuf d, e;
					HostBuf h;
					if (d.reserve((1 + (k * 7 + t) % 6) * kMB, pool) == cudaSuccess) d.release(pool);
					if (e.reserve((1 + (k + t) % 4) * kMB) == cudaSuccess) e.release();
					if (h.reserve((1 + (k * 5 + t) % 6) * kMB, pool) == cudaSuccess) h.release(pool);
				}
			});
		for (auto &t : th) t.join();
	}
	EXPECT(drv.used[0] == 0 && drv.used[1] == 0 && drv.errors == 0);
	return 0;
}

}  // extern "C"
