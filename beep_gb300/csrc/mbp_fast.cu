// MBP chains in the fast (mixed-precision) form: the fast kernel's chain
// variants (sim_fast.cuh with CH = true), compiled in their own translation
// unit.  A chain's two states hold, per step, the transition counts (int32)
// and means (FP32) of every column, [slot][chain][step][transition][column];
// the force of infection is formed from the counts every step, so Imap is not
// stored (INF_UPDATE and INF_DIF_UPDATE give the same map here).
#include <algorithm>

#include "sim_fast.cuh"

namespace beep {

int fast_chain_prepare()
{
	const int e = prepare_constants();
	return e != 0 ? e : fast_chain_ctas_prepare();
}

namespace {

template <int NT, int Q>
int launch_chain_q(const ModelDev &m, const BatchDev &b, size_t smem, cudaStream_t st)
{
	constexpr int MB = min_ctas(NT);
	auto kern = m.G <= 4 ? sim_fast_kernel<NT, 4, false, true, MB, kMaxT, false, Q>
	          : m.G <= 8 ? sim_fast_kernel<NT, 8, false, true, MB, kMaxT, false, Q>
	          : m.G <= 12 ? sim_fast_kernel<NT, 12, false, true, MB, kMaxT, false, Q>
	                      : sim_fast_kernel<NT, 16, false, true, MB, kMaxT, false, Q>;
	cudaError_t e = allow_dynamic_smem(kern, smem);
	if (e != cudaSuccess) return (int)e;
	kern<<<b.P, NT, smem, st>>>(m, b);
	return (int)cudaGetLastError();
}

template <int NT>
int launch_chain_nt(const ModelDev &m, const BatchDev &b, size_t smem, cudaStream_t st)
{
	return b.ch_queue ? launch_chain_q<NT, kQueueAlways>(m, b, smem, st) : launch_chain_q<NT, kQueueNever>(m, b, smem, st);
}

}  // namespace

int launch_sim_fast_chain(const ModelDev &m, const BatchDev &b_, void *stream)
{
	if (m.G > 16 || m.T > kMaxT || b_.foi_tc || !b_.ch_tn || !b_.ch_mean_f) return (int)cudaErrorInvalidValue;
	const int nt = b_.nt > 0 ? b_.nt : fast_pick_threads(m);
	size_t smem = fast_smem_bytes(m, b_.nslots, b_.m_in_smem != 0, b_.nefoi_stage, b_.gstate != nullptr,
	                              b_.tn_full ? m.T : m.tn_rows, b_.pop_single != 0, b_.tn_smem != 0, nt);
	// a proposal's draws are queued where that leaves the SM its chains at once (320-thread CTAs:
	// the layout's own number of them)
	BatchDev b = b_;
	int dev = 0, sms = 0;
	cudaError_t ce = cudaGetDevice(&dev);
	if (ce == cudaSuccess) ce = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
	if (ce != cudaSuccess) return (int)ce;
	const size_t queue = chain_queue_bytes(m.T, m.C, nt);
	const bool dual = nt == kDualThreads;
	const int most = dual ? b.ctas : min_ctas(nt), per_sm = dual ? b.ctas : (b.P + std::max(1, sms) - 1) / std::max(1, sms);
	b.ch_queue = b.mode == 1 && !b.simu_all && chain_queue_fits(smem, queue, most, per_sm) ? 1 : 0;
	if (b.ch_queue) smem += queue;
	if (nt == kDualThreads) return launch_sim_fast_chain_ctas(m, b, smem, stream);
	if (nt != fast_pick_threads(m)) return (int)cudaErrorInvalidValue;
	const int e = prepare_constants();
	if (e != 0) return e;
	cudaStream_t st = (cudaStream_t)stream;
	return nt == 128 ? launch_chain_nt<128>(m, b, smem, st) : nt == 256 ? launch_chain_nt<256>(m, b, smem, st)
	                                                                     : launch_chain_nt<640>(m, b, smem, st);
}

}  // namespace beep
