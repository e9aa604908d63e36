// PageRank on the GPU: fm::alg::PageRank (matrix/libmatrix-algs/
// PageRank.cpp:63-133) with the same float arithmetic, so that every vertex
// whose in-degree row is summed in the reference's order (at most
// FMX_EXACT_ROW_MAX entries) follows it bit for bit.
//
//   deg  = max(A 1, 1)                                (:49-59, :75)
//   pr   = 1.0 / n  (double, stored as float)         (:31-47, :80)
//   loop while converged < n and iters < max_iters    (:96-130):
//     in  = pr / deg;  pr1 = in * deg                 (:100-104)
//     out = A^T in                                    (:108, the transpose, :92)
//     pr2 = out * d + (1 - d) / n                     (:116-117, two roundings)
//     converged = #{ |pr1 - pr2| < 0.001 / n }        (:94, :118-123)
//     pr  = pr2
//
// One iteration of a small matrix is one pass: the SpMV on the transpose
// (k = 1) applies the damping, counts the converged vertices and writes the
// next input, and its hot pack, where it closes each row (rows summed in chunks
// by the warp whose chunk arrives last); the last block applies the loop test.
// Larger ones run the row kernel, its fixup and the update as a pass over the
// rows.  Input and pack are double-buffered (other rows still gather this
// iteration's while the next ones are written).  What bounds a small iteration
// is its kernels' latency: as four launches (pack, SpMV, fixup, loop test)
// R-MAT scale 16 took 27 us per iteration.  Iterations are queued in batches,
// one batch ahead of the host's read of the loop state; every kernel of an
// iteration queued after the loop ended returns at once, so the result and the
// count match a loop that tests on the host after every iteration.  A streamed
// matrix copies its entries for every queued iteration, so its batches are
// queued one at a time.
#include "fmx_internal.h"

#include <cuda_runtime.h>

#include <algorithm>
#include <vector>

namespace fmx {
namespace pagerank {

constexpr int kThreads = 256;
constexpr uint64_t kBatch = 8;          // iterations queued per host read of the loop state

#define PCUDA_TRY(call)                                                         \
	do {                                                                        \
		cudaError_t err__ = (call);                                             \
		if (err__ != cudaSuccess)                                               \
			return set_error(FMX_ERR_CUDA, "%s failed: %s (%s:%d)", #call,      \
					cudaGetErrorString(err__), __FILE__, __LINE__);             \
	} while (0)
#define P_TRY(call)                                                             \
	do {                                                                        \
		int rc__ = (call);                                                      \
		if (rc__ != FMX_OK) return rc__;                                        \
	} while (0)

__global__ void fill_kernel(float *p, int64_t n, float v)
{
	for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) p[i] = v;
}

// deg = max(deg, 1); pr = p0; in = pr / deg (and its slot of the hot pack);
// pr1 = in * deg
__global__ void init_kernel(float *__restrict__ deg, float *__restrict__ pr, float *__restrict__ in,
		float *__restrict__ pr1, const uint32_t *__restrict__ slot, float *__restrict__ xhot, int64_t n, float p0)
{
	for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
		const float d = fmaxf(deg[i], 1.0f);
		deg[i] = d;
		pr[i] = p0;
		const float x = __fdiv_rn(p0, d);
		in[i] = x;
		if (slot[i]) xhot[slot[i]] = x;
		pr1[i] = __fmul_rn(x, d);
	}
}

unsigned grid_for(int64_t n)
{
	int dev = 0, sms = 0;
	cudaGetDevice(&dev);
	cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
	return unsigned(std::max<int64_t>(1, std::min<int64_t>((n + kThreads - 1) / kThreads, int64_t(std::max(sms, 1)) * 8)));
}

} // namespace pagerank
} // namespace fmx

using namespace fmx;
using namespace fmx::pagerank;

extern "C" {

int fmx_pagerank(const fmx_matrix *m, uint64_t max_iters, float damping, float *pr, uint64_t *iters, void *stream)
{
	if (!m || !pr) return set_error(FMX_ERR_INVAL, "null argument");
	device_guard on_device(matrix_device(m));    // before the buffers: freed on the matrix's device
	if (!on_device.ok()) return set_error(FMX_ERR_CUDA, "cannot make the matrix's device %d current", matrix_device(m));
	uint64_t nr = 0, nc = 0, nz = 0;
	int prim = 0;
	P_TRY(fmx_matrix_info(m, &nr, &nc, &nz, &prim, nullptr));
	if (nr != nc) return set_error(FMX_ERR_DIM, "PageRank needs a square matrix");
	if (prim != FMX_P_BOOL && prim != FMX_P_FLOAT) return set_error(FMX_ERR_TYPE, "binary or float-weighted matrices");
	fmx_matrix *mt = nullptr;
	P_TRY(fmx_matrix_transpose(m, &mt));
	struct guard {
		fmx_matrix *t;
		cudaStream_t st;
		std::vector<void *> bufs;
		~guard()
		{
			for (void *p : bufs) cudaFreeAsync(p, st);
			fmx_matrix_free(t);
		}
	} g{mt, static_cast<cudaStream_t>(stream), {}};
	cudaStream_t st = g.st;
	const int64_t n = int64_t(nr);
	float *deg, *in0, *in1, *pr1, *xh0, *xh1, *out = nullptr;
	uint32_t *mask, *arrived, *chunk_heavy;
	unsigned long long *state;
	auto alloc = [&](void **q, size_t bytes) -> int {
		cudaError_t e = work_alloc(q, std::max<size_t>(bytes, 16), st);
		if (e != cudaSuccess) return set_error(FMX_ERR_OOM, "PageRank vectors: %s", cudaGetErrorString(e));
		g.bufs.push_back(*q);
		return FMX_OK;
	};
	const size_t mask_words = size_t((n + 31) / 32);
	for (float **b : {&deg, &in0, &in1, &pr1}) P_TRY(alloc(reinterpret_cast<void **>(b), size_t(n) * sizeof(float)));
	// one block of zeroed words: the loop state, the two hot packs (their slot
	// 0 stays zero), the mask and the arrival counts
	uint64_t n_hot = 0, n_heavy = 0, n_chunks = 0;
	pagerank_sizes(mt, &n_hot, &n_heavy, &n_chunks);
	const size_t pack = size_t(n_hot) + 1;
	const size_t zbytes = 8 * sizeof(unsigned long long) + (2 * pack + mask_words + n_heavy) * sizeof(uint32_t);
	P_TRY(alloc(reinterpret_cast<void **>(&state), zbytes));
	P_TRY(alloc(reinterpret_cast<void **>(&chunk_heavy), n_chunks * sizeof(uint32_t)));
	xh0 = reinterpret_cast<float *>(state + 8);
	xh1 = xh0 + pack;
	mask = reinterpret_cast<uint32_t *>(xh1 + pack);
	arrived = mask + mask_words;
	if (pagerank_needs_out(mt)) P_TRY(alloc(reinterpret_cast<void **>(&out), size_t(n) * sizeof(float)));
	// the loop state comes back through pinned words per host thread, one set
	// per batch in flight
	struct host_state { unsigned long long w[2 * 4]; };
	static thread_local thread_pinned<host_state> pinned;
	host_state *hs = nullptr;
	PCUDA_TRY(pinned.get(&hs));
	unsigned long long *hstate = hs->w;
	const unsigned gb = grid_for(n);
	fill_kernel<<<gb, kThreads, 0, st>>>(in1, n, 1.0f);
	PCUDA_TRY(cudaGetLastError());
	P_TRY(fmx_spmm(m, FMX_F32, in1, 1, FMX_F32, deg, 1, 1, nullptr, nullptr, st));
	const float p0 = float(1.0 / double(n));
	pr_epi e{};
	e.deg = deg;
	e.heavy_mask = mask;
	e.chunk_heavy = chunk_heavy;
	e.arrived = arrived;
	e.pr = pr;
	e.pr1 = pr1;
	e.state = state;
	e.damping = damping;
	e.teleport = float((1.0 - double(damping)) / double(n));
	e.eps = float(0.001 / double(n));
	e.n = uint64_t(n);
	e.max_iters = max_iters;
	PCUDA_TRY(cudaMemsetAsync(state, 0, zbytes, st));
	P_TRY(pagerank_maps(mt, mask, chunk_heavy, &e.slot, &e.heavy, st));
	init_kernel<<<gb, kThreads, 0, st>>>(deg, pr, in0, pr1, e.slot, xh0, n, p0);
	PCUDA_TRY(cudaGetLastError());
	struct events {
		cudaEvent_t e[2] = {nullptr, nullptr};
		~events() { for (cudaEvent_t x : e) if (x) cudaEventDestroy(x); }
	} ev;
	for (cudaEvent_t &x : ev.e) PCUDA_TRY(cudaEventCreateWithFlags(&x, cudaEventDisableTiming));
	const uint64_t ahead = pagerank_streamed(mt) ? 1 : 2;
	uint64_t it = 0, queued = 0, batches = 0, read = 0;
	bool done = n == 0 || max_iters == 0;
	while (!done) {
		// queue a batch, then read the state of the one before (of itself when streamed)
		if (queued < max_iters) {
			const uint64_t batch = std::min<uint64_t>(kBatch, max_iters - queued);
			for (uint64_t b = 0; b < batch; b++, queued++) {
				const bool odd = queued & 1;
				e.in_next = odd ? in0 : in1;
				e.xhot_next = odd ? xh0 : xh1;
				P_TRY(pagerank_iteration(mt, odd ? in1 : in0, odd ? xh1 : xh0, out, e, st));
			}
			PCUDA_TRY(cudaMemcpyAsync(hstate + 4 * (batches & 1), state, 4 * sizeof(unsigned long long), cudaMemcpyDeviceToHost, st));
			PCUDA_TRY(cudaEventRecord(ev.e[batches & 1], st));
			batches++;
			if (batches - read < ahead && queued < max_iters) continue;
		}
		PCUDA_TRY(cudaEventSynchronize(ev.e[read & 1]));
		it = hstate[4 * (read & 1) + 2];
		done = hstate[4 * (read & 1) + 1] || (++read == batches && queued >= max_iters);
	}
	PCUDA_TRY(cudaStreamSynchronize(st));
	if (iters) *iters = it;
	return FMX_OK;
}

} // extern "C"
