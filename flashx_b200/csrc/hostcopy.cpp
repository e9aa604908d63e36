// Copies between pageable host memory and the device for fmx_spmm_host, the
// call a FlashMatrix program makes on its own buffers.
//
// The driver moves pageable memory through its own pinned buffer with one host
// thread: 16.8 MB took 785 us in and 770 us out (21 GB/s) where the link moves
// pinned memory in 305 us.  Here several host threads copy chunks into pinned
// slots and enqueue them (143 us for 16.8 MB on 8 threads), so a direction runs
// at the link's rate; the same threads bring the result out.
//
// The slots (kBounceThreads x 2 x kBounceChunk = 8 MB) belong to the process,
// one set per device, allocated by the first call that needs them, used by one
// call at a time (a call that finds them taken copies directly) and handed
// back by fmx_release_cached.  The threads live for one call.
#include "fmx_internal.h"

#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstring>
#include <mutex>
#include <system_error>
#include <thread>
#include <vector>

namespace fmx {
namespace {

constexpr int kBounceThreads = 8;
constexpr size_t kBounceChunk = size_t(512) << 10;
constexpr size_t kBounceMin = size_t(1) << 20;       // bytes a copy must have for the threads to pay

struct slots {
	std::mutex mu;                                   // held by the call that uses the slots
	char *buf = nullptr;
	cudaEvent_t ev[2 * kBounceThreads] = {};

	int get()
	{
		if (buf) return FMX_OK;
		for (cudaEvent_t &e : ev)
			if (!e && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess)
				return set_error(FMX_ERR_CUDA, "event creation failed");
		void *p = nullptr;
		if (cudaHostAlloc(&p, 2 * kBounceThreads * kBounceChunk, cudaHostAllocDefault) != cudaSuccess) {
			cudaGetLastError();
			return set_error(FMX_ERR_OOM, "pinned copy slots: out of host memory");
		}
		buf = static_cast<char *>(p);
		return FMX_OK;
	}
};

slots *device_slots(int device)
{
	static slots *all = new slots[64];               // outlives every static destructor
	return device >= 0 && device < 64 ? &all[device] : nullptr;
}

// Rows of `width` bytes, `pitch` apart on the host and back to back on the
// device, in chunks of whole rows (or of bytes when the host rows are back to
// back too).
struct chunks {
	char *dev = nullptr, *host = nullptr;
	size_t width = 0, pitch = 0, unit = 0, total = 0, count = 0, per = 0;

	explicit chunks(const host_copy *c)
	{
		if (!c) return;
		dev = static_cast<char *>(c->dev);
		host = static_cast<char *>(c->host);
		width = c->width;
		pitch = c->pitch;
		const bool flat = pitch == width;
		unit = flat ? 1 : width;
		total = flat ? c->width * c->rows : c->rows;     // in units
		per = std::max<size_t>(1, kBounceChunk / unit);
		count = (total + per - 1) / per;
	}
	void span(size_t c, size_t &u0, size_t &n) const
	{
		u0 = c * per;
		n = std::min(per, total - u0);
	}
	void gather(size_t u0, size_t n, char *slot) const
	{
		if (unit == 1) memcpy(slot, host + u0, n);
		else for (size_t r = 0; r < n; r++) memcpy(slot + r * width, host + (u0 + r) * pitch, width);
	}
	void scatter(size_t u0, size_t n, const char *slot) const
	{
		if (unit == 1) memcpy(host + u0, slot, n);
		else for (size_t r = 0; r < n; r++) memcpy(host + (u0 + r) * pitch, slot + r * width, width);
	}
};

struct job {
	chunks in, out;
	slots *s;
	cudaStream_t st;
	int device;
	std::atomic<size_t> next_in{0}, next_out{0};
	std::atomic<int> failed{0};
	std::mutex mu;
	std::condition_variable cv;
	int arrived = 0, go = 0;                         // go: 1 bring the result out, -1 stop

	job(const host_copy *i, const host_copy *o, slots *sl, cudaStream_t stream, int dev)
		: in(i), out(o), s(sl), st(stream), device(dev) {}

	char *slot(int t, int b) const { return s->buf + size_t(2 * t + b) * kBounceChunk; }

	void copy_in(int t)
	{
		bool used[2] = {false, false};
		for (int i = 0; !failed; i++) {
			const size_t c = next_in++;
			if (c >= in.count) break;
			const int b = i & 1;
			cudaEvent_t ev = s->ev[2 * t + b];
			if (used[b] && cudaEventSynchronize(ev) != cudaSuccess) { failed = 1; break; }
			size_t u0, n;
			in.span(c, u0, n);
			in.gather(u0, n, slot(t, b));
			if (cudaMemcpyAsync(in.dev + u0 * in.unit, slot(t, b), n * in.unit, cudaMemcpyHostToDevice, st) != cudaSuccess ||
					cudaEventRecord(ev, st) != cudaSuccess)
				failed = 1;
			used[b] = true;
		}
	}
	// two chunks of a thread in flight; the slots' earlier copies precede on `st`
	void copy_out(int t)
	{
		size_t at[2], n[2];
		bool live[2] = {false, false};
		auto issue = [&](int b) {
			live[b] = false;
			if (failed) return;
			const size_t c = next_out++;
			if (c >= out.count) return;
			out.span(c, at[b], n[b]);
			if (cudaMemcpyAsync(slot(t, b), out.dev + at[b] * out.unit, n[b] * out.unit, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
					cudaEventRecord(s->ev[2 * t + b], st) != cudaSuccess) {
				failed = 1;
				return;
			}
			live[b] = true;
		};
		issue(0);
		issue(1);
		for (int b = 0; live[b]; b ^= 1) {
			if (cudaEventSynchronize(s->ev[2 * t + b]) != cudaSuccess) { failed = 1; return; }
			out.scatter(at[b], n[b], slot(t, b));
			issue(b);
		}
	}
	void worker(int t)
	{
		if (cudaSetDevice(device) != cudaSuccess) failed = 1;
		copy_in(t);
		{
			std::unique_lock<std::mutex> g(mu);
			arrived++;
			cv.notify_all();
			cv.wait(g, [&] { return go != 0; });
			if (go < 0) return;
		}
		copy_out(t);
	}
};

bool pageable(const void *p)
{
	cudaPointerAttributes a = {};
	if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
		cudaGetLastError();
		return true;
	}
	return a.type == cudaMemoryTypeUnregistered;
}

} // namespace

int run_host_copies(int device, cudaStream_t st, const host_copy &in, const host_copy &out, const std::function<int()> &run)
{
	auto direct = [&](const host_copy &c, cudaMemcpyKind kind) -> int {
		void *dst = kind == cudaMemcpyHostToDevice ? c.dev : c.host;
		const void *src = kind == cudaMemcpyHostToDevice ? c.host : c.dev;
		// one linear copy when the rows are contiguous (a pitched copy of
		// 64-byte rows moves far below the link rate)
		const cudaError_t e = c.pitch == c.width ? cudaMemcpyAsync(dst, src, c.width * c.rows, kind, st)
				: kind == cudaMemcpyHostToDevice ? cudaMemcpy2DAsync(dst, c.width, src, c.pitch, c.width, c.rows, kind, st)
				                                 : cudaMemcpy2DAsync(dst, c.pitch, src, c.width, c.width, c.rows, kind, st);
		if (e == cudaSuccess) return FMX_OK;
		return kind == cudaMemcpyHostToDevice ? set_error(FMX_ERR_CUDA, "copy of X to the device failed")
				: set_error(FMX_ERR_CUDA, "copy of Y to the host failed");
	};
	const bool bi = in.width * in.rows >= kBounceMin && in.width <= kBounceChunk && pageable(in.host);
	const bool bo = out.width * out.rows >= kBounceMin && out.width <= kBounceChunk && pageable(out.host);
	slots *s = bi || bo ? device_slots(device) : nullptr;
	std::unique_lock<std::mutex> hold;
	if (s) {
		hold = std::unique_lock<std::mutex>(s->mu, std::try_to_lock);
		if (!hold.owns_lock() || s->get() != FMX_OK) s = nullptr;
	}
	if (!s) {
		if (int rc = direct(in, cudaMemcpyHostToDevice)) return rc;
		if (int rc = run()) return rc;
		return direct(out, cudaMemcpyDeviceToHost);
	}
	job j(bi ? &in : nullptr, bo ? &out : nullptr, s, st, device);
	const size_t most = std::max(j.in.count, j.out.count);
	const int nt = int(std::min<size_t>({size_t(kBounceThreads), size_t(std::max(1, default_threads())), (most + 1) / 2}));
	std::vector<std::thread> th;
	int rc = FMX_OK;
	try {
		th.reserve(size_t(nt));
		for (int t = 1; t < nt; t++) th.emplace_back([&j, t] { j.worker(t); });
	} catch (const std::exception &) {
		// fewer threads do the same work
	}
	if (!bi) rc = direct(in, cudaMemcpyHostToDevice);
	j.copy_in(0);
	{
		std::unique_lock<std::mutex> g(j.mu);
		j.cv.wait(g, [&] { return j.arrived == int(th.size()); });
	}
	if (!rc && j.failed) rc = set_error(FMX_ERR_CUDA, "copy of X to the device failed");
	if (!rc) rc = run();
	{
		std::lock_guard<std::mutex> g(j.mu);
		j.go = rc ? -1 : 1;
	}
	j.cv.notify_all();
	if (!rc) {
		j.copy_out(0);
		if (!bo) rc = direct(out, cudaMemcpyDeviceToHost);
	}
	for (std::thread &x : th) x.join();
	if (!rc && j.failed) rc = set_error(FMX_ERR_CUDA, "copy of Y to the host failed");
	// the slots are the next call's: nothing of this one may still read them
	if (cudaStreamSynchronize(st) != cudaSuccess && !rc) rc = set_error(FMX_ERR_CUDA, "SpMM failed");
	return rc;
}

void release_host_slots(int device)
{
	slots *s = device_slots(device);
	if (!s) return;
	std::lock_guard<std::mutex> g(s->mu);
	if (s->buf) cudaFreeHost(s->buf);
	s->buf = nullptr;
	for (cudaEvent_t &e : s->ev) {
		if (e) cudaEventDestroy(e);
		e = nullptr;
	}
}

} // namespace fmx
