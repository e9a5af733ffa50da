// Pageable host copies through pinned chunks (host_copy.h).
//
// The driver moves pageable memory through a staging buffer of its own with one
// thread, 17 to 20 GB/s here where the link carries 53. WORKERS threads, the
// caller's among them, take chunks in turn, each with SLOTS of them, so that one is
// on the link while another is filled or emptied. The calls into the driver bound it
// then: 16.8 MB of fields up (with their transform) 918 -> 624 us and down 1046 ->
// 550 with 1 MB chunks, 720 and 665 with 512 KB, 990 and 940 with 256 KB and eight
// threads, which is no better than the driver alone.
//
// The chunks are registered huge pages, pinned in 0.9 to 2 ms; cudaHostAlloc takes 3.6 to
// 9.6 ms for the same 8 MB. That is still more than a few copies gain, so they are made
// only for a caller that has moved PAYS bytes (a handle that takes 16.8 MB of fields in
// and out once, with its end: 4.1 ms, 9.9 to 12.6 when its first copy made the chunks).
#include "host_copy.h"

#include <stdint.h>
#include <string.h>
#include <sys/mman.h>

#include <atomic>
#include <mutex>
#include <thread>

namespace pfcg {
namespace {

constexpr size_t CHUNK = 1 << 20;
constexpr int WORKERS = 4, SLOTS = 2;
// Below LEAST_UP the threads' start (some 15 us each) outweighs the faster copy. Down, a
// copy by several cores stalls in about half of the calls for 0.5 to 0.7 ms that neither
// fewer threads, other chunks nor one thread for all driver calls avoid (8 MB: 0.33 or 1.1
// ms, the driver alone 0.5; 16 MB: 0.5 or 1.1, the driver 0.9 to 1.05; 32 MB: 0.9 or 1.6, the
// driver 1.7 to 2.0 and 7.5 into an array that is new), so it is left to the driver below
// LEAST_DOWN, from where the mean of both gains.
constexpr size_t LEAST_UP = 4 << 20, LEAST_DOWN = 16 << 20;
// A caller's bytes from which the chunks are made: 64 MB gain 1 to 2 ms,
// the chunks cost 1.3 to 2.4 to make and give back.
constexpr size_t PAYS = 64 << 20;
constexpr size_t POOL = WORKERS * SLOTS * CHUNK, HUGE = 2 << 20;

std::mutex g_mu;                 // one staged copy at a time; others take the plain path
unsigned char* g_pool = nullptr; // WORKERS * SLOTS chunks, 8 MB for the process
void* g_map = nullptr;           // the mapping that holds them
int g_holds = 0;

// Other threads may be capturing streams: nothing here belongs to a capture.
struct Relaxed {
	cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
	Relaxed() { cudaThreadExchangeStreamCaptureMode(&mode); }
	~Relaxed() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

// The chunks, on huge pages where the system gives them; nullptr where they can't be had.
unsigned char* make_pool() {
	void* m = mmap(nullptr, POOL + HUGE, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
	if (m == MAP_FAILED) return nullptr;
	unsigned char* p = (unsigned char*)(((uintptr_t)m + HUGE - 1) & ~(uintptr_t)(HUGE - 1));
	madvise(p, POOL, MADV_HUGEPAGE);
	madvise(m, POOL + HUGE, MADV_DONTFORK); // a child's copies would take the pages from under the device
	Relaxed relaxed;
	if (cudaHostRegister(p, POOL, cudaHostRegisterPortable) != cudaSuccess) {
		cudaGetLastError();
		munmap(m, POOL + HUGE);
		return nullptr;
	}
	g_map = m;
	return p;
}

struct Job {
	unsigned char* host;
	unsigned char* devp;
	size_t n;
	bool up; // host to device
	cudaStream_t s;
	int dev;
	std::atomic<size_t> next{0};
	std::atomic<int> err{0};

	void work(int w) noexcept {
		Relaxed relaxed;
		cudaEvent_t ev[SLOTS] = {};
		size_t at[SLOTS] = {};
		bool busy[SLOTS] = {};
		cudaError_t e = cudaSetDevice(dev);
		for (int i = 0; i < SLOTS && e == cudaSuccess; i++) e = cudaEventCreateWithFlags(&ev[i], cudaEventDisableTiming);
		// waits for the chunk in slot i and, device to host, empties it
		auto finish = [&](int i) {
			if (!busy[i]) return;
			busy[i] = false;
			const cudaError_t f = cudaEventSynchronize(ev[i]);
			if (f != cudaSuccess) e = f;
			else if (!up) memcpy(host + at[i], slot(w, i), len(at[i]));
		};
		for (int k = 0; e == cudaSuccess && !err; k++) {
			const int i = k % SLOTS;
			finish(i);
			const size_t o = next.fetch_add(CHUNK);
			if (o >= n || e != cudaSuccess) break;
			at[i] = o;
			if (up) memcpy(slot(w, i), host + o, len(o));
			e = up ? cudaMemcpyAsync(devp + o, slot(w, i), len(o), cudaMemcpyHostToDevice, s)
			       : cudaMemcpyAsync(slot(w, i), devp + o, len(o), cudaMemcpyDeviceToHost, s);
			if (e == cudaSuccess) e = cudaEventRecord(ev[i], s);
			busy[i] = e == cudaSuccess;
		}
		for (int i = 0; i < SLOTS; i++) finish(i);
		for (int i = 0; i < SLOTS; i++)
			if (ev[i]) cudaEventDestroy(ev[i]);
		if (e != cudaSuccess) err = (int)e;
	}

private:
	static unsigned char* slot(int w, int i) { return g_pool + (w * SLOTS + i) * CHUNK; }
	size_t len(size_t o) const { return n - o < CHUNK ? n - o : CHUNK; }
};

} // namespace

cudaError_t host_copy(void* dst, const void* src, size_t n, cudaMemcpyKind kind, cudaStream_t s, int dev, HostHold* hold) {
	const bool up = kind == cudaMemcpyHostToDevice;
	if (n < (up ? LEAST_UP : LEAST_DOWN) || (!up && kind != cudaMemcpyDeviceToHost)) return cudaMemcpyAsync(dst, src, n, kind, s);
	cudaPointerAttributes at;
	cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
	const bool known = cudaPointerGetAttributes(&at, up ? src : dst) == cudaSuccess && cudaStreamIsCapturing(s, &cap) == cudaSuccess;
	if (!known) cudaGetLastError();
	std::unique_lock<std::mutex> lk(g_mu, std::defer_lock);
	// pinned and managed memory need no staging
	if (!known || at.type != cudaMemoryTypeUnregistered || cap != cudaStreamCaptureStatusNone || !lk.try_lock())
		return cudaMemcpyAsync(dst, src, n, kind, s);
	if (!g_pool) {
		hold->moved += n;
		if (hold->moved >= PAYS) g_pool = make_pool();
		if (!g_pool) {
			lk.unlock();
			return cudaMemcpyAsync(dst, src, n, kind, s);
		}
	}
	if (!hold->held) {
		hold->held = true;
		g_holds++;
	}
	int cur = dev;
	cudaGetDevice(&cur);
	Job job;
	job.host = (unsigned char*)(up ? const_cast<void*>(src) : dst);
	job.devp = (unsigned char*)(up ? dst : const_cast<void*>(src));
	job.n = n;
	job.up = up;
	job.s = s;
	job.dev = dev;
	std::thread th[WORKERS - 1];
	try {
		for (int w = 1; w < WORKERS; w++) th[w - 1] = std::thread([&job, w] { job.work(w); });
	} catch (...) { // no more threads to be had: the ones that started and this one do it
	}
	job.work(0);
	for (std::thread& t : th)
		if (t.joinable()) t.join();
	if (cur != dev) cudaSetDevice(cur);
	return (cudaError_t)job.err.load();
}

void host_copy_release(HostHold* hold) {
	if (!hold->held) return;
	hold->held = false;
	std::lock_guard<std::mutex> lk(g_mu);
	if (--g_holds) return;
	Relaxed relaxed;
	cudaHostUnregister(g_pool);
	munmap(g_map, POOL + HUGE);
	g_pool = nullptr;
	g_map = nullptr;
}

} // namespace pfcg
