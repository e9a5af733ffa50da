// pfc_b200/csrc/host_copy.cu over a stand-in for the CUDA runtime whose device memory
// is host memory: which copies go through pinned chunks, when those are made and given
// back, and the bytes that arrive. Prints the failures and their count.
#include <cuda_runtime.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <mutex>
#include <vector>

static std::mutex mu;
static unsigned char* pinned = nullptr; // the pinned memory
static size_t pinned_n = 0;
static int pins = 0, staged = 0, plain = 0; // pinned so far; copies through it and past it

extern "C" {
cudaError_t cudaHostRegister(void* p, size_t n, unsigned) {
	pinned = (unsigned char*)p;
	pinned_n = n;
	pins++;
	return cudaSuccess;
}
cudaError_t cudaHostUnregister(void* p) {
	if (p == pinned) pinned = nullptr;
	return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
	*p = malloc(n);
	return cudaHostRegister(*p, n, 0);
}
cudaError_t cudaFreeHost(void* p) {
	cudaHostUnregister(p);
	free(p);
	return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
	std::lock_guard<std::mutex> lk(mu);
	auto in = [&](const void* p) { return pinned && (const unsigned char*)p >= pinned && (const unsigned char*)p + n <= pinned + pinned_n; };
	(in(d) || in(s) ? staged : plain)++;
	memcpy(d, s, n);
	return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) {
	a->type = cudaMemoryTypeUnregistered;
	return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* c) {
	*c = cudaStreamCaptureStatusNone;
	return cudaSuccess;
}
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode*) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
	*e = (cudaEvent_t)1;
	return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) {
	*d = 0;
	return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
}

#include "../../pfc_b200/csrc/host_copy.cu"

using namespace pfcg;

static int failures = 0;
#define CHECK(c)                                            \
	do {                                                    \
		if (!(c)) {                                         \
			failures++;                                     \
			printf("line %d: %s\n", __LINE__, #c);          \
		}                                                   \
	} while (0)

static void copy(HostHold* h, size_t n, bool up) {
	std::vector<unsigned char> a(n + 1), b(n + 1, 0);
	for (size_t i = 0; i <= n; i++) a[i] = (unsigned char)(i * 2654435761u >> 13);
	CHECK(host_copy(b.data(), a.data(), n, up ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToHost, nullptr, 0, h) == cudaSuccess);
	CHECK(!memcmp(a.data(), b.data(), n) && b[n] == 0);
}

int main() {
	const size_t fields = 2 * 1024 * 1024 * sizeof(double); // two fields of 1024^2
	// callers that take their fields in and out once: nothing is pinned for them
	for (int i = 0; i < 8; i++) {
		HostHold h{};
		copy(&h, fields, true);
		copy(&h, fields, false);
		host_copy_release(&h);
	}
	CHECK(pins == 0 && staged == 0 && plain == 16);
	// one that goes on: pinned once, after which it copies through the chunks, in and out
	HostHold a{}, b{}, c{};
	for (int i = 0; i < 16; i++) copy(&a, fields, i % 2);
	CHECK(pins == 1 && staged > 0);
	// another one beside it uses them from its first copy on, whatever its length
	int was = plain;
	for (size_t n : {(size_t)4 << 20, ((size_t)4 << 20) + 1, ((size_t)5 << 20) - 3, ((size_t)8 << 20) + 8, fields + 5}) copy(&b, n, true);
	for (size_t n : {fields, fields + 1, ((size_t)17 << 20) - 3, ((size_t)25 << 20) + 8}) copy(&b, n, false);
	CHECK(plain == was && pins == 1);
	// short ones don't, which the driver copies as fast or faster
	int through = staged;
	copy(&b, 1 << 20, true);
	copy(&b, ((size_t)4 << 20) - 8, true);
	for (size_t mb : {1, 4, 6, 8, 12}) copy(&b, mb << 20, false);
	CHECK(plain == was + 7 && staged == through);
	// given back with the last of the two, and made again for one that pays
	host_copy_release(&a);
	CHECK(pinned);
	host_copy_release(&b);
	CHECK(!pinned);
	copy(&c, (size_t)100 << 20, true);
	CHECK(pinned && pins == 2);
	host_copy_release(&c);
	host_copy_release(&c);
	CHECK(!pinned);
	printf("%d failures\n", failures);
	return failures != 0;
}
