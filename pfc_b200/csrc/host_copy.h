// Copies between the device and ordinary (pageable) host memory.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>

namespace pfcg {

// What a caller (a handle) has of the pinned chunks. It goes back by host_copy_release.
struct HostHold {
	bool held = false; // it has used them
	size_t moved = 0;  // bytes copied without them, while there were none
};

// cudaMemcpyAsync of n bytes on stream s of device dev. Large copies from or to
// pageable memory go through pinned chunks that several threads fill or empty
// (host_copy.cu) and, device to host, are complete on return; all others are the plain call.
// The chunks are made for the first caller that has moved enough for them to pay.
cudaError_t host_copy(void* dst, const void* src, size_t n, cudaMemcpyKind kind, cudaStream_t s, int dev, HostHold* hold);

// gives the caller's hold back; the last one frees the chunks
void host_copy_release(HostHold* hold);

} // namespace pfcg
