// Copies between the device and ordinary (pageable) host memory.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>

namespace pfcg {

// cudaMemcpyAsync of n bytes on stream s of device dev. Large copies from or to
// pageable memory go through pinned chunks that several threads fill or empty
// (host_copy.cu) and, device to host, are complete on return; all others are the plain call.
// *held: whether the caller holds the chunks; set by the first copy that uses them.
cudaError_t host_copy(void* dst, const void* src, size_t n, cudaMemcpyKind kind, cudaStream_t s, int dev, bool* held);

// gives the caller's hold back; the last one frees the chunks
void host_copy_release(bool* held);

} // namespace pfcg
