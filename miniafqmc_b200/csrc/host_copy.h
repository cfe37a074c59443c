// Copies between the device and the caller's pageable memory, through a small pinned ring
// owned by one handle.
#pragma once
#include <cuda_runtime.h>
#include <cstddef>

namespace afq {

struct HostRing;   // allocated by the first large copy of a handle
void host_ring_destroy(HostRing* r);

// dst (host) <- src (device) or dst (device) <- src (host), in order on `st`.  Pageable host
// memory is free for use on return; the caller synchronises `st` before it reads dst or frees
// pinned memory.
cudaError_t copy_to_host(HostRing** ring, void* dst, const void* src, size_t bytes, cudaStream_t st);
cudaError_t copy_to_device(HostRing** ring, void* dst, const void* src, size_t bytes,
                           cudaStream_t st);

}  // namespace afq
