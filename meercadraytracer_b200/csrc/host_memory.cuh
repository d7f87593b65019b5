// Pinned host memory for results (mcrt_host_alloc, mcrt_host_free).
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

namespace mcrt {

// `bytes` of host memory that every device copies into directly, page aligned,
// made with the current device. Any thread.
cudaError_t host_alloc(size_t bytes, void** out);
// Gives it back. Any thread; the caller's current device stays as it is. False
// if `p` is not from host_alloc.
bool host_free(void* p);

// Makes room for at least `bytes` of blocks ahead, with the current device, so
// that host_alloc needs nothing of the driver until it is used up. Kept until
// as many host_unreserve calls have been made, and its blocks are back.
cudaError_t host_reserve(size_t bytes);
void host_unreserve();

}  // namespace mcrt
