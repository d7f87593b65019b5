// Pinned host memory for results (mcrt_host_alloc, mcrt_host_free).
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

namespace mcrt {

// `bytes` of zeroed host memory that every device copies into directly, page
// aligned, made with the current device. Any thread.
cudaError_t host_alloc(size_t bytes, void** out);
// Gives it back. Any thread; the caller's current device stays as it is. False
// if `p` is not from host_alloc.
bool host_free(void* p);

}  // namespace mcrt
