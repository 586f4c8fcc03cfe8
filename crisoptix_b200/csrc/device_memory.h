// device_memory.h -- device allocations of the library.
//
// The endpoint search keeps its workspace between calls (search.cu).  An allocation
// that fails for want of memory gives that back and tries once more, so that what is
// only kept never makes a call fail.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

namespace crisb {

// search.cu: gives back what the endpoint search keeps in the current context and
// does not use
void trim_search_workspace();

// alloc(), and after a failure for want of memory trim() and alloc() again
template <class Alloc, class Trim>
cudaError_t alloc_or_trim(Alloc alloc, Trim trim) {
    const cudaError_t e = alloc();
    if (e != cudaErrorMemoryAllocation) return e;
    cudaGetLastError();
    trim();
    return alloc();
}

inline cudaError_t device_malloc(void** p, size_t bytes) {
    return alloc_or_trim([&] { return cudaMalloc(p, bytes); }, trim_search_workspace);
}

}  // namespace crisb
