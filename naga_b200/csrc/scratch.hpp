// Stream-ordered allocations of the library (scratch.cpp); freed with
// cudaFreeAsync.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>

namespace naga {

// `bytes` of device memory of the current device, ordered on `st`
cudaError_t scratch_malloc_bytes(void** p, size_t bytes, cudaStream_t st);
template <class T>
cudaError_t scratch_malloc(T** p, size_t bytes, cudaStream_t st) {
    return scratch_malloc_bytes(reinterpret_cast<void**>(p), bytes, st);
}
// gives the current device's unused scratch back to the system
void scratch_trim();

// Unique id of the calling thread's current context (cuCtxGetId through the
// runtime's driver entry points, so the library needs no libcuda link);
// false when it cannot be had (no current context, an older driver).
bool current_context_id(unsigned long long* id);

}  // namespace naga
