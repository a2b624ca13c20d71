// Device memory of plans, solver states and scratch, from a pool per device that
// keeps at most 2 GB between objects: a solve that builds its plan (500 MB at
// 128x256x256) spent 1.2 ms in cudaMalloc and 1.4-4.6 ms in cudaFree.  Memory
// above that goes back to the driver as an object is freed, all of it when an
// allocation fails, in the pool or (by the driver) outside of it.  Host code only.
#pragma once

#include <cuda_runtime_api.h>

#include <cstddef>
#include <initializer_list>

namespace dk {

// Non-blocking stream of the current device for set-up work, or nullptr.
cudaStream_t setup_stream();

int device_pool(cudaMemPool_t* out);
// Memory that every stream may use at once.
int pool_alloc(void** p, size_t bytes, const char* what);
// Waits for the device's work, as cudaFree does, so that nothing still running
// can touch what the next object gets; once for all pointers (null ones are
// skipped).  Where the wait is refused the memory is held until a later one
// succeeds.
void pool_free(void* const* ptrs, size_t n);
inline void pool_free(std::initializer_list<void*> ptrs) { pool_free(ptrs.begin(), ptrs.size()); }

}  // namespace dk
