// Device scratch of the engine's calls (scratch.cu): stream-ordered allocations from a private memory
// pool per device while a scene lives there, from the default pool otherwise.
#pragma once

#include <cstddef>
#include <cuda_runtime.h>

namespace wobgb {

// Allocates / frees on the current device, in stream order.
cudaError_t scratch_alloc(void **p, size_t bytes, cudaStream_t stream);
cudaError_t scratch_free(void *p, cudaStream_t stream);

// A scene on `device` begins / ends its life. The first makes the pool (on no stream, so before any walk
// can be captured), which keeps up to 512 MB between calls while a scene of the device lives; the last one
// to go gives it back.
void scratch_retain(int device);
void scratch_release(int device);

}  // namespace wobgb
