// Stream-ordered scratch of the image passes (scratch.cpp).
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>

namespace rfk {

// `bytes` of device memory on `st`'s current device, freed with cudaFreeAsync on a stream
cudaError_t scratch_alloc(void** p, size_t bytes, cudaStream_t st);
template <class T>
cudaError_t scratch_alloc(T** p, size_t count, cudaStream_t st) {
    return scratch_alloc((void**)p, count * sizeof(T), st);
}
// gives the current device's unused scratch back
cudaError_t scratch_trim();

}  // namespace rfk
