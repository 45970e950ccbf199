// vpt_scratch.h - stream-ordered scratch of the entry points that keep no state between calls (vpt_scratch.cu).
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

namespace vpt {

// Scratch in stream order, to be returned with cudaFreeAsync.
cudaError_t scratch_alloc(void** p, size_t bytes, cudaStream_t s);
// Gives the scratch that no call is using on the current device back to the driver.
void scratch_trim();

}  // namespace vpt
