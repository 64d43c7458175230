// Copies between pageable host memory and the device, staged through pinned memory by several threads.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>

namespace rtg {

struct CopyPart {
    void* host;
    void* dev;
    size_t bytes;
};
// Copies the parts in `stream`'s order and waits for them. Calls must not overlap (the library's lock).
cudaError_t copy_planes(const CopyPart* parts, int n, bool to_device, cudaStream_t stream);
// Gives the pinned memory back.
void copy_release();

}  // namespace rtg
