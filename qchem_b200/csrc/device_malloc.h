// device_malloc.h -- device memory beside the library's idle buffers.
#pragma once
#include <cuda_runtime.h>

namespace qcg {

// cudaMalloc on the current device.  Where it finds no room, the idle buffers that the library keeps for later handles
// (runtime.cu) are freed and it is tried again.  A failure is only returned, not left for cudaGetLastError.
cudaError_t device_malloc(void** p, size_t bytes);
template <class T>
cudaError_t device_malloc(T** p, size_t bytes)
{
    return device_malloc((void**)p, bytes);
}

}   // namespace qcg
