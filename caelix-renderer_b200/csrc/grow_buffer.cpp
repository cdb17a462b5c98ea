// Device memory grown on demand (grow_buffer.h).
#include "grow_buffer.h"

#include <cuda_runtime.h>

namespace cx {

CaelixResult cuda_result(cudaError_t e, const char* what);

CaelixResult GrowBuffer::reserve(uint64_t want, const char* what)
{
    if (want <= bytes) return CAELIX_OK;
    release();
    const cudaError_t e = cudaMalloc(&ptr, want);
    if (e != cudaSuccess) {
        ptr = nullptr;
        return cuda_result(e, what);
    }
    bytes = want;
    return CAELIX_OK;
}

bool GrowBuffer::try_reserve(uint64_t want, uint64_t keep)
{
    if (want <= bytes) return true;
    if (bytes < keep) release();  // of no use either way: its room first
    void* grown = nullptr;
    if (cudaMalloc(&grown, want) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    release();
    ptr = grown;
    bytes = want;
    return true;
}

void GrowBuffer::release()
{
    if (ptr) cudaFree(ptr);
    ptr = nullptr;
    bytes = 0;
}

}  // namespace cx
