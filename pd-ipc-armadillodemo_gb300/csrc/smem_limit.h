// smem_limit.h — a kernel's limit on dynamic shared memory.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

namespace pdipc {

// Lets launches of kernel f have `smem` bytes of dynamic shared memory.  The limit is the
// kernel's, for every context and thread of the process, so it is always set to the
// same value, all that the device has beside f's static part: to raise it only as far as
// one context needs would be to read and write it in two steps, between which another
// thread may have raised it further.
inline cudaError_t allow_smem(const void* f, size_t smem) {
    int dev = 0, optin = 0;
    cudaFuncAttributes fa;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, f);
    if (e != cudaSuccess) return e;
    if (fa.sharedSizeBytes + smem > (size_t)optin) return cudaErrorInvalidValue;
    return cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - (int)fa.sharedSizeBytes);
}

}  // namespace pdipc
