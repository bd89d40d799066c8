// launch.cuh -- host-side launch helpers shared by the entry points.
#pragma once

#include <cuda_runtime.h>

namespace mma {

// Lets `kern` take all the dynamic shared memory the device gives.  The limit is one per kernel for the whole
// context: set to each call's own size, one thread's call could lower it between another's set and launch
// (which then fails).  Set to the same value by every call it has no order; the launch and the occupancy
// queries pass the size that they need.
template <typename K>
inline cudaError_t allow_smem(K* kern)
{
    int dev = 0, most = 0;
    cudaFuncAttributes a{};
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, kern);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, most - (int)a.sharedSizeBytes);
    if (e != cudaSuccess) cudaGetLastError();
    return e;
}

// False, with the runtime's record of the error cleared, for a call that failed.  The runtime keeps a failure
// until it is asked for: left there, the next launch's check takes it for its own.
inline bool succeeded(cudaError_t e)
{
    if (e != cudaSuccess) cudaGetLastError();
    return e == cudaSuccess;
}

}  // namespace mma
