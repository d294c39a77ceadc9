#pragma once

#include "common.cuh"

namespace ph {

// Dynamic shared memory above 48 KB, asked for once per kernel, host thread and device.
template <auto Kernel>
inline int allow_shared(size_t bytes, const char* what) {
    if (bytes <= 48 * 1024) return PH_OK;
    static thread_local unsigned long long done = 0;               // one bit per device
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return fail(PH_ERR_LAUNCH, "%s: no device", what);
    if (dev < 64 && (done >> dev & 1)) return PH_OK;
    const cudaError_t e = cudaFuncSetAttribute(Kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return fail(PH_ERR_LAUNCH, "%s: %s", what, cudaGetErrorString(e));
    if (dev < 64) done |= 1ull << dev;
    return PH_OK;
}

// Multiprocessors of the current device.
inline int multiprocessors() {
    static thread_local int known_dev = -1, known = 0;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 148;
    if (dev != known_dev && cudaDeviceGetAttribute(&known, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess) known_dev = dev;
    return known > 0 ? known : 148;
}

}  // namespace ph
