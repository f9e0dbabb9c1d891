// launch.cuh -- helpers shared by the launchers.
#pragma once
#include <algorithm>
#include <atomic>
#include <type_traits>

#include "launch.h"

// Dynamic shared memory above 48 KB needs an opt-in, and the largest carveout
// lets several blocks share an SM.
template <class K> static cudaError_t prep_smem(K kern, int bytes) {
    if (bytes > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
        if (e != cudaSuccess) return e;
    }
    if (bytes > 0)
        return cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout,
                                    (int)cudaSharedmemCarveoutMaxShared);
    return cudaSuccess;
}

template <class K> static int blocks_per_sm(K kern, int threads, int smem) {
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, threads, smem) != cudaSuccess) {
        cudaGetLastError();
        n = 1;
    }
    return n < 1 ? 1 : n;
}
