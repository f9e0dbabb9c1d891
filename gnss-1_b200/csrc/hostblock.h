// hostblock.h -- host side of a context's device block (make_device_block);
// no device code, so that it also compiles with the host compiler alone.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>

namespace gnss {

// Copies pageable host memory to the device and waits until it is there.
// cudaMemcpy from pageable memory may return once the data lies in its staging
// buffer, and work on a non-blocking stream does not wait for the stream that
// carries the rest of the copy.
inline cudaError_t upload_and_wait(void *dst, const void *src, size_t bytes) {
    const cudaError_t e = cudaMemcpy(dst, src, bytes, cudaMemcpyHostToDevice);
    return e == cudaSuccess ? cudaStreamSynchronize(cudaStreamLegacy) : e;
}

}  // namespace gnss
