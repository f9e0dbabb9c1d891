// A CUDA runtime on the host for tests of the code that drives it: "device"
// memory is host memory, and the work queued on a stream runs only when
// something waits for it (a synchronisation of the stream or the device, or a
// query of an event recorded on it).
#pragma once
#include <cuda_runtime.h>

#include <functional>

namespace fake {
constexpr int DEVICES = 2;
void enqueue(cudaStream_t s, std::function<void()> op);   // null: the legacy stream
void drain_all();                                         // what a device synchronisation does
int current_device();                                     // of the calling thread
int last_host_alloc_device();                             // current device at the last cudaMallocHost
}  // namespace fake
