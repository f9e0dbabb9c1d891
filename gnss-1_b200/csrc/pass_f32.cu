// pass_f32.cu -- FP32 instantiations of the pass launchers.
#include "pass_launch.cuh"

template cudaError_t launch_pass<float>(int, int, const PassPtrs<float> &, const PassSpec &, const void *, int, cudaStream_t,
                                     int, unsigned *);
template cudaError_t launch_zpass<float>(int, int, const FieldSet<float> &, int, long long, int, float, const void *,
                                      cudaStream_t);
