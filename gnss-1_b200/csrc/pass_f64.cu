// pass_f64.cu -- FP64 instantiations of the pass launchers.
#include "pass_launch.cuh"

template cudaError_t launch_pass<double>(int, int, const PassPtrs<double> &, const PassSpec &, const void *, int, cudaStream_t,
                                     int, unsigned *);
template cudaError_t launch_zpass<double>(int, int, const FieldSet<double> &, int, long long, int, double, const void *,
                                      cudaStream_t);
