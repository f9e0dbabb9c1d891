// z_f64.cu -- FP64 instantiations of the fused z stage's launchers.
#include "z_launch.cuh"

template cudaError_t launch_zphys<double>(int, const FieldSet<double> &, const ZRecipeSet &, int, int, int, long long, int, int,
                                      double, double, double, const void *, unsigned *, int, cudaStream_t, int, double *, int,
                                      long long);
template int zkernel_choice<double>(int, int, int, int, int, int);
template bool zreg_available<double>(int, int, int, int);
