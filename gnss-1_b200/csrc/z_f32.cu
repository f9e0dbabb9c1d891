// z_f32.cu -- FP32 instantiations of the fused z stage's launchers.
#include "z_launch.cuh"

template cudaError_t launch_zphys<float>(int, const FieldSet<float> &, const ZRecipeSet &, int, int, int, long long, int, int,
                                      float, float, double, const void *, unsigned *, int, cudaStream_t, int, double *, int,
                                      long long);
template int zkernel_choice<float>(int, int, int, int, int, int);
template bool zreg_available<float>(int, int, int, int);
