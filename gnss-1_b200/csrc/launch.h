// launch.h -- launchers of the pass and z kernels, one translation unit per
// family and precision (pass_f32.cu, pass_f64.cu, z_f32.cu, z_f64.cu).
#pragma once
#include <cuda_runtime.h>

#include <utility>

#include "gnss_b200.h"
#include "kernels.cuh"

using namespace gnss;

// Launch of a kernel of the step.  Within a PdlScope that allows it, the
// launch carries programmatic stream serialization: the kernel may start its
// prologue on SMs the previous kernel in the stream has left and waits
// (pdl_wait) before it touches the memory of the step.  Inside stream capture
// the dependency becomes a programmatic graph edge.  Measured per step (FP32,
// one scalar): 64^3 53.5 -> 40.9 us, 96^3 118.7 -> 107.3 us, 128^3 195.3 ->
// 181.7 us, 192^3 579 -> 565 us.  Steps of more than 2^23 points launch
// plainly: with programmatic launches the 256^3 and 512^3 FP64 steps measured
// 0.5 - 2% slower.
inline thread_local bool t_pdl = false;
struct PdlScope {
    bool prev;
    explicit PdlScope(bool on) : prev(t_pdl) { t_pdl = on; }
    ~PdlScope() { t_pdl = prev; }
};
constexpr long long PDL_MAX_POINTS = 1LL << 23;
template <typename... KA, typename... A>
static cudaError_t launch_dep(void (*kern)(KA...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A &&...args) {
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = at;
    cfg.numAttrs = t_pdl ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, std::forward<A>(args)...);
}

// x / y pass of length n (sign -1 forward, +1 inverse)
template <typename T>
cudaError_t launch_pass(int n, int sign, const PassPtrs<T> &P, const PassSpec &sp, const void *tw, int nsm,
                        cudaStream_t s, int pvariant, unsigned *err);
// z pass of length n over pairs of lines (dir -1: R2C, +1: C2R)
template <typename T>
cudaError_t launch_zpass(int n, int dir, const FieldSet<T> &f, int nfields, long long nlines, int nz2, T scale,
                         const void *tw, cudaStream_t s);
// fused z stage; diag != nullptr: with per-block vorticity sums (register kernels only)
template <typename T>
cudaError_t launch_zphys(int n, const FieldSet<T> &f, const ZRecipeSet &zr, int nph, int nraw, int nout,
                         long long nlines, int ncp, int nkz, T scale, T alpha, double dkz, const void *tw,
                         unsigned *err, int nsm, cudaStream_t s, int zvariant, double *diag = nullptr,
                         int nmem = 1, long long ms = 0);
// the z kernel a variant option selects (GNSS_VARIANT_*), and whether a register z kernel exists
template <typename T> int zkernel_choice(int n, int zvariant, int nph, int nraw, int nout, int ncp);
template <typename T> bool zreg_available(int n, int nph, int nraw, int ncp);

#define GNSS_SIZE_SWITCH(n, EXPR) GNSS_SIZE_SWITCH_OR(n, EXPR, return cudaErrorInvalidValue)
#define GNSS_SIZE_SWITCH_OR(n, EXPR, DEFAULT)       \
    switch (n) {                                    \
        case 8: { constexpr int NN_ = 8; EXPR; }    \
        case 12: { constexpr int NN_ = 12; EXPR; }  \
        case 16: { constexpr int NN_ = 16; EXPR; }  \
        case 24: { constexpr int NN_ = 24; EXPR; }  \
        case 32: { constexpr int NN_ = 32; EXPR; }  \
        case 48: { constexpr int NN_ = 48; EXPR; }  \
        case 64: { constexpr int NN_ = 64; EXPR; }  \
        case 96: { constexpr int NN_ = 96; EXPR; }  \
        case 128: { constexpr int NN_ = 128; EXPR; } \
        case 192: { constexpr int NN_ = 192; EXPR; } \
        case 256: { constexpr int NN_ = 256; EXPR; } \
        case 384: { constexpr int NN_ = 384; EXPR; } \
        case 512: { constexpr int NN_ = 512; EXPR; } \
        default: DEFAULT;                           \
    }
