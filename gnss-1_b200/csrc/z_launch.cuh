// z_launch.cuh -- launchers of the fused z stage, instantiated per precision
// by z_f32.cu and z_f64.cu.
#pragma once
#include "launch.cuh"
#include "zreg.cuh"

template <typename T, int N> struct ZLaunch {
    template <int NPH, int NRAW, bool PP>
    static cudaError_t zphys_k(const FieldSet<T> &f, const ZRecipeSet &zr, int nout, long long nlines, int ncp,
                               int nkz, T scale, T alpha, double dkz, const void *tw, unsigned *err, int nsm,
                               cudaStream_t s, int nmem, long long ms) {
        if (nmem > 1) return cudaErrorNotSupported;   // batches run the register z kernel
        using C = ZPCfg<T, N>;
        const int pipe_b = C::pipe_bytes(NPH, NRAW, ncp, PP);
        const int pipe = pipe_b <= C::SMEM_MAX ? 1 : 0;
        const int smem = pipe ? pipe_b : C::work_bytes(NPH, PP);
        auto kern = k_zphys<T, N, NPH, NRAW, PP>;
        cudaError_t e = prep_smem(kern, smem);
        if (e != cudaSuccess) return e;
        int per_sm = blocks_per_sm(kern, NPH * 32, smem);
        const long long mpairs = nlines / 2, npairs = mpairs * nmem;
        long long grid = (long long)per_sm * nsm;
        if (grid > npairs) grid = npairs;
        return launch_dep(kern, dim3((unsigned)grid), dim3(NPH * 32), smem, s, f, zr, nout, npairs, ncp, nkz, pipe,
                          scale, alpha, dkz, reinterpret_cast<const V2<T> *>(tw), err, mpairs, ms);
    }
    // ping-pong banks when they fit next to the staging area, else in place
    template <int NPH, int NRAW>
    static cudaError_t zphys_n(const FieldSet<T> &f, const ZRecipeSet &zr, int nout, long long nlines, int ncp,
                               int nkz, T scale, T alpha, double dkz, const void *tw, unsigned *err, int nsm,
                               cudaStream_t s, int nmem, long long ms) {
        using C = ZPCfg<T, N>;
        if (C::pipe_bytes(NPH, NRAW, ncp, true) <= C::SMEM_MAX)
            return zphys_k<NPH, NRAW, true>(f, zr, nout, nlines, ncp, nkz, scale, alpha, dkz, tw, err, nsm, s, nmem,
                                            ms);
        return zphys_k<NPH, NRAW, false>(f, zr, nout, nlines, ncp, nkz, scale, alpha, dkz, tw, err, nsm, s, nmem, ms);
    }
    // FP32: k_zpipe, FP64: k_zws
    template <int NPH> using ZBlock = std::conditional_t<sizeof(T) == 4, ZPipe<T, N, NPH>, ZWs<T, N, NPH>>;
    // the register z kernels (N = 64 .. 512, zr_size); diag != nullptr: the instantiation that also writes per-block vorticity sums.
    // Where the staged raw lines do not fit (FP64, N = 512: the colloid term, or a truncation that keeps more than
    // 2/3 of the modes with two scalars) the warps read them from global memory.
    template <int NPH, int NRAW, bool STAGED>
    static cudaError_t zpipe_k(const FieldSet<T> &f, const ZRecipeSet &zr, long long nlines, int ncp, int nkz, T scale,
                               T alpha, double dkz, const void *tw, unsigned *err, int nsm, cudaStream_t s, double *diag,
                               int nmem, long long ms) {
        using C = ZBlock<NPH>;
        const int smem = C::smem_bytes(STAGED ? NRAW : 0, ncp);
        auto pick = [&] {
            if constexpr (sizeof(T) == 4)
                return diag       ? k_zpipe<T, N, NPH, NRAW, true>
                       : nmem > 1 ? k_zpipe<T, N, NPH, NRAW, false, true>
                                  : k_zpipe<T, N, NPH, NRAW>;
            else
                return diag       ? k_zws<T, N, NPH, NRAW, true, false, STAGED>
                       : nmem > 1 ? k_zws<T, N, NPH, NRAW, false, true, STAGED>
                                  : k_zws<T, N, NPH, NRAW, false, false, STAGED>;
        };
        auto kern = pick();
        cudaError_t e = prep_smem(kern, smem);
        if (e != cudaSuccess) return e;
        const int per_sm = blocks_per_sm(kern, C::NT, smem);
        const long long mpairs = nlines / 2, npairs = mpairs * nmem;
        long long grid = (long long)per_sm * nsm;
        if (grid > npairs) grid = npairs;
        if (diag && grid > STAT_BLOCKS) grid = STAT_BLOCKS;   // one row of sums per block
        return launch_dep(kern, dim3((unsigned)grid), dim3(C::NT), smem, s, f, zr, npairs, ncp, nkz, scale, alpha, dkz,
                          reinterpret_cast<const V2<T> *>(tw), err, diag, mpairs, ms);
    }
    template <int NPH, int NRAW>
    static cudaError_t zpipe_n(const FieldSet<T> &f, const ZRecipeSet &zr, long long nlines, int ncp, int nkz, T scale,
                               T alpha, double dkz, const void *tw, unsigned *err, int nsm, cudaStream_t s, double *diag,
                               int nmem, long long ms) {
        if constexpr (zr_size(N)) {
            if (ZBlock<NPH>::smem_bytes(NRAW, ncp) <= ZPCfg<T, N>::SMEM_MAX)
                return zpipe_k<NPH, NRAW, true>(f, zr, nlines, ncp, nkz, scale, alpha, dkz, tw, err, nsm, s, diag, nmem, ms);
            if constexpr (sizeof(T) == 8 && N == 512 && NPH > 9)
                return zpipe_k<NPH, NRAW, false>(f, zr, nlines, ncp, nkz, scale, alpha, dkz, tw, err, nsm, s, diag, nmem, ms);
        }
        return cudaErrorNotSupported;
    }
    static cudaError_t zpipe(const FieldSet<T> &f, const ZRecipeSet &zr, int nph, int nraw, long long nlines, int ncp,
                             int nkz, T scale, T alpha, double dkz, const void *tw, unsigned *err, int nsm,
                             cudaStream_t s, double *diag, int nmem, long long ms) {
        if (nph == 9 && nraw == 10)
            return zpipe_n<9, 10>(f, zr, nlines, ncp, nkz, scale, alpha, dkz, tw, err, nsm, s, diag, nmem, ms);
        if (nph == 12 && nraw == 13)
            return zpipe_n<12, 13>(f, zr, nlines, ncp, nkz, scale, alpha, dkz, tw, err, nsm, s, diag, nmem, ms);
        if (nph == 14 && nraw == 14)
            return zpipe_n<14, 14>(f, zr, nlines, ncp, nkz, scale, alpha, dkz, tw, err, nsm, s, diag, nmem, ms);
        return cudaErrorInvalidValue;
    }
    // the lines GNSS_VARIANT_WARPSPEC names (z length 256 or 512; FP32 with one scalar, FP64 with one or two,
    // without the colloid term)
    static bool zws_fits(int nph, int nraw, int nout, int ncp) {
        const bool fp32 = sizeof(T) == 4 && nph == 9 && nraw == 10 && nout == 4;
        const bool fp64 = sizeof(T) == 8 && ((nph == 9 && nraw == 10 && nout == 4) ||
                                             (nph == 12 && nraw == 13 && nout == 5));
        if constexpr (N == 256 || N == 512) {
            const int smem = nph == 9 ? ZBlock<9>::smem_bytes(nraw, ncp) : ZBlock<12>::smem_bytes(nraw, ncp);
            return (fp32 || fp64) && smem <= ZPCfg<T, N>::SMEM_MAX;
        } else {
            return false;
        }
    }
    static bool zreg_fits(int nph, int nraw, int ncp) {
        if constexpr (zr_size(N)) {
            if (sizeof(T) == 8 && N == 512 && nph > 9) return true;   // unstaged where the staging does not fit
            const int smem = nph == 9    ? ZBlock<9>::smem_bytes(nraw, ncp)
                             : nph == 12 ? ZBlock<12>::smem_bytes(nraw, ncp)
                                         : ZBlock<14>::smem_bytes(nraw, ncp);
            return smem <= ZPCfg<T, N>::SMEM_MAX;
        } else {
            return false;
        }
    }
    // the z kernel a variant option selects: GNSS_VARIANT_WARPSPEC and _REGISTER both name the register kernel (k_zpipe
    // in FP32, k_zws in FP64; the first name where zws_fits, and AUTO answers so in FP64), _STAGED k_zphys
    static int zkernel(int zvariant, int nph, int nraw, int nout, int ncp) {
        const bool ws = zvariant == GNSS_VARIANT_WARPSPEC || (zvariant == GNSS_VARIANT_AUTO && sizeof(T) == 8);
        if (ws && zws_fits(nph, nraw, nout, ncp)) return GNSS_VARIANT_WARPSPEC;
        // AUTO takes a register kernel at every length one serves (measured on ensembles of 16 x 64^3 .. 2 x 192^3 and
        // single jets at 256^3, 512^3)
        return zvariant != GNSS_VARIANT_STAGED && zreg_fits(nph, nraw, ncp) ? GNSS_VARIANT_REGISTER : GNSS_VARIANT_STAGED;
    }
    // diag != nullptr: the register kernel with the fused vorticity sums (cudaErrorNotSupported where none exists)
    static cudaError_t zphys(const FieldSet<T> &f, const ZRecipeSet &zr, int nph, int nraw, int nout,
                             long long nlines, int ncp, int nkz, T scale, T alpha, double dkz, const void *tw,
                             unsigned *err, int nsm, cudaStream_t s, int zvariant, double *diag = nullptr,
                             int nmem = 1, long long ms = 0) {
        if (diag || zkernel(zvariant, nph, nraw, nout, ncp) != GNSS_VARIANT_STAGED)
            return zpipe(f, zr, nph, nraw, nlines, ncp, nkz, scale, alpha, dkz, tw, err, nsm, s, diag, nmem, ms);
        if (nph == 9 && nraw == 10)
            return zphys_n<9, 10>(f, zr, nout, nlines, ncp, nkz, scale, alpha, dkz, tw, err, nsm, s, nmem, ms);
        if (nph == 12 && nraw == 13)
            return zphys_n<12, 13>(f, zr, nout, nlines, ncp, nkz, scale, alpha, dkz, tw, err, nsm, s, nmem, ms);
        if (nph == 14 && nraw == 14)
            return zphys_n<14, 14>(f, zr, nout, nlines, ncp, nkz, scale, alpha, dkz, tw, err, nsm, s, nmem, ms);
        return cudaErrorInvalidValue;
    }
};

template <typename T>
cudaError_t launch_zphys(int n, const FieldSet<T> &f, const ZRecipeSet &zr, int nph, int nraw, int nout,
                                long long nlines, int ncp, int nkz, T scale, T alpha, double dkz, const void *tw,
                                unsigned *err, int nsm, cudaStream_t s, int zvariant, double *diag,
                                int nmem, long long ms) {
    GNSS_SIZE_SWITCH(n, return (ZLaunch<T, NN_>::zphys(f, zr, nph, nraw, nout, nlines, ncp, nkz, scale, alpha, dkz, tw,
                                                      err, nsm, s, zvariant, diag, nmem, ms)));
}
template <typename T> int zkernel_choice(int n, int zvariant, int nph, int nraw, int nout, int ncp) {
    GNSS_SIZE_SWITCH_OR(n, return (ZLaunch<T, NN_>::zkernel(zvariant, nph, nraw, nout, ncp)), return GNSS_VARIANT_STAGED);
}
template <typename T> bool zreg_available(int n, int nph, int nraw, int ncp) {
    GNSS_SIZE_SWITCH_OR(n, return (ZLaunch<T, NN_>::zreg_fits(nph, nraw, ncp)), return false);
}
