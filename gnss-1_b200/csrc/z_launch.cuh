// z_launch.cuh -- launchers of the fused z stage, instantiated per precision
// by z_f32.cu and z_f64.cu.
#pragma once
#include "launch.cuh"
#include "zreg.cuh"

// GNSS_VARIANT_AUTO takes a register z kernel at every length one serves
// (measured on ensembles of 16 x 64^3 .. 2 x 192^3 and single jets at 256^3, 512^3)
__host__ __device__ constexpr bool zr_auto_z(int n) { return zr_size(n); }

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
    // register-resident line transforms (N = 64 .. 512, zr_size) when their shared memory fits
    // diag != nullptr: the instantiation that also writes per-block vorticity sums there
    template <int NPH, int NRAW>
    static cudaError_t zreg_k(const FieldSet<T> &f, const ZRecipeSet &zr, int nout, long long nlines, int ncp, int nkz,
                              T scale, T alpha, double dkz, const void *tw, unsigned *err, int nsm, cudaStream_t s,
                              double *diag, int nmem, long long ms) {
        if constexpr (zr_size(N)) {
            const int smem = ZRCfg<T, N>::smem_bytes(NPH, NRAW, ncp);
            if (smem > ZPCfg<T, N>::SMEM_MAX) return cudaErrorNotSupported;
            auto kern = diag ? k_zreg<T, N, NPH, NRAW, true>
                             : (nmem > 1 ? k_zreg<T, N, NPH, NRAW, false, true> : k_zreg<T, N, NPH, NRAW, false>);
            cudaError_t e = prep_smem(kern, smem);
            if (e != cudaSuccess) return e;
            const int per_sm = blocks_per_sm(kern, NPH * 32, smem);
            const long long mpairs = nlines / 2, npairs = mpairs * nmem;
            long long grid = (long long)per_sm * nsm;
            if (grid > npairs) grid = npairs;
            if (diag && grid > STAT_BLOCKS) grid = STAT_BLOCKS;   // one row of sums per block
            return launch_dep(kern, dim3((unsigned)grid), dim3(NPH * 32), smem, s, f, zr, nout, npairs, ncp, nkz, scale,
                              alpha, dkz, reinterpret_cast<const V2<T> *>(tw), err, diag, mpairs, ms);
        } else {
            (void)f; (void)zr; (void)nout; (void)nlines; (void)ncp; (void)nkz; (void)scale; (void)alpha; (void)dkz;
            (void)tw; (void)err; (void)nsm; (void)s; (void)diag; (void)nmem; (void)ms;
            return cudaErrorNotSupported;
        }
    }
    // warp-specialised register z kernel (N = 256, 512; FP32 with 9 quantities and 4 products, FP64 with 9 and 4
    // or 12 and 5)
    static constexpr bool zws_size() { return N == 256 || N == 512; }
    template <int NPH, int NRAW>
    static cudaError_t zws_kt(const FieldSet<T> &f, const ZRecipeSet &zr, int nout, long long nlines, int ncp,
                              int nkz, T scale, T alpha, double dkz, const void *tw, unsigned *err, int nsm,
                              cudaStream_t s, int nmem, long long ms) {
        if (nmem > 1) return cudaErrorNotSupported;   // batches run the register z kernel
        if constexpr (zws_size()) {
            constexpr int NOUT = zws_nout<NPH>();
            const int smem = ZRCfg<T, N>::smem_bytes_ws(NPH, NOUT, NRAW, ncp);
            auto kern = k_zws<T, N, NPH, NRAW>;
            cudaError_t e = prep_smem(kern, smem);
            if (e != cudaSuccess) return e;
            const int nt = (NPH + NOUT) * 32;
            const int per_sm = blocks_per_sm(kern, nt, smem);
            const long long mpairs = nlines / 2, npairs = mpairs * nmem;
            long long grid = (long long)per_sm * nsm;
            if (grid > npairs) grid = npairs;
            return launch_dep(kern, dim3((unsigned)grid), dim3(nt), smem, s, f, zr, nout, npairs, ncp, nkz, scale, alpha,
                              dkz, reinterpret_cast<const V2<T> *>(tw), err, mpairs, ms);
        } else {
            (void)f; (void)zr; (void)nout; (void)nlines; (void)ncp; (void)nkz; (void)scale; (void)alpha; (void)dkz;
            (void)tw; (void)err; (void)nsm; (void)s; (void)nmem; (void)ms;
            return cudaErrorNotSupported;
        }
    }
    static cudaError_t zws_k(const FieldSet<T> &f, const ZRecipeSet &zr, int nph, int nraw, int nout, long long nlines,
                             int ncp, int nkz, T scale, T alpha, double dkz, const void *tw, unsigned *err, int nsm,
                             cudaStream_t s, int nmem, long long ms) {
        if (nph == 9 && nraw == 10)
            return zws_kt<9, 10>(f, zr, nout, nlines, ncp, nkz, scale, alpha, dkz, tw, err, nsm, s, nmem, ms);
        if (nph == 12 && nraw == 13)
            return zws_kt<12, 13>(f, zr, nout, nlines, ncp, nkz, scale, alpha, dkz, tw, err, nsm, s, nmem, ms);
        return cudaErrorNotSupported;
    }
    static bool zws_fits(int nph, int nraw, int nout, int ncp) {
        if constexpr (zws_size()) {
            const bool fp32 = sizeof(T) == 4 && nph == 9 && nraw == 10 && nout == 4;
            const bool fp64 = sizeof(T) == 8 && ((nph == 9 && nraw == 10 && nout == 4) ||
                                                 (nph == 12 && nraw == 13 && nout == 5));
            return (fp32 || fp64) && ZRCfg<T, N>::smem_bytes_ws(nph, nout, nraw, ncp) <= ZPCfg<T, N>::SMEM_MAX;
        } else {
            return false;
        }
    }
    static bool zreg_fits(int nph, int nraw, int ncp) {
        if constexpr (zr_size(N))
            return ZRCfg<T, N>::smem_bytes(nph, nraw, ncp) <= ZPCfg<T, N>::SMEM_MAX;
        else
            return false;
    }
    // the z kernel a variant option selects: GNSS_VARIANT_WARPSPEC, _REGISTER or _STAGED
    // AUTO: the warp-specialised kernel in FP64 where it fits (17 or 13 warps per SM against k_zreg's 12 or 9;
    // measured at 512^3 with two scalars: z 6.18 -> 5.53 ms, one scalar 5.48 -> 4.59 ms; 256^3 0.95 -> 0.80 ms),
    // the register kernel in FP32 (there k_zws measured slower: 2.52 -> 2.70 ms at 512^3)
    static int zkernel(int zvariant, int nph, int nraw, int nout, int ncp) {
        const bool ws = zvariant == GNSS_VARIANT_WARPSPEC || (zvariant == GNSS_VARIANT_AUTO && sizeof(T) == 8);
        if (ws && zws_fits(nph, nraw, nout, ncp)) return GNSS_VARIANT_WARPSPEC;
        const bool reg = zvariant == GNSS_VARIANT_REGISTER || zvariant == GNSS_VARIANT_WARPSPEC ||
                         (zvariant == GNSS_VARIANT_AUTO && zr_auto_z(N));
        return reg && zreg_fits(nph, nraw, ncp) ? GNSS_VARIANT_REGISTER : GNSS_VARIANT_STAGED;
    }
    // diag != nullptr: the register kernel with the fused vorticity sums (cudaErrorNotSupported where it does
    // not exist)
    static cudaError_t zphys(const FieldSet<T> &f, const ZRecipeSet &zr, int nph, int nraw, int nout,
                             long long nlines, int ncp, int nkz, T scale, T alpha, double dkz, const void *tw,
                             unsigned *err, int nsm, cudaStream_t s, int zvariant, double *diag = nullptr,
                             int nmem = 1, long long ms = 0) {
        if (diag) {
            if (!zreg_fits(nph, nraw, ncp)) return cudaErrorNotSupported;
            if (nph == 9 && nraw == 10)
                return zreg_k<9, 10>(f, zr, nout, nlines, ncp, nkz, scale, alpha, dkz, tw, err, nsm, s, diag, 1, 0);
            if (nph == 12 && nraw == 13)
                return zreg_k<12, 13>(f, zr, nout, nlines, ncp, nkz, scale, alpha, dkz, tw, err, nsm, s, diag, 1, 0);
            if (nph == 14 && nraw == 14)
                return zreg_k<14, 14>(f, zr, nout, nlines, ncp, nkz, scale, alpha, dkz, tw, err, nsm, s, diag, 1, 0);
            return cudaErrorInvalidValue;
        }
        const int kern = zkernel(zvariant, nph, nraw, nout, ncp);
        if (kern == GNSS_VARIANT_WARPSPEC)
            return zws_k(f, zr, nph, nraw, nout, nlines, ncp, nkz, scale, alpha, dkz, tw, err, nsm, s, nmem, ms);
        if (kern == GNSS_VARIANT_REGISTER) {
            if (nph == 9 && nraw == 10)
                return zreg_k<9, 10>(f, zr, nout, nlines, ncp, nkz, scale, alpha, dkz, tw, err, nsm, s, nullptr, nmem,
                                     ms);
            if (nph == 12 && nraw == 13)
                return zreg_k<12, 13>(f, zr, nout, nlines, ncp, nkz, scale, alpha, dkz, tw, err, nsm, s, nullptr, nmem,
                                      ms);
            if (nph == 14 && nraw == 14)
                return zreg_k<14, 14>(f, zr, nout, nlines, ncp, nkz, scale, alpha, dkz, tw, err, nsm, s, nullptr, nmem,
                                      ms);
            return cudaErrorInvalidValue;
        }
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
