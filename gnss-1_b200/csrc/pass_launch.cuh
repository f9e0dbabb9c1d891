// pass_launch.cuh -- launchers of the x / y passes and of the plain z pass,
// instantiated per precision by pass_f32.cu and pass_f64.cu.
#pragma once
#include "launch.cuh"
#include "passd.cuh"
#include "passtc.cuh"
#include "zreg.cuh"

template <typename T> static const V2<T> *pass_twiddles(const PassPtrs<T> &, const void *tw) {
    return reinterpret_cast<const V2<T> *>(tw);
}

// A persistent pass launch: one block per SM times the blocks that fit
// (looked up once per kernel, from any host thread), at most one per work item.
template <class K, class PP>
static cudaError_t launch_persistent(K kern, std::atomic<int> &per_sm, int nt, int smem, int nsm, long long nitems,
                                     cudaStream_t s, const PP &P, const PassSpec &sp, const void *tw,
                                     unsigned *err = nullptr, bool with_err = false) {
    cudaError_t e = prep_smem(kern, smem);
    if (e != cudaSuccess) return e;
    int ps = per_sm.load(std::memory_order_relaxed);
    if (ps == 0) {
        ps = blocks_per_sm(kern, nt, smem);
        per_sm.store(ps, std::memory_order_relaxed);
    }
    long long grid = (long long)ps * nsm;
    if (grid > nitems) grid = nitems;
    if (with_err) {
        if constexpr (std::is_invocable_v<K, PP, PassSpec, const float2 *, unsigned *>)
            return launch_dep(kern, dim3((unsigned)grid), dim3(nt), smem, s, P, sp, reinterpret_cast<const float2 *>(tw),
                              err);
    } else {
        if constexpr (!std::is_invocable_v<K, PP, PassSpec, const float2 *, unsigned *>)
            return launch_dep(kern, dim3((unsigned)grid), dim3(nt), smem, s, P, sp, pass_twiddles(P, tw));
    }
    return cudaGetLastError();
}

template <typename T, int N> struct PassLaunch {
    // every row starts on a 16-byte boundary if the buffer does
    static bool rows16(long long row, long long outer, long long member) {
        return sizeof(T) == 8 || ((row | outer | member) & 1) == 0;
    }
    // Members of a batch (sp.nmem > 1) run the MB instantiations, which exist for zr_size lengths (batches need the
    // register z kernel, and gnss_batch_supported wants x and y of its lengths); other lengths return
    // cudaErrorNotSupported for a batch.
    static cudaError_t pass(int sign, const PassPtrs<T> &P, const PassSpec &sp, const void *tw, int nsm,
                            cudaStream_t s, int pvariant, unsigned *err) {
        const bool mb = sp.nmem > 1;
        const int ci = (sign < 0 ? 0 : 1) + (mb ? 2 : 0);   // occupancy cache index
        if constexpr (sizeof(T) == 4 && ptc_size(N)) {
            // split-TF32 DFT-GEMM transforms on the tensor cores (tiles of 8 columns)
            if (pvariant == GNSS_VARIANT_TENSOR) {
                using C = PTCfg<N>;
                auto kern = mb ? (sign < 0 ? k_passtc<N, -1, true> : k_passtc<N, +1, true>)
                               : (sign < 0 ? k_passtc<N, -1> : k_passtc<N, +1>);
                static std::atomic<int> per_sm[4];
                PassSpec s8 = sp;
                const int cols = sp.ncols > sp.out_ncols ? sp.ncols : sp.out_ncols;
                s8.ncolblk = (cols + C::NB - 1) / C::NB;
                const long long nitems = (long long)s8.nmem * s8.nin * s8.outer.count() * s8.ncolblk;
                return launch_persistent(kern, per_sm[ci], C::NT, C::SMEM, nsm, nitems, s,
                                         reinterpret_cast<const PassPtrs<float> &>(P), s8, tw, err, true);
            }
        }
        if constexpr (pd_size(N)) {
            // k_passd at every length it serves; GNSS_VARIANT_STAGED keeps k_pass
            if (pvariant != GNSS_VARIANT_STAGED) {
                using C = PDCfg<T, N>;
                PassSpec sd = sp;
                const int cols = sp.ncols > sp.out_ncols ? sp.ncols : sp.out_ncols;
                sd.ncolblk = (cols + C::NB - 1) / C::NB;
                sd.cb_magic = sd.ncolblk == 1 ? 0u
                                              : (unsigned)(((1ULL << 32) + sd.ncolblk - 1) / (unsigned)sd.ncolblk);
                sd.in16 = rows16(sp.s_row, sp.s_out, sp.ms_in);
                sd.out16 = rows16(sp.d_row, sp.d_out, sp.ms_out) && sp.out_ncols % C::W == 0;
                bool gen = false;   // multipliers beyond 1 and i k_row
                for (int i = 0; i < sp.nin; ++i) {
                    sd.in16 = sd.in16 && reinterpret_cast<uintptr_t>(P.in[i]) % 16 == 0;
                    for (int v = 0; v < sp.nvar[i]; ++v) {
                        sd.out16 = sd.out16 && reinterpret_cast<uintptr_t>(P.out[(int)sp.vout[i][v]]) % 16 == 0;
                        gen = gen || sp.vmul[i][v] > V_IK_ROW;
                    }
                }
                const long long nitems =
                    (long long)sp.nmem * sp.nin * (sp.list ? sp.nlist : sp.outer.count() * sd.ncolblk);
                static std::atomic<int> per_sd[8];
                auto kern = sign < 0 ? k_passd<T, N, -1> : gen ? k_passd<T, N, +1, true> : k_passd<T, N, +1>;
                if constexpr (zr_size(N)) {
                    if (mb) kern = sign < 0 ? k_passd<T, N, -1, false, true>
                                   : gen    ? k_passd<T, N, +1, true, true>
                                            : k_passd<T, N, +1, false, true>;
                } else if (mb) {
                    return cudaErrorNotSupported;
                }
                return launch_persistent(kern, per_sd[ci + (gen ? 4 : 0)], C::NT, C::SMEM, nsm,
                                         nitems, s, P, sd, tw);
            }
        }
        const long long nitems = (long long)sp.nmem * sp.nin * sp.outer.count() * sp.ncolblk;
        using C = PassCfg<T, N>;
        static std::atomic<int> per_sm[4];
        if (mb) {
            if constexpr (zr_size(N)) {
                auto kern = sign < 0 ? k_pass<T, N, -1, true> : k_pass<T, N, +1, true>;
                return launch_persistent(kern, per_sm[ci], C::NT, C::SMEM, nsm, nitems, s, P, sp, tw);
            } else {
                return cudaErrorNotSupported;
            }
        }
        auto kern = sign < 0 ? k_pass<T, N, -1> : k_pass<T, N, +1>;
        return launch_persistent(kern, per_sm[ci], C::NT, C::SMEM, nsm, nitems, s, P, sp, tw);
    }
    static cudaError_t zpass(int dir, const FieldSet<T> &f, int nfields, long long nlines, int nz2, T scale,
                             const void *tw, cudaStream_t s) {
        // register transforms where they round no more than k_zpass; forward + inverse with all passes:
        // 192 x 256 x 128 FP64 241 us with k_zpass, 202 with k_zline; FP32 123 and 113 us, 256 x 256 x 512 689 and 526
        if constexpr (zline_size(N, sizeof(T) == 8)) {
            using Z = ZRCfg<T, N>;
            const int smem = (Z::FINE_ROWS * 32 + ZLINE_WARPS * Z::SCR) * (int)sizeof(V2<T>);
            auto kern = dir < 0 ? k_zline<T, N, -1> : k_zline<T, N, +1>;
            cudaError_t e = prep_smem(kern, smem);
            if (e != cudaSuccess) return e;
            const long long np = nlines / 2;
            const long long blocks = (np + ZLINE_WARPS - 1) / ZLINE_WARPS;
            kern<<<dim3((unsigned)std::min<long long>(blocks, 148LL * 16), (unsigned)nfields), ZLINE_WARPS * 32, smem, s>>>(
                f, (int)np, nz2, scale, reinterpret_cast<const V2<T> *>(tw));
            return cudaGetLastError();
        } else {
            using C = ZCfg<T, N>;
            long long npairs = (nlines + 1) / 2;
            dim3 grid((unsigned)((npairs + ZWARPS - 1) / ZWARPS), (unsigned)nfields);
            const V2<T> *t = reinterpret_cast<const V2<T> *>(tw);
            auto kern = dir < 0 ? k_zpass<T, N, -1> : k_zpass<T, N, +1>;
            cudaError_t e = prep_smem(kern, C::SMEM);
            if (e != cudaSuccess) return e;
            kern<<<grid, ZWARPS * 32, C::SMEM, s>>>(f, nlines, nz2, scale, t);
            return cudaGetLastError();
        }
    }
};

template <typename T>
cudaError_t launch_pass(int n, int sign, const PassPtrs<T> &P, const PassSpec &sp, const void *tw, int nsm,
                               cudaStream_t s, int pvariant, unsigned *err) {
    GNSS_SIZE_SWITCH(n, return (PassLaunch<T, NN_>::pass(sign, P, sp, tw, nsm, s, pvariant, err)));
}
template <typename T>
cudaError_t launch_zpass(int n, int dir, const FieldSet<T> &f, int nfields, long long nlines, int nz2, T scale,
                                const void *tw, cudaStream_t s) {
    GNSS_SIZE_SWITCH(n, return (PassLaunch<T, NN_>::zpass(dir, f, nfields, nlines, nz2, scale, tw, s)));
}
