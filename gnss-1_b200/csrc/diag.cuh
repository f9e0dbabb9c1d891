// diag.cuh -- turbulence diagnostics of a spectral state (calcTurbStats_mgpu,
// statistics.cu:2039-2156): the spectral sums behind Vrms, KE, epsilon, the
// integral length and chi, the rms of each vorticity component and the volume
// average of |omega| over the grid, and the mean profiles along y.
//
// Spectral sums run over the full spectrum through the kz mirror (weight 1 on
// kz = 0 and kz = nz/2, 2 elsewhere, as calcVrmsKernel_mgpu's kp = NZ - k
// branch, statistics.cu:1505-1532), Kahan-compensated per thread and reduced
// in a fixed order.  The vorticity statistics are taken, as in the
// reference, over the physical vorticity (statistics.cu:2097-2106): a
// spectral (Parseval) sum would differ from the grid average whenever
// Nyquist modes survive the dealiasing (grids thinner than nx along y or z),
// because the inverse transform drops their imaginary parts.  The
// mean profile of a field along y (calcYprof, statistics.cu:1943-2003: the
// average over x and z) is the inverse DFT in y of its kx = kz = 0 modes.
#pragma once
#include "kernels.cuh"

namespace gnss {

constexpr int TURB_SUMS = 4;   // e, k^2 e, e/(2|k|), k^2 |s|^2
constexpr int VORT_SUMS = 4;   // |w|, w_x^2, w_y^2, w_z^2 over the grid

template <typename T> struct TurbMode { V2<T> f[4]; };

template <typename T>
__global__ void __launch_bounds__(STAT_THREADS, WALK_PER_SM)
k_turb_partial(const __grid_constant__ FieldSet<T> st, int has_s, Geom g, double *__restrict__ partial) {
    using V = V2<T>;
    Kahan acc[TURB_SUMS];
    spec_sum<T, TurbMode<T>>(
        g,
        [&](long long i) {
            return TurbMode<T>{{st.p[0][i], st.p[1][i], st.p[2][i], has_s ? st.p[3][i] : V{}}};
        },
        [&](const SpecWalk &w, const TurbMode<T> &m) {
            const V a = m.f[0], b = m.f[1], c = m.f[2];
            const double ax = a.x, ay = a.y, bx = b.x, by = b.y, cx = c.x, cy = c.y;
            const double e = ax * ax + ay * ay + bx * bx + by * by + cx * cx + cy * cy;
            const double ms = abs2(m.f[3]);
            if (e == 0.0 && ms == 0.0) return;
            const double k1 = wavenum(w.kx, g.nx, g.dkx), k2 = wavenum(w.ky, g.ny, g.dky), k3 = wavenum(w.kz, g.nz, g.dkz);
            const double ksq = ksq3(k1, k2, k3);
            const double wt = (w.kz == 0 || 2 * w.kz == g.nz) ? 1.0 : 2.0;
            acc[0].add(wt * e);                                      // calcVrmsKernel_mgpu
            acc[1].add(wt * ksq * e);                                // calcEpsilonKernel_mgpu
            if (ksq > 0.0) acc[2].add(wt * e / (2.0 * sqrt(ksq)));   // calcIntegralLengthKernel_mgpu (:1693-1700)
            if (has_s) acc[3].add(wt * ksq * ms);                    // calcScalarDissipationKernel_mgpu
        });
    block_row<TURB_SUMS>(acc, partial + blockIdx.x * TURB_SUMS);
}

// Sums over the physical points of the three padded real vorticity fields
// [nx][ny][2 nz2]: sqrt(w1^2 + w2^2 + w3^2) (VectorMagnitude + volumeAverage,
// statistics.cu:2005-2040, 1211-1283) and w1^2, w2^2, w3^2
// (volumeAverage_rms, :1285-1305); one row of VORT_SUMS partials per block.
template <typename T>
__global__ void __launch_bounds__(STAT_THREADS)
k_vort_partial(const T *__restrict__ w1, const T *__restrict__ w2, const T *__restrict__ w3, Geom g,
               double *__restrict__ partial) {
    Kahan acc[VORT_SUMS];
    const long long npts = (long long)g.nx * g.ny * g.nz;
    for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < npts;
         p += (long long)gridDim.x * blockDim.x) {
        const long long line = p / g.nz;
        const long long idx = line * 2 * g.nz2 + (p - line * g.nz);
        const double a = w1[idx], b = w2[idx], c = w3[idx];
        acc[0].add(sqrt(a * a + b * b + c * c));
        acc[1].add(a * a);
        acc[2].add(b * b);
        acc[3].add(c * c);
    }
    block_row<VORT_SUMS>(acc, partial + blockIdx.x * VORT_SUMS);
}

template <int NS>
__global__ void __launch_bounds__(NS * FINAL_WARPS * 32)
k_sums_final(const double *__restrict__ partial, int nblocks, double *__restrict__ out) {
    __shared__ double red[NS][FINAL_WARPS];
    const double v = sum_rows<NS>(partial, nblocks, red);
    if (threadIdx.x % (32 * FINAL_WARPS) == 0) out[threadIdx.x / (32 * FINAL_WARPS)] = v;
}

// Mean profile along y of field f (blockIdx.x), from its kx = kz = 0 modes.
// With the reference's inverse scaling (1/NN, cudafuncs.cu:20-31) the x-z
// average of the physical field is
//   prof[j] = (1/NN) sum_ky Re(f(0, ky, 0) exp(+2 pi i ky j / ny));
// tw holds exp(-2 pi i m / ny).  One point j per thread.  The sum over ky is a
// serial chain (compensated, in the order of ky), so all else is kept out of
// it: the line and the twiddles are read into shared memory first, and the
// twiddle index advances by j instead of by a division.  256 points: 98 -> 13 us.
constexpr int YPROF_THREADS = 64;
constexpr int YPROF_MAX = 512;   // the longest axis
template <typename T>
__global__ void __launch_bounds__(YPROF_THREADS)
k_yprof(const __grid_constant__ FieldSet<T> st, Geom g, const V2<T> *__restrict__ tw, double *__restrict__ prof) {
    __shared__ V2<T> line[YPROF_MAX], w[YPROF_MAX];
    const V2<T> *f = st.p[blockIdx.x];
    double *out = prof + (long long)blockIdx.x * g.ny;
    const int j = blockIdx.y * YPROF_THREADS + threadIdx.x;
    if (!f) {
        if (j < g.ny) out[j] = 0.0;
        return;
    }
    const long long stride = (long long)g.nx * g.nz2;   // ky stride of the (kx = 0, kz = 0) line
    for (int i = threadIdx.x; i < g.ny; i += YPROF_THREADS) {
        line[i] = f[i * stride];
        w[i] = tw[i];
    }
    __syncthreads();
    if (j >= g.ny) return;
    Kahan acc;
    for (int ky = 0, m = 0; ky < g.ny; ++ky) {
        const V2<T> a = line[ky], b = w[m];
        acc.add((double)a.x * (double)b.x + (double)a.y * (double)b.y);   // Re(a conj(w))
        m += j;
        if (m >= g.ny) m -= g.ny;
    }
    out[j] = acc.s / ((double)g.nx * g.ny * g.nz);
}

}  // namespace gnss
