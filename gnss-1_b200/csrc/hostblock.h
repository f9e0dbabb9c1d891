// hostblock.h -- host side of a context's device block (make_device_block);
// no device code, so that it also compiles with the host compiler alone.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <vector>

namespace gnss {

// k^2 as the device forms it (ksq3): every product and sum rounded by itself.  What lies in the dealiasing sphere is
// decided here for the tables and on the device for the modes, and a mode on its edge must fall on the same side, so
// `volatile` keeps a host compiler from contracting the products and sums to fused ones.
inline double host_ksq(double a, double b, double c) {
    volatile double aa = a * a, bb = b * b, cc = c * c;
    volatile double ab = aa + bb;
    return ab + cc;
}
inline double host_wavenum(int i, int n, double dk) {
    return i < n / 2 ? dk * (double)i : dk * ((double)i - (double)n);
}

// The tables of the dealiasing sphere for k_passd.  The kept rows of a column are those whose |index| does not exceed
// its bound, since k^2 grows with the row's wavenumber; the bounds use the test k^2 > kmax^2 (solver.cu:36) in the
// reference's order of evaluation.
struct SphereAxis { int n; double dk; };
struct SphereTables {
    // [nky + 1][ncp]: the largest kept |kx| of each (kept ky, kz) column, then the largest kept |ky| of each kz
    // column; -1: none, and in the padding columns from nkz on
    std::vector<short> bound;
    // the x passes' tiles with a mode inside the sphere, kept ky << 8 | column block: those whose first column has
    // one, since the bounds fall with kz
    std::vector<int> tiles;
};
// ky(i): index of the i-th kept ky; nb: columns per tile
template <class Ky>
SphereTables sphere_tables(SphereAxis x, SphereAxis y, SphereAxis z, double kmax2, int nky, Ky ky, int nkz, int ncp,
                           int nb) {
    SphereTables t;
    t.bound.assign((size_t)(nky + 1) * ncp, (short)-1);
    for (int i = 0; i < nky; ++i) {
        short *r = t.bound.data() + (size_t)i * ncp;
        const double ko = host_wavenum(ky(i), y.n, y.dk);
        for (int k = 0, d = x.n / 2; k < nkz; ++k) {
            while (d >= 0 && host_ksq(x.dk * (double)d, ko, host_wavenum(k, z.n, z.dk)) > kmax2) --d;
            r[k] = (short)d;
        }
        for (int b = 0; b < ncp / nb; ++b)
            if (r[b * nb] >= 0) t.tiles.push_back(i << 8 | b);
    }
    short *r = t.bound.data() + (size_t)nky * ncp;
    for (int k = 0, d = y.n / 2; k < nkz; ++k) {
        while (d >= 0 && host_ksq(0.0, y.dk * (double)d, host_wavenum(k, z.n, z.dk)) > kmax2) --d;
        r[k] = (short)d;
    }
    return t;
}

// Copies pageable host memory to the device and waits until it is there.
// cudaMemcpy from pageable memory may return once the data lies in its staging
// buffer, and work on a non-blocking stream does not wait for the stream that
// carries the rest of the copy.  (That stream alone is waited for: a device
// synchronisation would break a capture on another thread, as the server's
// scheduler makes them.)
inline cudaError_t upload_and_wait(void *dst, const void *src, size_t bytes) {
    const cudaError_t e = cudaMemcpy(dst, src, bytes, cudaMemcpyHostToDevice);
    return e == cudaSuccess ? cudaStreamSynchronize(cudaStreamLegacy) : e;
}

// What of the kept box lies inside the sphere: modes (the ones k_update touches after the first step); columns (ky, kz)
// with a kept mode, and those of the x passes' tiles; modes the x forward pass stores (all columns of a tile with the
// rows of its first one).  From the columns' bounds, a few operations each: the box has millions of modes.
struct SphereCount {
    double modes = 0, cols = 0, tile_cols = 0, stored = 0;
};
template <class Ky>
SphereCount count_sphere(SphereAxis x, SphereAxis y, SphereAxis z, double kmax2, int nky, Ky ky, int nkz, int nb) {
    SphereCount n;
    for (int i = 0; i < nky; ++i) {
        const double ko = host_wavenum(ky(i), y.n, y.dk);
        for (int k = 0, d = x.n / 2; k < nkz; ++k) {
            while (d >= 0 && host_ksq(x.dk * (double)d, ko, host_wavenum(k, z.n, z.dk)) > kmax2) --d;
            if (d < 0) break;   // the bounds fall with kz
            const int rows = 2 * d >= x.n ? x.n : 2 * d + 1;
            n.modes += rows;
            n.cols += 1;
            if (k % nb == 0) {
                n.tile_cols += nb;
                n.stored += (double)nb * rows;
            }
        }
    }
    return n;
}

}  // namespace gnss
