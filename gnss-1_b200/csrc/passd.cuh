// passd.cuh -- strided x / y passes with the transform spread over the block
// (N = 48 .. 512).
//
// Same contract as k_pass (PassSpec / PassPtrs).  A tile is N rows of 128
// bytes: 8 elements of 16 bytes (8 FP64 or 16 FP32 columns, pk.cuh), so the 8
// lanes of a quarter warp touch one row and no access to a tile has bank
// conflicts.  Thread (t, u) owns rows t + r N/8 of element u: it copies exactly
// these to shared memory ahead of time (cp.async, two tiles), reads them back
// without a barrier, and the length-N transform runs as two or three Stockham
// stages exchanged in place in the tile; the last stage stores from registers
// to global memory.  Eight elements per thread keep it at 80 registers, 24
// warps per SM (16 at N = 512, whose two tiles fill an SM's shared memory).
//   What bounds it: instruction issue and shared-memory wavefronts (ncu, 512
//   rows: LSU wavefronts 60-65% FP64, 53-56% FP32, issue 38 / 45%), so what is fixed
//   for the launch stays out of the loop: the rows a thread reads and stores
//   as bit masks, work items advanced by the grid size instead of divided,
//   two base pointers (lower and upper half of the rows: the gap of a compact
//   axis lies between them) plus a uniform stride.
//   Measured against the register kernel it replaced (one warp per column, 8
//   FP64 / 16 FP32 warps per SM), the four passes of a step: 512^3 FP64 with
//   two scalars 7.98 -> 6.48 ms, 512^3 FP32 4.09 -> 2.99, 256^3 FP32 0.71 ->
//   0.36, 192^3 FP32 0.36 -> 0.18 ms.
//   The dealiasing sphere: rows outside it are not read, tiles outside it are
//   not visited (21% of the x passes' tiles), and rows no later stage reads
//   are not stored; the bounds are tables of the context (make_device_block).
// A second output of a tile copies the tile again (from L2) rather than hold
// its 8 elements in registers through the first transform.
#pragma once
#include "kernels.cuh"
#include "pk.cuh"

namespace gnss {

// radix of stage s: 512 = 8 8 8, 384 = 8 8 6, 256 = 8 8 4, 192 = 8 8 3, 128 = 8 4 4, 96 = 8 4 3, 64 = 8 8, 48 = 8 6
__host__ __device__ constexpr int pd_radix(int n, int s) {
    if (s == 0) return 8;
    if (s == 1) return n == 48 ? 6 : (n == 128 || n == 96) ? 4 : 8;
    return n / (8 * pd_radix(n, 1));
}
__host__ __device__ constexpr int pd_stages(int n) { return 8 * pd_radix(n, 1) == n ? 2 : 3; }
__host__ __device__ constexpr int pd_span(int n, int s) { return s == 0 ? 1 : s == 1 ? 8 : 8 * pd_radix(n, 1); }

template <typename T, int N> struct PDCfg {
    static constexpr int U = 8;                              // 16-byte elements per tile row
    static constexpr int W = PkOf<T>::W;                     // columns per element
    static constexpr int NB = U * W;                         // columns per tile
    static constexpr int TPC = N == 48 ? 8 : N / 8;   // threads per column element
    static constexpr int NT = U * TPC;
    static constexpr int SMEM = 2 * N * U * 16 + N * 16 + N * 8;   // two tiles, twiddles, row wavenumbers
    // threads per SM the registers are sized for: 80 each, and 96 where 80 spill and few tiles make up for it (48^3
    // FP32 transform 16.5 -> 14.5 us, FP64 step 41.5 -> 37.3; 64^3 FP64 step 41.1 -> 38.7; 64 x 512 x 512 unchanged)
    static constexpr int THREADS = N == 48 || (N == 64 && W == 1) ? 640 : 768;
    static constexpr int FIT = (227 * 1024) / (SMEM + 1024);
    static constexpr int MINB = FIT < THREADS / NT ? FIT : THREADS / NT;
    static constexpr int RL = pd_radix(N, pd_stages(N) - 1);   // radix of the last stage
    // the rows a thread reads and stores in the last stage are those it copies, so no barrier separates them from
    // the next copy
    static constexpr bool OWN_LAST = RL == 8;
};

// One stage: jobs jj = t, t + TPC, ... < N / R.  LD(row) -> element, ST(i, row, element) with i = p R + r;
// SYNC: a barrier between the reads and the writes.
template <typename T, int N, int STAGE, int SIGN, bool SYNC, class LD, class ST>
__device__ __forceinline__ void pd_stage(int t, const CP<typename PkOf<T>::P> *tw, LD ld, ST st) {
    constexpr int TPC = PDCfg<T, N>::TPC;
    constexpr int R = pd_radix(N, STAGE), NS = pd_span(N, STAGE), M = N / R, TSTEP = N / (NS * R);
    constexpr int PER = (M + TPC - 1) / TPC;
    CP<typename PkOf<T>::P> v[PER][R];
#pragma unroll
    for (int p = 0; p < PER; ++p) {
        const int jj = t + p * TPC;
        if (M % TPC == 0 || jj < M) {
            const int k = NS == M ? jj : jj % NS;
            // Every power from the table: as products of three of them the twiddles' error, 3.3e-17, grew to 7 - 9e-17.
            // Each load stands beside its product, else seven twiddles in flight spill (FP64 passes of 384 x 384 x 256:
            // 2.71 ms, 2.19 so); where the powers' addresses, kept from tile to tile, spill too (FP64 192) or make
            // the loads wait (512), they are formed on the way (192^3 319 -> 288 us; 512 x 512 x 256 with two scalars
            // 5.67 -> 5.45 ms; at 384 this spills instead).
            constexpr bool CHAIN = N == 512 || (N == 192 && sizeof(T) == 8);
            const CP<typename PkOf<T>::P> *wr = tw;
            int step = k * TSTEP;
            v[p][0] = ld(jj);
#pragma unroll
            for (int r = 1; r < R; ++r) {
                if constexpr (CHAIN) {
                    asm volatile("" : "+r"(step));
                    wr += step;
                } else {
                    wr = tw + r * k * TSTEP;
                }
                const CP<typename PkOf<T>::P> w = *wr;
                v[p][r] = cmulp(ld(jj + r * M), w.x, w.y);
            }
            PDft<R, SIGN>::run(v[p]);
        }
    }
    if constexpr (SYNC) __syncthreads();
#pragma unroll
    for (int p = 0; p < PER; ++p) {
        const int jj = t + p * TPC;
        if (M % TPC == 0 || jj < M) {
            const int d = (jj / NS) * NS * R + jj % NS;
#pragma unroll
            for (int r = 0; r < R; ++r) st(p * R + r, d + r * NS, v[p][r]);
        }
    }
}

// bits r = 0 .. 7 of the rows t + r N/8 with |row| <= d
template <int N> __device__ __forceinline__ unsigned pd_rows(int t, int d) {
    constexpr int M0 = N / 8;
    if (d >= N / 2) return 0xffu;
    if (d < 0) return 0u;
    const int a = (d - t + M0) / M0;               // rows 0 .. d: r < a (d - t + M0 > 0)
    const int rb = (N - d - t + M0 - 1) / M0;      // rows N - d ..: r >= rb
    return ((1u << a) - 1u) | ((0xffu << rb) & 0xffu);
}

template <typename T, int N, int SIGN, bool GEN = false, bool MB = false>
__global__ void __launch_bounds__(PDCfg<T, N>::NT, PDCfg<T, N>::MINB)
k_passd(const __grid_constant__ PassPtrs<T> Pp, const __grid_constant__ PassSpec sp, const V2<T> *__restrict__ twg) {
    using V = V2<T>;
    using C = PDCfg<T, N>;
    using P = typename PkOf<T>::P;
    using E = CP<P>;
    constexpr int U = C::U, W = C::W, NB = C::NB, TPC = C::TPC, NT = C::NT, M0 = N / 8, TILE = N * U;
    constexpr int LAST = pd_stages(N) - 1;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    E *X = reinterpret_cast<E *>(smem_raw);
    E *tw = X + 2 * TILE;
    P *krow = reinterpret_cast<P *>(tw + N);
    const int tid = threadIdx.x, u = tid % U, t = tid / U;
    const bool own = M0 == TPC || t < M0;   // this thread has rows of stage 0
    const int ntiles = sp.list ? sp.nlist : sp.outer.count() * sp.ncolblk;
    const int nin = sp.nin;
    const int nitems = (MB ? sp.nmem : 1) * nin * ntiles;
    int item = blockIdx.x;
    if (item >= nitems) return;
    for (int i = tid; i < N; i += NT) {
        const V w = twg[i];
        tw[i] = E{PkOf<T>::dup(w.x), PkOf<T>::dup(SIGN > 0 ? -w.y : w.y)};
        if constexpr (W == 1) krow[i] = wavenum(i, sp.n_row, sp.dk_row);
        else krow[i] = pconst<P>((float)sp.dk_row * (float)(i < N / 2 ? i : i - N));
    }
    __syncthreads();
    pdl_wait();
    // what a thread reads and stores, fixed for the launch: the rows t + r M0 that the source / destination has (bit
    // r), the element strides between them, and the gap before the rows of the upper half where they are compact
    unsigned lm = 0, km = 0;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        lm |= (own && sp.row_in.kept(t + r * M0) ? 1u : 0u) << r;
        km |= (sp.row_out.kept(t + r * M0) ? 1u : 0u) << r;
    }
    const int srow = (int)sp.s_row, drow = (int)sp.d_row;
    const int sgap = sp.row_in_compact ? (N - sp.row_in.count()) * srow : 0;
    const int dgap = sp.row_out_compact ? (N - sp.row_out.count()) * drow : 0;
    const int soff = t * srow + u * W, doff = t * drow + u * W;

    // items advance by the grid size
    struct Item { int tt, fi, mi, oc, cb; };
    const int grid = gridDim.x;
    const int g_t = grid % ntiles, g_f = (grid / ntiles) % nin, g_m = MB ? grid / (ntiles * nin) : 0;
    auto locate = [&](Item &q) {   // outer index and column block of tile tt
        if (sp.list) {
            const int e = __ldg(sp.list + q.tt);
            q.oc = e >> 8;
            q.cb = e & 255;
        } else {
            q.oc = sp.cb_magic ? (int)__umulhi((unsigned)q.tt, sp.cb_magic) : q.tt;
            q.cb = q.tt - q.oc * sp.ncolblk;
        }
    };
    auto advance = [&](Item &q) {
        q.tt += g_t;
        q.fi += g_f;
        if (q.tt >= ntiles) { q.tt -= ntiles; ++q.fi; }
        if constexpr (MB) q.mi += g_m;
        if (q.fi >= nin) { q.fi -= nin; if constexpr (MB) ++q.mi; }
        locate(q);
    };
    // bound of the thread's own columns (two 16-bit values) and of the tile's first column
    auto bounds = [&](const Item &q, int &own_b, int &tile_b) {
        own_b = W == 2 ? 0x3fff3fff : 0x3fff;
        tile_b = 0x3fff;
        if (sp.dtab) {
            const short *row = sp.dtab + q.oc * sp.dstride + q.cb * NB;
            if (sp.bound_in) own_b = W == 2 ? __ldg(reinterpret_cast<const int *>(row) + u) : (int)__ldg(row + u);
            if (sp.bound_out) tile_b = __ldg(row);
        }
    };
    auto rows = [&](const Item &q, int own_b) -> unsigned {   // rows read: bits 0-7 first column, 8-15 second
        const int c = q.cb * NB + u * W;
        const unsigned m = c < sp.ncols ? lm & pd_rows<N>(t, (short)own_b) : 0u;
        if constexpr (W == 1) return m;
        return m | ((c + 1 < sp.ncols ? lm & pd_rows<N>(t, own_b >> 16) : 0u) << 8);
    };
    auto prefetch = [&](const Item &q, unsigned m, E *dst) {
        const V *lo = Pp.in[q.fi] + (MB ? q.mi * sp.ms_in : 0LL) +
                      (long long)(sp.outer_in_compact ? q.oc : sp.outer.expand(q.oc)) * sp.s_out + q.cb * NB + soff;
        const V *hi = lo - sgap;
        E *d = dst + tid;   // element (t + r M0, u) of the tile
        if (W == 1 || sp.in16) {
#pragma unroll
            for (int r = 0; r < 8; ++r)
                if ((m >> r) & 1u) cp_async16(d + r * M0 * U, (r < 4 ? lo : hi) + r * (M0 * srow), 16);
        } else {
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                const V *p = (r < 4 ? lo : hi) + r * (M0 * srow);
                if ((m >> r) & 1u) cp_async8(d + r * M0 * U, p, 8);
                if ((m >> (8 + r)) & 1u) cp_async8(reinterpret_cast<V *>(d + r * M0 * U) + 1, p + 1, 8);
            }
        }
    };

    Item cur, nxt;
    cur.fi = (item / ntiles) % nin;
    cur.mi = MB ? item / (ntiles * nin) : 0;
    cur.tt = item % ntiles;
    locate(cur);
    int tile_b, own_b;
    bounds(cur, own_b, tile_b);
    unsigned m = rows(cur, own_b);
    prefetch(cur, m, X);
    cp_async_commit();
    int var = 0, buf = 0, nown = own_b, ntile = tile_b;
    nxt = cur;
    if (item + grid < nitems) {
        advance(nxt);
        bounds(nxt, nown, ntile);
    }
    for (;;) {
        // the next output: another one of this tile (read again, from L2), or the first of the next tile
        const bool more = var + 1 < sp.nvar[cur.fi];
        const int nitem = more ? item : item + grid;
        const bool go = nitem < nitems;
        unsigned nm = m;
        if (go) {
            if (more) {
                prefetch(cur, m, X + (buf ^ 1) * TILE);
            } else {
                nm = rows(nxt, nown);
                prefetch(nxt, nm, X + (buf ^ 1) * TILE);
            }
        }
        cp_async_commit();
        cp_async_wait<1>();
        E *in = X + buf * TILE;
        E v[8];
        if (own) {
            const int mul = sp.vmul[cur.fi][var];
            const E *s = in + tid;
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                v[r] = E{pconst<P>(0.0), pconst<P>(0.0)};
                if ((m >> r) & 1u) {
                    if constexpr (W == 1) {
                        v[r] = s[r * M0 * U];
                    } else {
                        const float4 a = *reinterpret_cast<const float4 *>(&s[r * M0 * U]);
                        const bool b = (m >> (8 + r)) & 1u;
                        v[r] = E{f2(a.x, b ? a.z : 0.0f), f2(a.y, b ? a.w : 0.0f)};
                    }
                }
            }
            if (mul == V_IK_ROW) {
#pragma unroll
                for (int r = 0; r < 8; ++r) {
                    const P kr = krow[t + r * M0];
                    v[r] = E{pneg(kr * v[r].y), kr * v[r].x};
                }
            } else if (GEN && mul != V_ONE) {   // V_LAP
                const int c = cur.cb * NB + u * W;
                const double ko = sp.n_out ? wavenum(sp.outer.expand(cur.oc), sp.n_out, sp.dk_out) : 0.0;
                const double k0 = wavenum(c, sp.n_col, sp.dk_col), k1 = wavenum(c + 1, sp.n_col, sp.dk_col);
#pragma unroll
                for (int r = 0; r < 8; ++r) {
                    const double kr = wavenum(t + r * M0, sp.n_row, sp.dk_row);
                    P k2;
                    if constexpr (W == 1) k2 = -ksq3(kr, ko, k0);
                    else k2 = f2((float)-ksq3(kr, ko, k0), (float)-ksq3(kr, ko, k1));
                    v[r] = E{k2 * v[r].x, k2 * v[r].y};
                }
            }
            PDft<8, SIGN>::run(v);
        }
        __syncthreads();
        if (own) {
#pragma unroll
            for (int r = 0; r < 8; ++r) in[(t * 8 + r) * U + u] = v[r];
        }
        __syncthreads();
        if constexpr (LAST == 2) {
            pd_stage<T, N, 1, SIGN, true>(
                t, tw, [&](int row) -> E { return in[row * U + u]; }, [&](int, int row, E e) { in[row * U + u] = e; });
            __syncthreads();
        }
        // the tile after the next: looked up here, used in the next round
        Item nn = nxt;
        int nnown = nown, nntile = ntile;
        if (!more && nitem + grid < nitems) {
            advance(nn);
            bounds(nn, nnown, nntile);
        }
        V *dlo = Pp.out[sp.vout[cur.fi][var]] + (MB ? cur.mi * sp.ms_out : 0LL) +
                 (long long)(sp.outer_out_compact ? cur.oc : sp.outer.expand(cur.oc)) * sp.d_out + cur.cb * NB + doff;
        V *dhi = dlo - dgap;
        const int left = sp.out_ncols - (cur.cb * NB + u * W);
        auto put = [&](V *p, E e) {
            if constexpr (W == 1) {
                *p = V{e.x, e.y};
            } else {
                float x0, x1, y0, y1;
                f2_get(e.x, x0, x1);
                f2_get(e.y, y0, y1);
                if (sp.out16) {
                    *reinterpret_cast<float4 *>(p) = float4{x0, y0, x1, y1};
                } else {
                    p[0] = V{x0, y0};
                    if (left > 1) p[1] = V{x1, y1};
                }
            }
        };
        const unsigned sm = left > 0 ? km & pd_rows<N>(t, tile_b) : 0u;
        pd_stage<T, N, LAST, SIGN, false>(
            t, tw, [&](int row) -> E { return in[row * U + u]; },
            [&](int i, int row, E e) {
                if constexpr (C::OWN_LAST) {   // row t + i M0
                    if ((sm >> i) & 1u) put((i < 4 ? dlo : dhi) + i * (M0 * drow), e);
                } else {
                    const int dist = row <= N / 2 ? row : N - row;
                    if (left > 0 && sp.row_out.kept(row) && dist <= tile_b)
                        put((row < N / 2 ? dlo : dhi) + (row - t) * drow, e);
                }
            });
        if (!go) break;
        if constexpr (!C::OWN_LAST) __syncthreads();   // the tiles are free
        if (more) {
            ++var;
        } else {
            var = 0;
            cur = nxt;
            tile_b = ntile;
            nxt = nn;
            nown = nnown;
            ntile = nntile;
            m = nm;
        }
        item = nitem;
        buf ^= 1;
    }
}

}  // namespace gnss
