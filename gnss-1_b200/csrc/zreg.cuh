// zreg.cuh -- fused z pass with register-resident line transforms
// (N = 64, 96, 128, 192, 256, 512).
//
// Same work as k_zphys (kz factors and vorticity combinations, C2R of every
// physical quantity of a line pair, the pointwise products, R2C of the
// products), with a different line transform: a warp holds its line in
// registers, E = N/32 elements per lane.  For N = 64 .. 192 (E = 2, 3, 4, 6)
// the transform uses lane shuffles only (zs_fft).  For N = 256, 512 it runs
//   N = E * 32,   32 = E * G   (G = 32/E lanes per group)
//   step A: E-point DFT in registers over elements lane + 32 m, twiddle
//           W_N^(lane k1);
//   one transpose through a padded per-warp scratch;
//   step B: E-point DFT in registers, twiddle W_32^(j k2'), and a G-point
//           DFT across the lanes of a group with shuffles.
// so a line crosses shared memory once per transform (instead of once per
// radix-8 stage).  The C2R packing is done while loading the registers.  The
// forward transform is the inverse one's flow graph reversed (zr_fft_rev), so
// it takes the products where the inverse transforms leave their lines and
// ends with the modes in order.  Two kernels use these pieces: k_zpipe (FP32)
// and k_zws (FP64).
#pragma once
#include "kernels.cuh"
#include "pk.cuh"

#include <type_traits>

namespace gnss {

// cos(2 pi e / 32) for e = 0..8; other angles by symmetry.
__host__ __device__ constexpr double cos32_tab(int e) {
    return e == 0   ? 1.0
           : e == 1 ? 0.98078528040323044912618223613424
           : e == 2 ? 0.92387953251128675612818318939679
           : e == 3 ? 0.83146961230254523707878837761791
           : e == 4 ? 0.70710678118654752440084436210485
           : e == 5 ? 0.55557023301960222474283081394853
           : e == 6 ? 0.38268343236508977172845998403040
           : e == 7 ? 0.19509032201612826784828486847702
                    : 0.0;
}
__host__ __device__ constexpr double cos32(int e) {
    e = ((e % 32) + 32) % 32;
    return e <= 8 ? cos32_tab(e) : e <= 16 ? -cos32_tab(16 - e) : e <= 24 ? -cos32_tab(e - 16) : cos32_tab(32 - e);
}
__host__ __device__ constexpr double sin32(int e) { return cos32(e - 8); }

// v * exp(S 2 pi i e / 32) with compile-time e.  FINE (FP32): the factor in two parts, without its rounding error.
template <int S, int EXP, bool FINE = false, typename V> __device__ __forceinline__ V mul_w32(V v) {
    using T = decltype(v.x);
    constexpr int e = ((EXP % 32) + 32) % 32;
    if constexpr (e == 0) {
        return v;
    } else if constexpr (e == 8) {
        return mul_si<S>(v);
    } else if constexpr (e == 16) {
        return V{-v.x, -v.y};
    } else if constexpr (e == 24) {
        return mul_si<-S>(v);
    } else {
        constexpr T c = (T)cos32(e);
        constexpr T s = (T)((double)S * sin32(e));
        if constexpr (FINE && sizeof(T) == 4) {
            constexpr T cl = (T)(cos32(e) - (double)c), sl = (T)((double)S * sin32(e) - (double)s);
            return V{fma(v.x, c, fma(-v.y, s, v.x * cl - v.y * sl)), fma(v.x, s, fma(v.y, c, v.x * sl + v.y * cl))};
        }
        return V{v.x * c - v.y * s, v.x * s + v.y * c};
    }
}

// 16-point DFT in natural order: n = 4 n1 + n2, k = k1 + 4 k2.
template <int S, bool FINE = false, typename V> __device__ __forceinline__ void dft16(V *v) {
#pragma unroll
    for (int n2 = 0; n2 < 4; ++n2) dft4<S>(v[n2], v[4 + n2], v[8 + n2], v[12 + n2]);
    // v[4 k1 + n2] = y[n2][k1]; twiddle W_16^(n2 k1) = W_32^(2 n2 k1)
    v[5] = mul_w32<S, 2, FINE>(v[5]);
    v[9] = mul_w32<S, 4, FINE>(v[9]);
    v[13] = mul_w32<S, 6, FINE>(v[13]);
    v[6] = mul_w32<S, 4, FINE>(v[6]);
    v[10] = mul_w32<S, 8, FINE>(v[10]);
    v[14] = mul_w32<S, 12, FINE>(v[14]);
    v[7] = mul_w32<S, 6, FINE>(v[7]);
    v[11] = mul_w32<S, 12, FINE>(v[11]);
    v[15] = mul_w32<S, 18, FINE>(v[15]);
#pragma unroll
    for (int k1 = 0; k1 < 4; ++k1) dft4<S>(v[4 * k1], v[4 * k1 + 1], v[4 * k1 + 2], v[4 * k1 + 3]);
    // v[4 k1 + k2] = X[k1 + 4 k2] -> natural order
    V t[16];
#pragma unroll
    for (int k1 = 0; k1 < 4; ++k1)
#pragma unroll
        for (int k2 = 0; k2 < 4; ++k2) t[k1 + 4 * k2] = v[4 * k1 + k2];
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = t[i];
}
template <int S, typename V> struct Dft<16, S, V> {
    static __device__ __forceinline__ void run(V *v) { dft16<S>(v); }
};

template <typename T, int N> struct ZRCfg {
    static_assert(zr_size(N), "register transforms serve N = 64, 96, 128, 192, 256, 512");
    static constexpr int E = N / 32;                    // elements per lane
    static constexpr bool SHFL = E != 8 && E != 16;     // lane-shuffle scheme (no transpose)
    static constexpr int G = SHFL ? 1 : 32 / E;         // lanes per group in step B (transpose scheme)
    static constexpr int S = 32 + G;                    // transpose row stride (conflict-free both ways)
    // table rows: the powers W_N^(lane r), r = 1 2 3 4 (and 8 12 where E = 16), of the transpose scheme's step-A
    // twiddles, so that each other one is a product of two; FP64 lines of 512 points keep to r = 1 2 4 8 (POW2), since
    // their staged lines fill the shared memory (two scalars, 192 kept kz columns).  The shuffle scheme reads
    // W_N^(lane k1), k1 = 1 .. E-1, then W_32^lane.
    static constexpr bool POW2 = E == 16 && sizeof(T) == 8;
    static constexpr int ROWS = SHFL ? E : POW2 ? 4 : (E == 16 ? 6 : 4);
    // line padding.  Transpose scheme: a warp's stores of a transform's
    // output (zr_fft: lane groups j = lane % G at E^2 sigma(j) apart,
    // lanes of a group on consecutive entries) take one wavefront per 128
    // bytes when every group starts on its own bank range, so PADP entries
    // follow every PADB = E^2: 64 bytes for E = 16 (two groups), 32 for E = 8
    // (four) (measured at 512^3: FP64 z 6.42 -> 6.20 ms, FP32 2.61 -> 2.53 ms;
    // at 256^3 FP64 1.11 -> 0.96 ms).  Shuffle scheme: c entries per E, so
    // that a warp's stores of one output element (positions q + E j,
    // j = 0 .. 31) fall in distinct bank pairs.
    static constexpr int PADB = SHFL ? E : E * E;
    static constexpr int PADP = SHFL ? 0 : (E == 16 ? 64 : 32) / (int)sizeof(V2<T>);
    static constexpr int PADC = SHFL ? ((E & 1) ? 2 : 1) : 0;
    __host__ __device__ static constexpr int pidx(int n) {
        return SHFL ? n + PADC * (n / E) : n + PADP * (n / PADB);
    }
    static constexpr int PL = SHFL ? N + PADC * 32 : N + PADP * (N / PADB);   // line length in shared memory
    static constexpr int SCR = SHFL ? PL : E * S;       // scratch line per warp (transposes, physical line)
    static_assert(SCR >= PL, "scratch holds a padded line");
    // index into the length-N table exp(-2 pi i j / N) of twiddle-table entry i
    __host__ __device__ static constexpr int tw_index(int i) {
        const int row = i >> 5, l = i & 31;
        if (SHFL) return row < E - 1 ? (l * (row + 1)) % N : (E * l) % N;
        return (l * (POW2 ? 1 << row : row < 4 ? row + 1 : 4 * row - 8)) % N;
    }
    // the table of k_zline: every power W_N^(lane k1), k1 = 1 .. E-1 (and W_32^lane)
    static constexpr int FINE_ROWS = SHFL ? E : E - 1;
    __host__ __device__ static constexpr int tw_fine(int i) {
        const int row = i >> 5, l = i & 31;
        return row < E - 1 ? (l * (row + 1)) % N : (E * l) % N;
    }
};

// 6-point DFT in natural order: n = 3 n1 + 2 n2, k = 3 k1 + 4 k2 (mod 6), two
// 3-point DFTs and one 2-point stage without twiddles.
template <int S, typename V> struct Dft<6, S, V> {
    static __device__ __forceinline__ void run(V *v) {
        V a[3] = {v[0], v[2], v[4]}, b[3] = {v[3], v[5], v[1]};
        Dft<3, S, V>::run(a);
        Dft<3, S, V>::run(b);
#pragma unroll
        for (int k2 = 0; k2 < 3; ++k2) {
            v[(4 * k2) % 6] = cadd(a[k2], b[k2]);
            v[(3 + 4 * k2) % 6] = csub(a[k2], b[k2]);
        }
    }
};

// Output slot of a lane group member after the G-point cross-lane DFT.
template <int G> __device__ __forceinline__ int zr_sigma(int j) {
    return G == 2 ? j : ((j >> 1) | ((j & 1) << 1));
}

// v * W_32^(j Q): lane group member j multiplies, the others keep v
template <int S, int Q, int G, bool FINE, typename V> __device__ __forceinline__ V zr_tw32(V v, int j) {
    using T = decltype(v.x);
    if constexpr (G == 2) {
        if (j) v = mul_w32<S, Q, FINE>(v);
        return v;
    } else if constexpr (FINE && sizeof(T) == 4) {
        if (j == 1) return mul_w32<S, Q, true>(v);
        if (j == 2) return mul_w32<S, 2 * Q, true>(v);
        if (j == 3) return mul_w32<S, 3 * Q, true>(v);
        return v;
    } else {
        constexpr T c1 = (T)cos32(Q), s1 = (T)((double)S * sin32(Q));
        constexpr T c2 = (T)cos32(2 * Q), s2 = (T)((double)S * sin32(2 * Q));
        constexpr T c3 = (T)cos32(3 * Q), s3 = (T)((double)S * sin32(3 * Q));
        if (j == 0) return v;
        const T c = j == 1 ? c1 : j == 2 ? c2 : c3;
        const T s = j == 1 ? s1 : j == 2 ? s2 : s3;
        return V{v.x * c - v.y * s, v.x * s + v.y * c};
    }
}
template <int S, int G, int Q, int E, bool FINE, typename V> __device__ __forceinline__ void zr_tw32_all(V *x, int j) {
    if constexpr (Q < E) {
        x[Q] = zr_tw32<S, Q, G, FINE>(x[Q], j);
        zr_tw32_all<S, G, Q + 1, E, FINE>(x, j);
    }
}

// elementwise products of two real lines (x, y)
__device__ __forceinline__ float2 lmul(float2 a, float2 b) {
    float2 o;
    f2_get(f2(a.x, a.y) * f2(b.x, b.y), o.x, o.y);
    return o;
}
__device__ __forceinline__ double2 lmul(double2 a, double2 b) { return double2{a.x * b.x, a.y * b.y}; }
__device__ __forceinline__ float2 lfma(float2 a, float2 b, float2 c) {
    float2 o;
    f2_get(pfma(f2(a.x, a.y), f2(b.x, b.y), f2(c.x, c.y)), o.x, o.y);
    return o;
}
__device__ __forceinline__ double2 lfma(double2 a, double2 b, double2 c) {
    return double2{a.x * b.x + c.x, a.y * b.y + c.y};
}
template <typename V> __device__ __forceinline__ V lneg(V a) { return V{-a.x, -a.y}; }
// and of one
__device__ __forceinline__ double lmul(double a, double b) { return a * b; }
__device__ __forceinline__ double lfma(double a, double b, double c) { return a * b + c; }
template <> __device__ __forceinline__ double lneg<double>(double a) { return -a; }

template <typename V> __device__ __forceinline__ V shfl_xor_v(V v, int m) {
    return V{__shfl_xor_sync(0xffffffffu, v.x, m), __shfl_xor_sync(0xffffffffu, v.y, m)};
}

// Transpose layout of zr_fft in a warp's own scratch line: row k1 of 32 + G
// entries (conflict-free both ways).
template <typename T, int N> struct ZrScratch {
    __device__ __forceinline__ int operator()(int k1, int i) const { return k1 * ZRCfg<T, N>::S + i; }
};

// The 32-point DFT across lanes, all E elements of a lane at once, in radix-2
// steps taken in pairs (4 4 2): of the two twiddles of a pair only a factor
// i has to be applied between its steps, the rest is one product after them
// (before them in the reversed flow graph).  zs32_tw: that product's factors
// W_32^(SIGN e) of the steps 16, 8 and 4, 2.
template <typename T, int SIGN> struct Zs32 {
    V2<T> w16, w4;
    bool i16, i4;
    __device__ __forceinline__ Zs32(int lane, const V2<T> *w32) {
        const int b0 = lane & 1, b1 = (lane >> 1) & 1, b2 = (lane >> 2) & 1, b3 = (lane >> 3) & 1, b4 = lane >> 4;
        w16 = w32[(lane & 7) * (b4 + 2 * b3)];
        w4 = w32[4 * b0 * (b2 + 2 * b1)];
        if (SIGN > 0) { w16.y = -w16.y; w4.y = -w4.y; }
        i16 = b4 && b3;
        i4 = b2 && b1;
    }
};
// p + x on the lanes without bit h, p - x on those with it (p: the partner's value)
template <typename T> __device__ __forceinline__ V2<T> zs_step(int lane, V2<T> x, int h) {
    const T s = (lane & h) ? T(-1) : T(1);
    return lfma(V2<T>{s, s}, x, shfl_xor_v(x, h));
}

// Length-N DFT (N = 32 E, E = 2, 3, 4, 6) of one line held by a warp, with
// lane shuffles only.  On entry x[m] is element lane + 32 m; on return x[q]
// is element q + E bitrev5(lane) of the transform.  n = lane + 32 m,
// k = k1 + E k2: an E-point DFT over m in registers, the twiddle
// W_N^(lane k1), then for every k1 a 32-point DFT across the lanes
// (decimation in frequency).  tws rows: W_N^(lane k1), k1 = 1 .. E-1, then
// W_32^lane (exp(-2 pi i ./.), conjugated for SIGN > 0).
template <typename T, int N, int SIGN>
__device__ __forceinline__ void zs_fft(int lane, V2<T> *x, const V2<T> *tws) {
    using V = V2<T>;
    constexpr int E = N / 32;
    Dft<E, SIGN, V>::run(x);
#pragma unroll
    for (int k1 = 1; k1 < E; ++k1) {
        V t = tws[32 * (k1 - 1) + lane];
        if (SIGN > 0) t.y = -t.y;
        x[k1] = cmul(x[k1], t);
    }
    const Zs32<T, SIGN> z(lane, tws + 32 * (E - 1));
#pragma unroll
    for (int q = 0; q < E; ++q) {
        x[q] = zs_step<T>(lane, x[q], 16);
        if (z.i16) x[q] = mul_si<SIGN>(x[q]);
    }
#pragma unroll
    for (int q = 0; q < E; ++q) x[q] = cmul(zs_step<T>(lane, x[q], 8), z.w16);
#pragma unroll
    for (int q = 0; q < E; ++q) {
        x[q] = zs_step<T>(lane, x[q], 4);
        if (z.i4) x[q] = mul_si<SIGN>(x[q]);
    }
#pragma unroll
    for (int q = 0; q < E; ++q) x[q] = cmul(zs_step<T>(lane, x[q], 2), z.w4);
#pragma unroll
    for (int q = 0; q < E; ++q) x[q] = zs_step<T>(lane, x[q], 1);
}

// x[k1] *= W_N^(SIGN lane k1), the step-A twiddles of zr_fft (transpose scheme): FINE reads every power from the table
// of k_zline, else those outside the table are products of entries.  (With rows for the powers of two only, powers like
// 7 and 13 take two products: a step's FP32 right-hand side was 2% and 5% further off at 256 and 512 points, in the
// same time.)
template <typename T, int N, int SIGN, bool FINE>
__device__ __forceinline__ void zr_twiddle(int lane, V2<T> *x, const V2<T> *tws) {
    using V = V2<T>;
    constexpr int E = ZRCfg<T, N>::E;
    auto tw_at = [&](int b) {
        V t = tws[32 * b + lane];
        if (SIGN > 0) t.y = -t.y;
        return t;
    };
    if constexpr (FINE) {
#pragma unroll
        for (int r = 1; r < E; ++r) x[r] = cmul(x[r], tw_at(r - 1));
    } else {
        constexpr bool POW2 = ZRCfg<T, N>::POW2;
        const V w1 = tw_at(0), w2 = tw_at(1), w3 = POW2 ? cmul(w1, w2) : tw_at(2), w4 = tw_at(POW2 ? 2 : 3);
        if constexpr (E == 16) {
            const V w8 = tw_at(POW2 ? 3 : 4);
            x[8] = cmul(x[8], w8);
            x[9] = cmul(x[9], cmul(w1, w8));
            x[10] = cmul(x[10], cmul(w2, w8));
            x[11] = cmul(x[11], cmul(w3, w8));
            if constexpr (POW2) {   // no register for the power 12 across these (k_zws, two scalars: z 5.10 against 5.35 ms)
                x[12] = cmul(x[12], cmul(w4, w8));
                x[13] = cmul(x[13], cmul(cmul(w1, w4), w8));
                x[14] = cmul(x[14], cmul(cmul(w2, w4), w8));
                x[15] = cmul(x[15], cmul(cmul(w3, w4), w8));
            } else {
                const V w12 = tw_at(5);
                x[12] = cmul(x[12], w12);
                x[13] = cmul(x[13], cmul(w1, w12));
                x[14] = cmul(x[14], cmul(w2, w12));
                x[15] = cmul(x[15], cmul(w3, w12));
            }
        }
        x[1] = cmul(x[1], w1);
        x[2] = cmul(x[2], w2);
        x[3] = cmul(x[3], w3);
        x[4] = cmul(x[4], w4);
        x[5] = cmul(x[5], cmul(w1, w4));
        x[6] = cmul(x[6], cmul(w2, w4));
        x[7] = cmul(x[7], cmul(w3, w4));
    }
}

template <int E, int S, bool FINE, typename V> __device__ __forceinline__ void zr_dft(V *x) {
    if constexpr (E == 16) dft16<S, FINE>(x);
    else Dft<E, S, V>::run(x);
}

// Length-N DFT of one line held by a warp.  On entry x[m] is element
// lane + 32 m; on return x[q] is element k1 + E q + E^2 zr_sigma(j) of the
// transform, with k1 = lane / G, j = lane % G.  The one transpose goes
// through scr at offsets at(k1, i) (row k1 = 0..E-1, entry i = 0..31);
// tws: the twiddle table of ZRCfg (FINE: the one of k_zline).
template <typename T, int N, int SIGN, bool FINE = false>
__device__ __forceinline__ void zr_fft(int lane, V2<T> *x, V2<T> *scr, const V2<T> *tws) {
    const ZrScratch<T, N> at;
    using V = V2<T>;
    using Z = ZRCfg<T, N>;
    constexpr int E = Z::E, G = Z::G;
    if constexpr (Z::SHFL) {   // N = 64, 96, 128, 192: no transpose
        (void)scr;
        (void)at;
        zs_fft<T, N, SIGN>(lane, x, tws);
        return;
    } else {
    zr_dft<E, SIGN, FINE>(x);
    zr_twiddle<T, N, SIGN, FINE>(lane, x, tws);
#pragma unroll
    for (int k1 = 0; k1 < E; ++k1) scr[at(k1, lane)] = x[k1];
    __syncwarp();
    const int k1 = lane / G, j = lane % G;
#pragma unroll
    for (int l = 0; l < E; ++l) x[l] = scr[at(k1, G * l + j)];
    __syncwarp();
    zr_dft<E, SIGN, FINE>(x);
    zr_tw32_all<SIGN, G, 1, E, FINE>(x, j);
    // G-point DFT across the group: each radix-2 step is p + s x with s = +1 on
    // the lower and -1 on the upper member (p the partner's value)
    if constexpr (G == 2) {
        const T sg = j == 0 ? T(1) : T(-1);
#pragma unroll
        for (int q = 0; q < E; ++q) {
            const V p = shfl_xor_v(x[q], 1);
            x[q] = V{p.x + sg * x[q].x, p.y + sg * x[q].y};
        }
    } else {
        const int j0 = j & 1, j1 = j >> 1;
        const T s1 = j1 == 0 ? T(1) : T(-1), s0 = j0 == 0 ? T(1) : T(-1);
#pragma unroll
        for (int q = 0; q < E; ++q) {
            const V p = shfl_xor_v(x[q], 2);
            V c = V{p.x + s1 * x[q].x, p.y + s1 * x[q].y};
            if (j0 && j1) c = mul_si<SIGN>(c);
            const V p2 = shfl_xor_v(c, 1);
            x[q] = V{p2.x + s0 * c.x, p2.y + s0 * c.y};
        }
    }
    }
}

// The reverse of zr_fft: on entry x[q] is the element that zr_fft returns there,
// on return x[m] is element lane + 32 m of the length-N DFT.  With input index
// n = k1 + E k2 and output index k = l + 32 m, W_N^(n k) = W_E^(k1 m)
// W_N^(k1 l) W_32^(k2 l): a 32-point DFT over k2 (k2 = q + E s, l = G l' + j:
// a G-point DFT across the lanes, W_32^(q j), an E-point DFT over q), the
// transpose, W_N^(k1 l) and an E-point DFT over k1.
template <typename T, int N, int SIGN, bool FINE = false>
__device__ __forceinline__ void zr_fft_rev(int lane, V2<T> *x, V2<T> *scr, const V2<T> *tws) {
    using V = V2<T>;
    using Z = ZRCfg<T, N>;
    constexpr int E = Z::E, G = Z::G;
    if constexpr (Z::SHFL) {   // the reverse of zs_fft: bit-reversed input, decimation in time
        (void)scr;
        const Zs32<T, SIGN> z(lane, tws + 32 * (E - 1));
#pragma unroll
        for (int q = 0; q < E; ++q) x[q] = cmul(zs_step<T>(lane, x[q], 1), z.w4);
#pragma unroll
        for (int q = 0; q < E; ++q) {
            x[q] = zs_step<T>(lane, x[q], 2);
            if (z.i4) x[q] = mul_si<SIGN>(x[q]);
        }
#pragma unroll
        for (int q = 0; q < E; ++q) x[q] = cmul(zs_step<T>(lane, x[q], 4), z.w16);
#pragma unroll
        for (int q = 0; q < E; ++q) {
            x[q] = zs_step<T>(lane, x[q], 8);
            if (z.i16) x[q] = mul_si<SIGN>(x[q]);
        }
#pragma unroll
        for (int q = 0; q < E; ++q) x[q] = zs_step<T>(lane, x[q], 16);
#pragma unroll
        for (int k1 = 1; k1 < E; ++k1) {
            V t = tws[32 * (k1 - 1) + lane];
            if (SIGN > 0) t.y = -t.y;
            x[k1] = cmul(x[k1], t);
        }
    } else {
        const int k1 = lane / G, j = lane % G;
        if constexpr (G == 2) {
            const T sg = j == 0 ? T(1) : T(-1);
#pragma unroll
            for (int q = 0; q < E; ++q) {
                const V p = shfl_xor_v(x[q], 1);
                x[q] = V{p.x + sg * x[q].x, p.y + sg * x[q].y};
            }
        } else {
            const T s0 = (j & 1) ? T(-1) : T(1), s1 = (j & 2) ? T(-1) : T(1);
#pragma unroll
            for (int q = 0; q < E; ++q) {
                const V p = shfl_xor_v(x[q], 1);
                V c = V{p.x + s0 * x[q].x, p.y + s0 * x[q].y};
                if (j == 3) c = mul_si<SIGN>(c);
                const V p2 = shfl_xor_v(c, 2);
                x[q] = V{p2.x + s1 * c.x, p2.y + s1 * c.y};
            }
        }
        zr_tw32_all<SIGN, G, 1, E, FINE>(x, j);
        zr_dft<E, SIGN, FINE>(x);
        const ZrScratch<T, N> at;
#pragma unroll
        for (int l = 0; l < E; ++l) scr[at(k1, G * l + j)] = x[l];
        __syncwarp();
#pragma unroll
        for (int k = 0; k < E; ++k) x[k] = scr[at(k, lane)];
        __syncwarp();
        zr_twiddle<T, N, SIGN, FINE>(lane, x, tws);
    }
    zr_dft<E, SIGN, FINE>(x);
}

// C2R packing of one physical quantity (recipe rc: +-raw[r0] times (i kz)^ikz0, minus raw[r1] times (i kz)^ikz1
// where there is a second term) into x[m] = Z_n, n = lane + 32 m: Z_k = A_k + i B_k and Z_{N-k} = conj A_k + i conj B_k
// from the raw line pairs (line A: ncp values, then line B; the first nkz are the kept modes), the imaginary parts of
// A, B at k = 0 and N/2 ignored.  Each kept mode is read once: element n's mirror N - n lies in lane 32 - l, element
// E - 1 - m (lane 0: E - m), and gets there by shuffle.
// FORM >= 0 fixes the recipe (bit 0: kz on the first term, bit 1: a second term, bit 2: kz on it), -1 tests it at run
// time.  One copy for the plain lines and one for all others serve most kernels; a copy per recipe (FIXED) makes a
// 13-warp block stall on instruction fetches (FP64, 512^3, one scalar: z 4.71 against 4.24 ms) but pays in the 17-warp
// block with its 96 registers (two scalars: 5.10 against 5.58 ms).
template <typename T, int N, int FORM>
__device__ __forceinline__ void zl_pack_form(int lane, V2<T> *x, const ZRecipe rc, const V2<T> *a0, const V2<T> *a1,
                                             int ncp, int nkz, const T *tkz) {
    using V = V2<T>;
    constexpr int E = N / 32, H = (E + 1) / 2;
    const int mirror = (32 - lane) & 31;
    const bool two = FORM < 0 ? rc.r[1] >= 0 : (FORM & 2) != 0, kz0 = FORM < 0 ? rc.ikz[0] != 0 : (FORM & 1) != 0;
    const bool kz1 = FORM < 0 ? rc.ikz[1] != 0 : (FORM & 4) != 0;
    auto mode = [&](int k, V &a, V &b) {
        a = a0[k];
        b = a0[ncp + k];
        if (kz0) {
            const T kz = tkz[k];
            a = V{-kz * a.y, kz * a.x};
            b = V{-kz * b.y, kz * b.x};
        }
        if (two) {
            V c = a1[k], d = a1[ncp + k];
            if (kz1) {
                const T kz = tkz[k];
                c = V{-kz * c.y, kz * c.x};
                d = V{-kz * d.y, kz * d.x};
            }
            a = csub(a, c);
            b = csub(b, d);
        }
    };
#pragma unroll
    for (int m = 0; m < E; ++m) x[m] = V{T(0), T(0)};
#pragma unroll
    for (int m = 0; m < H; ++m) {
        if (32 * m >= nkz) continue;   // uniform: no kept mode in this element
        const int k = lane + 32 * m;
        V a = V{T(0), T(0)}, b = a;
        if (k < nkz && 2 * k <= N) {
            mode(k, a, b);
            if ((m == 0 && lane == 0) || (E % 2 == 1 && 2 * k == N)) { a.y = T(0); b.y = T(0); }
        }
        const V lo = V{a.x - b.y, a.y + b.x}, hi = V{a.x + b.y, b.x - a.y};
        const V in = V{__shfl_sync(0xffffffffu, hi.x, mirror), __shfl_sync(0xffffffffu, hi.y, mirror)};
        if (m > 0 && lane == 0) x[E - m] = hi;
        if (E % 2 == 1 && m == H - 1) {   // middle element: k <= N/2 in lanes 0 .. 16
            x[m] = lane <= 16 ? lo : in;
        } else {
            x[m] = lo;
            x[E - 1 - m] = lane == 0 ? V{T(0), T(0)} : in;
        }
    }
    if (E % 2 == 0 && 2 * nkz > N) {   // lane 0 of element E/2 is the Nyquist mode
        V a, b;
        mode(N / 2, a, b);
        if (lane == 0) x[E / 2] = V{a.x, b.x};
    }
}

template <typename T, int N, bool FIXED = false>
__device__ __forceinline__ void zl_pack(int lane, V2<T> *x, const ZRecipe rc, const V2<T> *a0, const V2<T> *a1, int ncp,
                                        int nkz, const T *tkz) {
    if constexpr (FIXED) {
        const int form = (rc.ikz[0] ? 1 : 0) | (rc.r[1] >= 0 ? (rc.ikz[1] ? 6 : 2) : 0);
        if (form == 0) zl_pack_form<T, N, 0>(lane, x, rc, a0, a1, ncp, nkz, tkz);
        else if (form == 1) zl_pack_form<T, N, 1>(lane, x, rc, a0, a1, ncp, nkz, tkz);
        else if (form == 2) zl_pack_form<T, N, 2>(lane, x, rc, a0, a1, ncp, nkz, tkz);
        else if (form == 3) zl_pack_form<T, N, 3>(lane, x, rc, a0, a1, ncp, nkz, tkz);
        else zl_pack_form<T, N, 6>(lane, x, rc, a0, a1, ncp, nkz, tkz);
    } else if (rc.r[1] < 0 && !rc.ikz[0]) {
        zl_pack_form<T, N, 0>(lane, x, rc, a0, a1, ncp, nkz, tkz);
    } else {
        zl_pack_form<T, N, -1>(lane, x, rc, a0, a1, ncp, nkz, tkz);
    }
}

// R2C unpacking of x[m] = Z_(lane + 32 m): A_k = (Z_k + conj Z_{N-k})/2, B_k = (Z_k - conj Z_{N-k})/(2i) of the kept
// modes to the line pair at d (line A: ncp values, then line B; columns beyond N/2 are zero).
template <typename T, int N>
__device__ __forceinline__ void zl_unpack(int lane, const V2<T> *x, V2<T> *d, int ncp) {
    using V = V2<T>;
    constexpr int E = N / 32;
    const int mirror = (32 - lane) & 31;
#pragma unroll
    for (int m = 0; m <= E / 2; ++m) {
        if (32 * m >= ncp) continue;   // uniform
        const int k = lane + 32 * m;
        const V s = lane == 0 ? x[(E - m) % E] : x[E - 1 - m];
        const V zm = V{__shfl_sync(0xffffffffu, s.x, mirror), __shfl_sync(0xffffffffu, s.y, mirror)};
        const V zk = x[m];
        V A = V{T(0.5) * (zk.x + zm.x), T(0.5) * (zk.y - zm.y)};
        V B = V{T(0.5) * (zk.y + zm.y), T(-0.5) * (zk.x - zm.x)};
        if (2 * k > N) A = B = V{T(0), T(0)};
        if (k < ncp) {
            d[k] = A;
            d[ncp + k] = B;
        }
    }
    for (int k = lane + 32 * (E / 2 + 1); k < ncp; k += 32) d[k] = d[ncp + k] = V{T(0), T(0)};   // padding of short lines
}

// Physical lines and their products.  A warp leaves a physical line in shared
// memory where its transform ends: x[q] of zr_fft at zl_base(lane) + q
// zl_stride() of the line, which is its element's place (PADB / PADC padding:
// no bank conflicts), and the forward warps read the products' factors at the same
// places.  Quantities: 0 u, 1 v, 2 w, 3 w1, 4 w2, 5 w3, 6 sx, 7 sy, 8 sz,
// [9 cx, 10 cy, 11 cz], [12 c, 13 lap s].
template <typename T, int N> __device__ __forceinline__ int zl_base(int lane) {
    using Z = ZRCfg<T, N>;
    if constexpr (Z::SHFL)
        return (Z::E + Z::PADC) * (int)(__brev((unsigned)lane) >> 27);
    else
        return lane / Z::G + (Z::E * Z::E + Z::PADP) * zr_sigma<Z::G>(lane % Z::G);
}
template <typename T, int N> __host__ __device__ constexpr int zl_stride() {
    return ZRCfg<T, N>::SHFL ? 1 : ZRCfg<T, N>::E;
}
// The plain z pass (gnss_forward / gnss_inverse) with register transforms, one
// warp per pair of lines of one field: DIR < 0 real padded lines -> nz2 complex
// per line, DIR > 0 the reverse, scaled, with the padding reals zeroed; in
// place.  Modes go between global memory and registers, points through a
// shared line, so that both sides are coalesced.  A field has an even number
// of lines.
//   Bound by HBM and by how many lines are in flight: a warp holds one pair at
// a time, so four warps per block and as many blocks as fit keep loads going
// while others transform.  Measured against k_zpass (a shared-memory round trip
// per radix-8 stage), forward + inverse of a 192 x 256 x 128 FP64 field, all
// six passes: 241 -> 202 us.
//   It must not round more than k_zpass.  With twiddles formed as products and
// FP32 constants the error of transforms along z (relative RMS, 256 and 512
// points) was 1.07 and 1.10 times k_zpass's in FP32, 1.03 and 1.01 in FP64;
// FINE, at no measurable cost here, makes it 0.98 and 0.97, 1.00 and 0.97.
// 64 points in FP32 stay on k_zpass, which rounds 2.2% less there and takes the
// same time; the other lane-shuffle lengths are within 1% of it.
__host__ __device__ constexpr bool zline_size(int n, bool fp64) { return zr_size(n) && (fp64 || n != 64); }
constexpr int ZLINE_WARPS = 4;
template <typename T, int N, int DIR>
__global__ void __launch_bounds__(ZLINE_WARPS * 32)
k_zline(const __grid_constant__ FieldSet<T> f, int npairs, int nz2, T scale, const V2<T> *__restrict__ tw) {
    using V = V2<T>;
    using Z = ZRCfg<T, N>;
    constexpr int E = Z::E, ST = zl_stride<T, N>(), M = N / 32;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    V *tws = reinterpret_cast<V *>(smem_raw);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    V *line = tws + Z::FINE_ROWS * 32 + warp * Z::SCR;
    for (int i = threadIdx.x; i < Z::FINE_ROWS * 32; i += ZLINE_WARPS * 32) tws[i] = tw[Z::tw_fine(i)];
    __syncthreads();
    V *field = f.p[blockIdx.y];
    for (int pair = blockIdx.x * ZLINE_WARPS + warp; pair < npairs; pair += gridDim.x * ZLINE_WARPS) {
        V *modes = field + (long long)pair * 2 * nz2;
        T *ra = reinterpret_cast<T *>(modes), *rb = ra + 2 * nz2;
        V *at = line + zl_base<T, N>(lane);
        V x[E];
        if constexpr (DIR < 0) {
#pragma unroll
            for (int m = 0; m < M; ++m) {
                const int n = lane + 32 * m;
                line[Z::pidx(n)] = V{ra[n], rb[n]};
            }
            __syncwarp();
#pragma unroll
            for (int q = 0; q < E; ++q) x[q] = at[q * ST];
            __syncwarp();
            zr_fft_rev<T, N, -1, true>(lane, x, line, tws);
            zl_unpack<T, N>(lane, x, modes, nz2);
        } else {
            const ZRecipe rc{{0, -1}, {0, 0}, {1, 1}, {0, 0}};
            zl_pack_form<T, N, 0>(lane, x, rc, modes, modes, nz2, nz2, nullptr);
            zr_fft<T, N, +1, true>(lane, x, line, tws);
#pragma unroll
            for (int q = 0; q < E; ++q) at[q * ST] = x[q];
            __syncwarp();
#pragma unroll
            for (int m = 0; m < M; ++m) {
                const int n = lane + 32 * m;
                const V z = line[Z::pidx(n)];
                ra[n] = z.x * scale;
                rb[n] = z.y * scale;
            }
            if (lane < 2 * nz2 - N) ra[N + lane] = rb[N + lane] = T(0);
        }
        __syncwarp();   // the line is free
    }
}

// The inverse transforms leave the lines unscaled; their 1/N^3 enters as
// scale^2 on u, v, w (one factor of every product), except with the colloid
// term, whose products have none of them: there every line is scaled.
template <int NPH> __host__ __device__ constexpr bool zr_fold_scale() { return NPH < 14; }
template <typename T, int NPH> __device__ __forceinline__ T zr_line_scale(int q, T scale) {
    return zr_fold_scale<NPH>() ? (q < 3 ? scale * scale : T(1)) : scale;
}
// Product f at this lane's points: (w x u)_f (crossProductKernel_mgpu,
// solver.cu:139-164) for f < 3, u . grad s (dotKernel_mgpu, solver.cu:342-356)
// for 3, u . grad c and the colloid term (colloidAdvectionKernel_mgpu,
// solver.cu:374-388) for 4.  With DIAG each of the first four warps
// also adds the vorticity sums of a quarter of the points to acc
// (ZR_VORT_SUMS: |w|, w_x^2, w_y^2, w_z^2, both lines;
// statistics.cu:1211-1305).
constexpr int ZR_VORT_SUMS = 4;
template <typename T, int N, int NPH, bool DIAG>
__device__ __forceinline__ void zl_product(int f, int lane, V2<T> *x, const V2<T> *lines, T alpha, T scale, double *acc) {
    using V = V2<T>;
    using Z = ZRCfg<T, N>;
    constexpr int E = Z::E, ST = zl_stride<T, N>(), L = Z::SCR;
    const V *p = lines + zl_base<T, N>(lane);
    if constexpr (DIAG) {   // the FP64 sums shared out: with one warp on all of them the others
        // waited for it (256^3 FP32 432 us against 331, 325 without the sums)
        const double s = zr_fold_scale<NPH>() ? (double)scale : 1.0;
        for (int q = f; q < (f < 4 ? E : 0); q += 4) {
            const V w1 = p[3 * L + q * ST], w2 = p[4 * L + q * ST], w3 = p[5 * L + q * ST];
            const double ax = s * w1.x, ay = s * w2.x, az = s * w3.x, bx = s * w1.y, by = s * w2.y, bz = s * w3.y;
            acc[0] += sqrt(ax * ax + ay * ay + az * az) + sqrt(bx * bx + by * by + bz * bz);
            acc[1] += ax * ax + bx * bx;
            acc[2] += ay * ay + by * by;
            acc[3] += az * az + bz * bz;
        }
    }
    if (f < 3) {
        // w2 w - w3 v, w3 u - w1 w, w1 v - w2 u
        const V *a = p + (f == 2 ? 3 : f + 4) * L, *b = p + (f == 0 ? 2 : f - 1) * L;
        const V *c = p + (f == 0 ? 5 : f + 2) * L, *d = p + (f == 0 ? 1 : f == 1 ? 2 : 0) * L;
#pragma unroll
        for (int q = 0; q < E; ++q) x[q] = lfma(a[q * ST], b[q * ST], lneg(lmul(c[q * ST], d[q * ST])));
    } else {
        const V *g = p + (f == 3 ? 6 : 9) * L;
#pragma unroll
        for (int q = 0; q < E; ++q)
            x[q] = lfma(p[2 * L + q * ST], g[2 * L + q * ST],
                        lfma(p[L + q * ST], g[L + q * ST], lmul(p[q * ST], g[q * ST])));
        if constexpr (NPH >= 14) {
            if (f == 4) {
                const V al = V{alpha, alpha};
#pragma unroll
                for (int q = 0; q < E; ++q) {
                    const V *h = p + q * ST;
                    V dr = lmul(h[13 * L], h[12 * L]);
#pragma unroll
                    for (int i = 0; i < 3; ++i) dr = lfma(h[(9 + i) * L], h[(6 + i) * L], dr);
                    x[q] = lfma(al, dr, x[q]);
                }
            }
        }
    }
}

// Shared memory and block shape of k_zpipe: one physical line per inverse
// warp (its transposes run in it, too), transpose scratch per forward warp
// (lengths with a transpose), the staged raw line pairs, an mbarrier, the kz
// table.
template <int NPH> __host__ __device__ constexpr int z_nout() { return NPH >= 12 ? 5 : 4; }
template <typename T, int N, int NPH> struct ZPipe {   // FP32
    using Z = ZRCfg<T, N>;
    static constexpr int NOUT = z_nout<NPH>(), NT = (NPH + NOUT) * 32;
    static constexpr int LINE = Z::SCR;
    static constexpr int FSCR = Z::SHFL ? 0 : Z::SCR;
    // blocks per SM the registers are sized for
    static constexpr int MINB = NPH <= 9 ? (N <= 192 ? 3 : 2) : NPH == 12 || N <= 192 ? 2 : 1;
    __host__ __device__ static constexpr int smem_bytes(int nraw, int ncp) {
        return (Z::ROWS * 32 + NPH * LINE + NOUT * FSCR + nraw * 2 * ncp) * (int)sizeof(V2<T>) + 16 + ncp * (int)sizeof(T);
    }
};

// The fused z stage in FP32 as a pipeline over line pairs, NPH inverse and NOUT
// forward warps per block; block b handles line pairs b, b + gridDim.x, ... of
// all members of a batch (npairs in all, mpairs per member, members ms
// elements apart).  Between two block barriers,
//   A  the inverse warps pack pair p + 1 (registers) while the forward warps
//      read pair p's physical lines and form its products (registers);
//   B  the inverse warps transform p + 1 and leave its physical lines while
//      the forward warps transform p's products and store them over raw
//      fields 0 .. NOUT-1 of the pair.
// Every warp carries one line in registers and the products never pass through
// shared memory.  The raw lines of the pair after the next arrive by
// cp.async.bulk (CTA-local, no multicast) during B; a wait that times out
// sets bit 0 of *err and the block stops.  With DIAG the block writes one row
// of ZR_VORT_SUMS vorticity sums over its points to diag[blockIdx.x], for the
// statistics of the state the step starts from.
//   What bounds it (ncu, 512-point lines): issue 57%, shared-memory wavefronts
// 63%.  Against a block of NPH warps of which NOUT run the forward transforms
// after a products phase (two more barriers, NPH - NOUT warps idle): 512^3 one
// scalar 2.52 -> 2.08 ms, 256^3 one scalar 0.380 -> 0.314, two scalars 0.725 ->
// 0.402 ms (there one block per SM before).  In FP64 the forward warps' reads
// of the factors (96 lines of 512 bytes per product) bound phase A: 512^3 two
// scalars 5.95 ms against 5.10 of k_zws.
template <typename T, int N, int NPH, int NRAW, bool DIAG = false, bool MB = false>
__global__ void __launch_bounds__(ZPipe<T, N, NPH>::NT, ZPipe<T, N, NPH>::MINB)
k_zpipe(const __grid_constant__ FieldSet<T> f, const __grid_constant__ ZRecipeSet zr, long long npairs, int ncp,
        int nkz, T scale, T alpha, double dkz, const V2<T> *__restrict__ tw, unsigned *__restrict__ err,
        double *__restrict__ diag, long long mpairs, long long ms) {
    using V = V2<T>;
    using Z = ZRCfg<T, N>;
    using C = ZPipe<T, N, NPH>;
    constexpr int E = Z::E, ST = zl_stride<T, N>();
    double acc[DIAG ? ZR_VORT_SUMS : 1] = {};
    const int rawf = 2 * ncp;
    const unsigned raw_bytes = (unsigned)(rawf * sizeof(V));
    extern __shared__ __align__(16) unsigned char smem_raw[];
    V *tws = reinterpret_cast<V *>(smem_raw);
    V *lines = tws + Z::ROWS * 32;
    V *fscr = lines + NPH * C::LINE;
    V *raw = fscr + C::NOUT * C::FSCR;
    uint64_t *bar = reinterpret_cast<uint64_t *>(raw + NRAW * rawf);
    T *tkz = reinterpret_cast<T *>(bar + 2);   // kz wavenumbers of the kept modes (ncp entries)
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    long long next = blockIdx.x;
    if (next >= npairs) return;   // uniform for the block
    for (int i = threadIdx.x; i < Z::ROWS * 32; i += C::NT) tws[i] = tw[Z::tw_index(i)];
    for (int k = threadIdx.x; k < ncp; k += C::NT) tkz[k] = (T)wavenum(k, N, dkz);
    if (threadIdx.x == 0) {
        mbar_init(bar, 1);
        mbar_fence_init();
    }
    __syncthreads();
    pdl_wait();
    const WaitCtl wc(err);
    auto issue = [&](long long p, bool withhold = false) {
        mbar_arrive_expect_tx(bar, NRAW * raw_bytes);
        if (!withhold)
            for (int q = 0; q < NRAW; ++q)
                bulk_g2s(raw + q * rawf, f.p[q] + pair_offset<MB>(p, mpairs, ms, rawf), raw_bytes, bar);
    };
    if (threadIdx.x == 0) issue(next, wc.withhold);
    const int step = gridDim.x;
    // barriers 1 (A ends) and 2 (B ends) over the whole block, reached from both loops the same number of times
    const SyncNamed end_b{2, C::NT};
    if (warp < NPH) {   // inverse warps: pair `next`
        const ZRecipe rc = zr.q[warp];
        const T ls = zr_line_scale<T, NPH>(warp, scale);
        const V lsc = V{ls, ls};
        V *const line = lines + warp * C::LINE;
        unsigned parity = 0;
        for (; next < npairs; next += step) {
            V x[E];
            const bool ok = mbar_wait_bounded(bar, parity, wc.limit);
            zl_pack<T, N>(lane, x, rc, raw + rc.r[0] * rawf, raw + rc.r[1] * rawf, ncp, nkz, tkz);
            if (bar_named_or(1, C::NT, !ok)) {   // the raw lines and the physical lines have been read
                if (threadIdx.x == 0) {
                    atomicOr(err, 1u);
                    mbar_wait_bounded(bar, parity, wc.limit);   // let an overdue copy land before leaving
                }
                return;
            }
            parity ^= 1u;
            if (threadIdx.x == 0 && next + step < npairs) {
                fence_proxy_async_smem();
                issue(next + step);
            }
            zr_fft<T, N, +1>(lane, x, line, tws);   // ends its scratch reads with __syncwarp
            V *d = line + zl_base<T, N>(lane);
#pragma unroll
            for (int q = 0; q < E; ++q) d[q * ST] = lmul(x[q], lsc);
            end_b();   // the physical lines of `next` are complete
        }
        bar_named_or(1, C::NT, false);   // the forward warps' last pair
    } else {            // forward warps: the pair before
        const int q = warp - NPH;
        V *const scr = fscr + q * C::FSCR;
        if (bar_named_or(1, C::NT, false)) return;
        end_b();
        for (;;) {
            V x[E];
            zl_product<T, N, NPH, DIAG>(q, lane, x, lines, alpha, scale, acc);
            if (bar_named_or(1, C::NT, false)) return;
            zr_fft_rev<T, N, -1>(lane, x, scr, tws);
            zl_unpack<T, N>(lane, x, f.p[q] + pair_offset<MB>(next, mpairs, ms, rawf), ncp);
            next += step;
            if (next >= npairs) break;
            end_b();
        }
    }
    if constexpr (DIAG) {   // the sums lie in the lanes of four warps: added in a fixed order
        __shared__ double red[ZR_VORT_SUMS][4];
        if (warp >= NPH && warp < NPH + 4) {
#pragma unroll
            for (int q = 0; q < ZR_VORT_SUMS; ++q) {
                double v = acc[q];
                for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
                if (lane == 0) red[q][warp - NPH] = v;
            }
        }
        __syncthreads();
        if (threadIdx.x < ZR_VORT_SUMS) {
            const double *r = red[threadIdx.x];
            diag[blockIdx.x * ZR_VORT_SUMS + threadIdx.x] = ((r[0] + r[1]) + r[2]) + r[3];
        }
    }
}

// Products of one line pair by the whole block (k_zws): quantities in the
// lines `phys`, product f into line f of `out` (both stride SCR).  A thread
// takes both lines' values of a point, or one of them where that fills the
// rounds better (N = 512 with 13 warps: 3 rounds of single values against 2
// of double the work).  DIAG adds the vorticity sums to acc.
template <typename T, int N, int NPH, int NT, bool DIAG>
__device__ __forceinline__ void zr_products(const V2<T> *phys, V2<T> *out, T alpha, T scale, double *acc) {
    using Z = ZRCfg<T, N>;
    constexpr bool HALF = (2 * N + NT - 1) / NT < 2 * ((N + NT - 1) / NT);
    using W = std::conditional_t<HALF, T, V2<T>>;
    constexpr int L = (HALF ? 2 : 1) * Z::SCR;
    for (int i = threadIdx.x; i < (HALF ? 2 : 1) * N; i += NT) {
        const int at = HALF ? 2 * Z::pidx(i >> 1) + (i & 1) : Z::pidx(i);
        const W *p = reinterpret_cast<const W *>(phys) + at;
        const W u = p[0], v = p[L], w = p[2 * L], o1 = p[3 * L], o2 = p[4 * L], o3 = p[5 * L];
        const W sx = p[6 * L], sy = p[7 * L], sz = p[8 * L];
        if constexpr (DIAG) {
            const double s = zr_fold_scale<NPH>() ? (double)scale : 1.0;
            auto add = [&](double ax, double ay, double az) {
                acc[0] += sqrt(ax * ax + ay * ay + az * az);
                acc[1] += ax * ax;
                acc[2] += ay * ay;
                acc[3] += az * az;
            };
            if constexpr (HALF) {
                add(s * o1, s * o2, s * o3);
            } else {
                add(s * o1.x, s * o2.x, s * o3.x);
                add(s * o1.y, s * o2.y, s * o3.y);
            }
        }
        W *o = reinterpret_cast<W *>(out) + at;
        o[0] = lfma(o2, w, lneg(lmul(o3, v)));
        o[L] = lfma(o3, u, lneg(lmul(o1, w)));
        o[2 * L] = lfma(o1, v, lneg(lmul(o2, u)));
        o[3 * L] = lfma(w, sz, lfma(v, sy, lmul(u, sx)));
        if constexpr (NPH >= 12) {
            const W cx = p[9 * L], cy = p[10 * L], cz = p[11 * L];
            W n = lfma(w, cz, lfma(v, cy, lmul(u, cx)));
            if constexpr (NPH >= 14) {
                const W dr = lfma(cz, sz, lfma(cy, sy, lfma(cx, sx, lmul(p[13 * L], p[12 * L]))));
                W al;
                if constexpr (HALF) al = alpha;
                else al = W{alpha, alpha};
                n = lfma(al, dr, n);
            }
            o[4 * L] = n;
        }
    }
}

// Block shape of k_zws: one line per warp, NPH inverse and NOUT forward ones.
template <typename T, int N, int NPH> struct ZWs {
    using Z = ZRCfg<T, N>;
    static constexpr int NOUT = z_nout<NPH>(), NT = (NPH + NOUT) * 32;
    // blocks per SM the registers are sized for
    static constexpr int MINB = N == 512 ? 1 : N == 256 ? (NPH == 9 ? 2 : 1) : (NPH <= 12 ? 2 : 1);
    __host__ __device__ static constexpr int smem_bytes(int nraw, int ncp) {
        return (Z::ROWS * 32 + (NPH + NOUT) * Z::SCR + nraw * 2 * ncp) * (int)sizeof(V2<T>) + 16 + ncp * (int)sizeof(T);
    }
};

// The fused z stage in FP64, same arguments and contract as k_zpipe (STAGED =
// false: the staging does not fit, the inverse warps read the raw lines from
// global memory).  Per line pair, between two block barriers, the inverse warps pack and transform the
// quantities of pair p while the forward warps transform and store the
// products of the pair before (held in their own lines); then the whole block
// forms the products of p into the forward warps' lines.  The raw lines of the
// next pair are requested as soon as every inverse warp has packed (named
// barrier 1).
//   What bounds it (ncu, 512-point lines): shared-memory wavefronts 65%, the
// FP64 pipe 42%, with one block of 13 or 17 warps per SM.  Reading each raw
// mode once (the mirrored half by shuffle), transforming the products in the
// reversed flow graph and storing them from registers took 512^3 from 5.53 to
// 5.10 ms (two scalars) and 4.59 to 4.24 ms (one), 192^3 from 0.375 to 0.330.
template <typename T, int N, int NPH, int NRAW, bool DIAG = false, bool MB = false, bool STAGED = true>
__global__ void __launch_bounds__(ZWs<T, N, NPH>::NT, ZWs<T, N, NPH>::MINB)
k_zws(const __grid_constant__ FieldSet<T> f, const __grid_constant__ ZRecipeSet zr, long long npairs, int ncp, int nkz,
      T scale, T alpha, double dkz, const V2<T> *__restrict__ tw, unsigned *__restrict__ err,
      double *__restrict__ diag, long long mpairs, long long ms) {
    using V = V2<T>;
    using Z = ZRCfg<T, N>;
    using C = ZWs<T, N, NPH>;
    constexpr int E = Z::E, SCR = Z::SCR, ST = zl_stride<T, N>();
    constexpr unsigned NINV = NPH * 32;   // threads of the inverse warps (named barrier 1)
    constexpr bool FIXED = N == 512 && NPH >= 12;
    double acc[DIAG ? ZR_VORT_SUMS : 1] = {};
    const int rawf = 2 * ncp;
    const unsigned raw_bytes = (unsigned)(rawf * sizeof(V));
    extern __shared__ __align__(16) unsigned char smem_raw[];
    V *tws = reinterpret_cast<V *>(smem_raw);
    V *lines = tws + Z::ROWS * 32;   // NPH + NOUT lines, one per warp
    V *raw = lines + (NPH + C::NOUT) * SCR;
    uint64_t *bar = reinterpret_cast<uint64_t *>(raw + (STAGED ? NRAW * rawf : 0));
    T *tkz = reinterpret_cast<T *>(bar + 2);   // kz wavenumbers of the kept modes (ncp entries)
    __shared__ int stop;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    long long pair = blockIdx.x;
    if (pair >= npairs) return;   // uniform for the block
    for (int i = threadIdx.x; i < Z::ROWS * 32; i += C::NT) tws[i] = tw[Z::tw_index(i)];
    for (int k = threadIdx.x; k < ncp; k += C::NT) tkz[k] = (T)wavenum(k, N, dkz);
    if (threadIdx.x == 0) {
        stop = 0;
        mbar_init(bar, 1);
        mbar_fence_init();
    }
    __syncthreads();
    pdl_wait();
    const WaitCtl wc(err);
    auto issue = [&](long long p, bool withhold = false) {
        mbar_arrive_expect_tx(bar, NRAW * raw_bytes);
        if (!withhold)
            for (int q = 0; q < NRAW; ++q)
                bulk_g2s(raw + q * rawf, f.p[q] + pair_offset<MB>(p, mpairs, ms, rawf), raw_bytes, bar);
    };
    if (STAGED && threadIdx.x == 0) issue(pair, wc.withhold);
    unsigned parity = 0;
    const bool inv = warp < NPH;
    const ZRecipe rc = zr.q[inv ? warp : 0];
    V *scr = lines + warp * SCR;
    const T ls = zr_line_scale<T, NPH>(warp, scale);
    const V lsc = V{ls, ls};
    long long prev = -1;
    for (;;) {
        if (inv) {
            if (pair < npairs) {
                V x[E];
                bool ok = true;
                if constexpr (STAGED) {
                    ok = mbar_wait_bounded(bar, parity, wc.limit);
                    zl_pack<T, N, FIXED>(lane, x, rc, raw + rc.r[0] * rawf, raw + rc.r[1] * rawf, ncp, nkz, tkz);
                } else {
                    const long long off = pair_offset<MB>(pair, mpairs, ms, rawf);
                    zl_pack<T, N>(lane, x, rc, f.p[rc.r[0]] + off, f.p[rc.r[1] >= 0 ? rc.r[1] : 0] + off, ncp, nkz, tkz);
                }
                if (STAGED && bar_named_or(1, NINV, !ok)) {   // every inverse warp has packed, or one gave up
                    if (threadIdx.x == 0) {
                        stop = 1;
                        mbar_wait_bounded(bar, parity, wc.limit);   // let an overdue copy land before leaving
                    }
                } else {
                    parity ^= 1u;
                    if (STAGED && threadIdx.x == 0 && pair + gridDim.x < npairs) {
                        fence_proxy_async_smem();
                        issue(pair + gridDim.x);
                    }
                    zr_fft<T, N, +1>(lane, x, scr, tws);   // ends its scratch reads with __syncwarp
                    V *d = scr + zl_base<T, N>(lane);
#pragma unroll
                    for (int q = 0; q < E; ++q) d[q * ST] = lmul(x[q], lsc);
                }
            }
        } else if (prev >= 0) {   // z R2C of product warp - NPH of the previous pair
            V x[E];
            const V *d = scr + zl_base<T, N>(lane);
#pragma unroll
            for (int q = 0; q < E; ++q) x[q] = d[q * ST];
            __syncwarp();
            zr_fft_rev<T, N, -1>(lane, x, scr, tws);
            zl_unpack<T, N>(lane, x, f.p[warp - NPH] + pair_offset<MB>(prev, mpairs, ms, rawf), ncp);
        }
        __syncthreads();   // quantities of `pair` in the inverse warps' lines; the forward lines are free
        if (STAGED && stop) {
            if (threadIdx.x == 0) atomicOr(err, 1u);
            return;
        }
        if (pair >= npairs) break;
        zr_products<T, N, NPH, C::NT, DIAG>(lines, lines + NPH * SCR, alpha, scale, acc);
        __syncthreads();   // products of `pair` in the forward warps' lines
        prev = pair;
        pair += gridDim.x;
    }
    if constexpr (DIAG) {   // warp shuffles, then the block's warps in order
        constexpr int NW = NPH + C::NOUT;
        __shared__ double red[ZR_VORT_SUMS][NW];
#pragma unroll
        for (int q = 0; q < ZR_VORT_SUMS; ++q) {
            double v = acc[q];
            for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
            if (lane == 0) red[q][warp] = v;
        }
        __syncthreads();
        if (threadIdx.x < ZR_VORT_SUMS) {
            double v = 0.0;
            for (int w = 0; w < NW; ++w) v += red[threadIdx.x][w];
            diag[blockIdx.x * ZR_VORT_SUMS + threadIdx.x] = v;
        }
    }
}

}  // namespace gnss
