// pk.cuh -- complex arithmetic on 16-byte elements.
//
// A complex element of the direct kernels is 16 bytes wide: one FP64 complex
// value (P = double), or two FP32 complex values of neighbouring columns
// (P = F2, the packed pairs of sm_100: add, sub, mul and fma on two floats
// per instruction).  Real and imaginary parts of a pair lie in a register
// pair each, so multiplications by i are register renamings, and one source
// serves both precisions.
#pragma once
#include "fft.cuh"

namespace gnss {

struct F2 { unsigned long long b; };
__device__ __forceinline__ F2 f2(float lo, float hi) {
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.b) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void f2_get(F2 a, float &lo, float &hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(a.b));
}
__device__ __forceinline__ F2 operator+(F2 a, F2 b) {
    F2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.b) : "l"(a.b), "l"(b.b));
    return r;
}
__device__ __forceinline__ F2 operator-(F2 a, F2 b) {
    F2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.b) : "l"(a.b), "l"(b.b));
    return r;
}
__device__ __forceinline__ F2 operator*(F2 a, F2 b) {
    F2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.b) : "l"(a.b), "l"(b.b));
    return r;
}
__device__ __forceinline__ F2 pfma(F2 a, F2 b, F2 c) {
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.b) : "l"(a.b), "l"(b.b), "l"(c.b));
    return r;
}
__device__ __forceinline__ double pfma(double a, double b, double c) { return fma(a, b, c); }

// T: the scalar type; P: the 16-byte element's component
template <typename T> struct PkOf;
template <> struct PkOf<double> {
    using P = double;
    static constexpr int W = 1;   // columns per element
    static __device__ __forceinline__ P dup(double v) { return v; }
};
template <> struct PkOf<float> {
    using P = F2;
    static constexpr int W = 2;
    static __device__ __forceinline__ P dup(double v) { return f2((float)v, (float)v); }
};
template <typename P> struct ScalarOf;
template <> struct ScalarOf<double> { using T = double; };
template <> struct ScalarOf<F2> { using T = float; };
template <typename P> __device__ __forceinline__ P pconst(double v) { return PkOf<typename ScalarOf<P>::T>::dup(v); }
template <typename P> __device__ __forceinline__ P pneg(P a) { return a * pconst<P>(-1.0); }
template <> __device__ __forceinline__ double pneg<double>(double a) { return -a; }

template <typename P> struct CP { P x, y; };
template <typename P> __device__ __forceinline__ CP<P> operator+(CP<P> a, CP<P> b) { return {a.x + b.x, a.y + b.y}; }
template <typename P> __device__ __forceinline__ CP<P> operator-(CP<P> a, CP<P> b) { return {a.x - b.x, a.y - b.y}; }
// a + S i b, a - S i b
template <int S, typename P> __device__ __forceinline__ CP<P> add_i(CP<P> a, CP<P> b) {
    return S > 0 ? CP<P>{a.x - b.y, a.y + b.x} : CP<P>{a.x + b.y, a.y - b.x};
}
template <int S, typename P> __device__ __forceinline__ CP<P> sub_i(CP<P> a, CP<P> b) { return add_i<-S>(a, b); }
// a * (wr + i wi)
template <typename P> __device__ __forceinline__ CP<P> cmulp(CP<P> a, P wr, P wi) {
    return {pfma(a.x, wr, a.y * pneg(wi)), pfma(a.x, wi, a.y * wr)};
}
template <> __device__ __forceinline__ CP<double> cmulp<double>(CP<double> a, double wr, double wi) {
    return {a.x * wr - a.y * wi, a.x * wi + a.y * wr};
}

// ------------------------------------------------------------ small DFTs, natural order
// Constant factors enter as fused multiply-adds: the packed instructions are not contracted by the compiler.
template <int S, typename P> __device__ __forceinline__ void pdft4(CP<P> &a0, CP<P> &a1, CP<P> &a2, CP<P> &a3) {
    const CP<P> s02 = a0 + a2, d02 = a0 - a2, s13 = a1 + a3, d13 = a1 - a3;
    a0 = s02 + s13;
    a2 = s02 - s13;
    a1 = add_i<S>(d02, d13);
    a3 = sub_i<S>(d02, d13);
}
template <int R, int S> struct PDft;
template <int S> struct PDft<2, S> {
    template <typename P> static __device__ __forceinline__ void run(CP<P> *v) {
        const CP<P> t = v[0];
        v[0] = t + v[1];
        v[1] = t - v[1];
    }
};
template <int S> struct PDft<3, S> {
    template <typename P> static __device__ __forceinline__ void run(CP<P> *v) {
        const P c3 = pconst<P>(-0.5), s3 = pconst<P>(S * 0.86602540378443864676372317075294);
        const P n3 = pconst<P>(-S * 0.86602540378443864676372317075294);
        const CP<P> s = v[1] + v[2], d = v[1] - v[2];
        const CP<P> m{pfma(c3, s.x, v[0].x), pfma(c3, s.y, v[0].y)};
        v[0] = v[0] + s;
        v[1] = {pfma(n3, d.y, m.x), pfma(s3, d.x, m.y)};
        v[2] = {pfma(s3, d.y, m.x), pfma(n3, d.x, m.y)};
    }
};
template <int S> struct PDft<4, S> {
    template <typename P> static __device__ __forceinline__ void run(CP<P> *v) { pdft4<S>(v[0], v[1], v[2], v[3]); }
};
template <int S> struct PDft<6, S> {   // n = 3 n1 + 2 n2, k = 3 k1 + 4 k2 (mod 6): no twiddles
    template <typename P> static __device__ __forceinline__ void run(CP<P> *v) {
        CP<P> a[3] = {v[0], v[2], v[4]}, b[3] = {v[3], v[5], v[1]};
        PDft<3, S>::run(a);
        PDft<3, S>::run(b);
#pragma unroll
        for (int k2 = 0; k2 < 3; ++k2) {
            v[(4 * k2) % 6] = a[k2] + b[k2];
            v[(3 + 4 * k2) % 6] = a[k2] - b[k2];
        }
    }
};
template <int S> struct PDft<8, S> {
    template <typename P> static __device__ __forceinline__ void run(CP<P> *v) {
        const P h = pconst<P>(0.70710678118654752440084436210485), mh = pconst<P>(-0.70710678118654752440084436210485);
        pdft4<S>(v[0], v[2], v[4], v[6]);
        pdft4<S>(v[1], v[3], v[5], v[7]);
        // odd outputs o1, o2, o3 in v[3], v[5], v[7] times W_8^1, W_8^2, W_8^3
        const CP<P> e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6], o0 = v[1], o2 = v[5];
        const CP<P> p1 = add_i<S>(v[3], v[3]);    // o1 (1 + S i)
        const CP<P> p3 = sub_i<S>(v[7], v[7]);    // o3 (1 - S i); o3 (-1 + S i) is its negative
        v[0] = e0 + o0;
        v[4] = e0 - o0;
        v[2] = add_i<S>(e2, o2);
        v[6] = sub_i<S>(e2, o2);
        v[1] = {pfma(h, p1.x, e1.x), pfma(h, p1.y, e1.y)};
        v[5] = {pfma(mh, p1.x, e1.x), pfma(mh, p1.y, e1.y)};
        v[3] = {pfma(mh, p3.x, e3.x), pfma(mh, p3.y, e3.y)};
        v[7] = {pfma(h, p3.x, e3.x), pfma(h, p3.y, e3.y)};
    }
};

}  // namespace gnss
