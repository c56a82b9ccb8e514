// Register DFTs of 1 to 32 points, natural order in and out.
#pragma once
#include "cplx.cuh"
#include "plan_dev.h"
#include "roots.h"

namespace csipm {

// ---------------------------------------------------------------- butterflies
template <bool INV, typename C> __device__ __forceinline__ C rot_mi(C a) {   // a * (-i) forward, a * (+i) inverse
    return INV ? cmul_i(a) : cmul_mi(a);
}

template <int R, bool INV, typename T> struct Dft;

template <bool INV, typename T> struct Dft<1, INV, T> {
    __device__ __forceinline__ static void run(cplx_t<T>*) {}
};

template <bool INV, typename T> struct Dft<2, INV, T> {
    using C = cplx_t<T>;
    __device__ __forceinline__ static void run(C* a) {
        C t = a[0];
        a[0] = cadd(t, a[1]);
        a[1] = csub(t, a[1]);
    }
};

template <bool INV, typename T> struct Dft<4, INV, T> {
    using C = cplx_t<T>;
    __device__ __forceinline__ static void run(C* a) {
        C t0 = cadd(a[0], a[2]), t1 = csub(a[0], a[2]);
        C t2 = cadd(a[1], a[3]), t3 = rot_mi<INV>(csub(a[1], a[3]));
        a[0] = cadd(t0, t2);
        a[2] = csub(t0, t2);
        a[1] = cadd(t1, t3);
        a[3] = csub(t1, t3);
    }
};

template <bool INV, typename T> struct Dft<8, INV, T> {
    using C = cplx_t<T>;
    __device__ __forceinline__ static void run(C* a) {
        const T h = (T)0.7071067811865476;   // sqrt(2)/2
        C e[4] = {a[0], a[2], a[4], a[6]};
        C o[4] = {a[1], a[3], a[5], a[7]};
        Dft<4, INV, T>::run(e);
        Dft<4, INV, T>::run(o);
        // o[k] *= W8^k  (W8 = exp(-i*pi/4) forward)
        C o1, o2, o3;
        if (!INV) {
            o1 = mk((o[1].x + o[1].y) * h, (o[1].y - o[1].x) * h);
            o2 = cmul_mi(o[2]);
            o3 = mk((o[3].y - o[3].x) * h, -(o[3].x + o[3].y) * h);
        } else {
            o1 = mk((o[1].x - o[1].y) * h, (o[1].x + o[1].y) * h);
            o2 = cmul_i(o[2]);
            o3 = mk(-(o[3].x + o[3].y) * h, (o[3].x - o[3].y) * h);
        }
        a[0] = cadd(e[0], o[0]); a[4] = csub(e[0], o[0]);
        a[1] = cadd(e[1], o1);   a[5] = csub(e[1], o1);
        a[2] = cadd(e[2], o2);   a[6] = csub(e[2], o2);
        a[3] = cadd(e[3], o3);   a[7] = csub(e[3], o3);
    }
};

template <bool INV, typename T> struct Dft<3, INV, T> {
    using C = cplx_t<T>;
    __device__ __forceinline__ static void run(C* a) {
        const T s = (T)0.8660254037844386;   // sin(2*pi/3)
        C t1 = cadd(a[1], a[2]), t2 = csub(a[1], a[2]);
        C m = mk(a[0].x - (T)0.5 * t1.x, a[0].y - (T)0.5 * t1.y);
        a[0] = cadd(a[0], t1);
        // forward: y1 = m - i*s*t2, y2 = m + i*s*t2
        C st = mk(s * t2.x, s * t2.y);
        C ist = cmul_i(st);
        if (!INV) { a[1] = csub(m, ist); a[2] = cadd(m, ist); }
        else      { a[1] = cadd(m, ist); a[2] = csub(m, ist); }
    }
};

template <bool INV, typename T> struct Dft<5, INV, T> {
    using C = cplx_t<T>;
    __device__ __forceinline__ static void run(C* a) {
        const T c1 = (T)0.30901699437494745, c2 = (T)-0.8090169943749475;
        const T s1 = (T)0.9510565162951535, s2 = (T)0.5877852522924731;
        C t1 = cadd(a[1], a[4]), t2 = cadd(a[2], a[3]);
        C t3 = csub(a[1], a[4]), t4 = csub(a[2], a[3]);
        C b1 = mk(a[0].x + c1 * t1.x + c2 * t2.x, a[0].y + c1 * t1.y + c2 * t2.y);
        C b2 = mk(a[0].x + c2 * t1.x + c1 * t2.x, a[0].y + c2 * t1.y + c1 * t2.y);
        C e1 = mk(s1 * t3.x + s2 * t4.x, s1 * t3.y + s2 * t4.y);
        C e2 = mk(s2 * t3.x - s1 * t4.x, s2 * t3.y - s1 * t4.y);
        a[0] = cadd(a[0], cadd(t1, t2));
        C ie1 = cmul_i(e1), ie2 = cmul_i(e2);
        if (!INV) { a[1] = csub(b1, ie1); a[4] = cadd(b1, ie1); a[2] = csub(b2, ie2); a[3] = cadd(b2, ie2); }
        else      { a[1] = cadd(b1, ie1); a[4] = csub(b1, ie1); a[2] = cadd(b2, ie2); a[3] = csub(b2, ie2); }
    }
};

template <bool INV, typename T> struct Dft<7, INV, T> {
    using C = cplx_t<T>;
    __device__ __forceinline__ static void run(C* a) {
        const T c1 = (T)0.6234898018587335, c2 = (T)-0.2225209339563144, c3 = (T)-0.9009688679024191;
        const T s1 = (T)0.7818314824680298, s2 = (T)0.9749279121818236, s3 = (T)0.4338837391175581;
        C t1 = cadd(a[1], a[6]), t2 = cadd(a[2], a[5]), t3 = cadd(a[3], a[4]);
        C d1 = csub(a[1], a[6]), d2 = csub(a[2], a[5]), d3 = csub(a[3], a[4]);
        C x0 = a[0];
        C b1 = mk(x0.x + c1 * t1.x + c2 * t2.x + c3 * t3.x, x0.y + c1 * t1.y + c2 * t2.y + c3 * t3.y);
        C b2 = mk(x0.x + c2 * t1.x + c3 * t2.x + c1 * t3.x, x0.y + c2 * t1.y + c3 * t2.y + c1 * t3.y);
        C b3 = mk(x0.x + c3 * t1.x + c1 * t2.x + c2 * t3.x, x0.y + c3 * t1.y + c1 * t2.y + c2 * t3.y);
        C e1 = mk(s1 * d1.x + s2 * d2.x + s3 * d3.x, s1 * d1.y + s2 * d2.y + s3 * d3.y);
        C e2 = mk(s2 * d1.x - s3 * d2.x - s1 * d3.x, s2 * d1.y - s3 * d2.y - s1 * d3.y);
        C e3 = mk(s3 * d1.x - s1 * d2.x + s2 * d3.x, s3 * d1.y - s1 * d2.y + s2 * d3.y);
        a[0] = cadd(x0, cadd(t1, cadd(t2, t3)));
        C i1 = cmul_i(e1), i2 = cmul_i(e2), i3 = cmul_i(e3);
        if (!INV) {
            a[1] = csub(b1, i1); a[6] = cadd(b1, i1);
            a[2] = csub(b2, i2); a[5] = cadd(b2, i2);
            a[3] = csub(b3, i3); a[4] = cadd(b3, i3);
        } else {
            a[1] = cadd(b1, i1); a[6] = csub(b1, i1);
            a[2] = cadd(b2, i2); a[5] = csub(b2, i2);
            a[3] = cadd(b3, i3); a[4] = csub(b3, i3);
        }
    }
};

// Composite radix R = R1*R2 in registers: R2 DFTs of size R1 over
// a[n2 + R2*n1], twiddles W_R^{n2*k1} (compile-time constants), then R1 DFTs
// of size R2; output X[k1 + R1*k2].
template <int R1, int R2, bool INV, typename T> struct DftComp {
    using C = cplx_t<T>;
    static constexpr int R = R1 * R2;
    __device__ __forceinline__ static void run(C* a) {
        C y[R];
#pragma unroll
        for (int n2 = 0; n2 < R2; ++n2) {
            C t[R1];
#pragma unroll
            for (int n1 = 0; n1 < R1; ++n1) t[n1] = a[n2 + R2 * n1];
            Dft<R1, INV, T>::run(t);
#pragma unroll
            for (int k1 = 0; k1 < R1; ++k1) {
                const int m = (n2 * k1) % R;
                C v = t[k1];
                if (m != 0) {
                    const C w = mk((T)RootTab<R>::re(m), (T)RootTab<R>::im(m));
                    v = INV ? cmulc(v, w) : cmul(v, w);
                }
                y[k1 * R2 + n2] = v;
            }
        }
#pragma unroll
        for (int k1 = 0; k1 < R1; ++k1) {
            C t[R2];
#pragma unroll
            for (int n2 = 0; n2 < R2; ++n2) t[n2] = y[k1 * R2 + n2];
            Dft<R2, INV, T>::run(t);
#pragma unroll
            for (int k2 = 0; k2 < R2; ++k2) a[k1 + R1 * k2] = t[k2];
        }
    }
};

template <bool INV, typename T> struct Dft<6, INV, T> : DftComp<2, 3, INV, T> {};
template <bool INV, typename T> struct Dft<9, INV, T> : DftComp<3, 3, INV, T> {};
template <bool INV, typename T> struct Dft<10, INV, T> : DftComp<2, 5, INV, T> {};
template <bool INV, typename T> struct Dft<12, INV, T> : DftComp<4, 3, INV, T> {};
template <bool INV, typename T> struct Dft<15, INV, T> : DftComp<3, 5, INV, T> {};
template <bool INV, typename T> struct Dft<16, INV, T> : DftComp<4, 4, INV, T> {};
template <bool INV, typename T> struct Dft<20, INV, T> : DftComp<4, 5, INV, T> {};
template <bool INV, typename T> struct Dft<25, INV, T> : DftComp<5, 5, INV, T> {};
template <bool INV, typename T> struct Dft<32, INV, T> : DftComp<8, 4, INV, T> {};
template <bool INV, typename T> struct Dft<18, INV, T> : DftComp<2, 9, INV, T> {};
template <bool INV, typename T> struct Dft<24, INV, T> : DftComp<8, 3, INV, T> {};
template <bool INV, typename T> struct Dft<27, INV, T> : DftComp<3, 9, INV, T> {};
template <bool INV, typename T> struct Dft<30, INV, T> : DftComp<5, 6, INV, T> {};

}  // namespace csipm
