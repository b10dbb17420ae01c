// In-register butterflies of radix 2, 4 and 8 shared by the FFT passes.
#pragma once

#include "common.cuh"

namespace ffcm {

// Small DFTs: forward uses exp(-2 pi i q s / R), inverse the conjugate.
template <typename T, int R>
struct SmallDft;

template <typename T>
struct SmallDft<T, 2> {
    __device__ __forceinline__ static void run(cplx<T>* v, bool) {
        cplx<T> a = v[0], b = v[1];
        v[0] = cadd(a, b);
        v[1] = csub(a, b);
    }
};

template <typename T>
__device__ __forceinline__ void dft4(cplx<T>& a0, cplx<T>& a1, cplx<T>& a2, cplx<T>& a3, bool inv) {
    cplx<T> s02 = cadd(a0, a2), d02 = csub(a0, a2);
    cplx<T> s13 = cadd(a1, a3), d13 = csub(a1, a3);
    cplx<T> r = inv ? mul_pi(d13) : mul_mi(d13);
    a0 = cadd(s02, s13);
    a2 = csub(s02, s13);
    a1 = cadd(d02, r);
    a3 = csub(d02, r);
}

template <typename T>
struct SmallDft<T, 4> {
    __device__ __forceinline__ static void run(cplx<T>* v, bool inv) {
        dft4(v[0], v[1], v[2], v[3], inv);
    }
};

template <typename T>
struct SmallDft<T, 8> {
    __device__ __forceinline__ static void run(cplx<T>* v, bool inv) {
        cplx<T> e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6];
        cplx<T> o0 = v[1], o1 = v[3], o2 = v[5], o3 = v[7];
        dft4(e0, e1, e2, e3, inv);
        dft4(o0, o1, o2, o3, inv);
        const T c = T(0.70710678118654752440084436210484903928);
        // W8^1, W8^2, W8^3 (forward: exp(-i pi k/4))
        cplx<T> t1 = inv ? cplx<T>{c * (o1.x - o1.y), c * (o1.x + o1.y)}
                         : cplx<T>{c * (o1.x + o1.y), c * (o1.y - o1.x)};
        cplx<T> t2 = inv ? mul_pi(o2) : mul_mi(o2);
        cplx<T> t3 = inv ? cplx<T>{-c * (o3.x + o3.y), c * (o3.x - o3.y)}
                         : cplx<T>{c * (o3.y - o3.x), -c * (o3.x + o3.y)};
        v[0] = cadd(e0, o0); v[4] = csub(e0, o0);
        v[1] = cadd(e1, t1); v[5] = csub(e1, t1);
        v[2] = cadd(e2, t2); v[6] = csub(e2, t2);
        v[3] = cadd(e3, t3); v[7] = csub(e3, t3);
    }
};

}  // namespace ffcm
