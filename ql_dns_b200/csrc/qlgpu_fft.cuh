// qlgpu_fft.cuh -- FP64 complex arithmetic and the register DFTs of the
// z-transforms (qlgpu_xform.cuh).
//
// Conventions follow FFTW as used by the reference (QL_DNS/Auxiliary/
// fftwPlans.cpp:48-51): backward = exp(+2 pi i jk/N), forward =
// exp(-2 pi i jk/N), both unnormalised.
#pragma once
#include <cuda_runtime.h>

namespace qlgpu {

struct __align__(16) cplx {
    double x, y;
};

__device__ __forceinline__ cplx mk(double a, double b) { cplx r; r.x = a; r.y = b; return r; }
__device__ __forceinline__ cplx cadd(cplx a, cplx b) { return mk(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ cplx csub(cplx a, cplx b) { return mk(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ cplx cmul(cplx a, cplx b) {
    return mk(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ cplx cscale(cplx a, double s) { return mk(a.x * s, a.y * s); }
// multiply by +i (DIR>0) or -i (DIR<0)
template <int DIR>
__device__ __forceinline__ cplx mul_i(cplx a) {
    return DIR > 0 ? mk(-a.y, a.x) : mk(a.y, -a.x);
}
__device__ __forceinline__ cplx conjc(cplx a) { return mk(a.x, -a.y); }

// ---------------------------------------------------------------------------
// In-register DFTs, natural order in and out.  DIR = +1 backward, -1 forward.
// ---------------------------------------------------------------------------
template <int DIR>
__device__ __forceinline__ void dft2(cplx& a, cplx& b) {
    cplx t = a;
    a = cadd(t, b);
    b = csub(t, b);
}

template <int DIR>
__device__ __forceinline__ void dft4(cplx& x0, cplx& x1, cplx& x2, cplx& x3) {
    cplx y0 = cadd(x0, x2), y1 = csub(x0, x2);
    cplx y2 = cadd(x1, x3), y3 = mul_i<DIR>(csub(x1, x3));
    x0 = cadd(y0, y2);
    x2 = csub(y0, y2);
    x1 = cadd(y1, y3);
    x3 = csub(y1, y3);
}

// (1 + DIR i)/sqrt(2) * a  and (-1 + DIR i)/sqrt(2) * a
#define QLGPU_RSQRT2 0.70710678118654752440
template <int DIR>
__device__ __forceinline__ cplx w8_1(cplx a) {
    // (a.x + i a.y)(1 + D i)/sqrt2 = (a.x - D a.y, a.y + D a.x)/sqrt2
    return DIR > 0 ? mk((a.x - a.y) * QLGPU_RSQRT2, (a.y + a.x) * QLGPU_RSQRT2)
                   : mk((a.x + a.y) * QLGPU_RSQRT2, (a.y - a.x) * QLGPU_RSQRT2);
}
template <int DIR>
__device__ __forceinline__ cplx w8_3(cplx a) {
    // (a.x + i a.y)(-1 + D i)/sqrt2 = (-a.x - D a.y, -a.y + D a.x)/sqrt2
    return DIR > 0 ? mk((-a.x - a.y) * QLGPU_RSQRT2, (a.x - a.y) * QLGPU_RSQRT2)
                   : mk((a.y - a.x) * QLGPU_RSQRT2, (-a.y - a.x) * QLGPU_RSQRT2);
}

template <int DIR>
__device__ __forceinline__ void dft8(cplx* x) {
    cplx e0 = x[0], e1 = x[2], e2 = x[4], e3 = x[6];
    cplx o0 = x[1], o1 = x[3], o2 = x[5], o3 = x[7];
    dft4<DIR>(e0, e1, e2, e3);
    dft4<DIR>(o0, o1, o2, o3);
    o1 = w8_1<DIR>(o1);
    o2 = mul_i<DIR>(o2);
    o3 = w8_3<DIR>(o3);
    x[0] = cadd(e0, o0); x[4] = csub(e0, o0);
    x[1] = cadd(e1, o1); x[5] = csub(e1, o1);
    x[2] = cadd(e2, o2); x[6] = csub(e2, o2);
    x[3] = cadd(e3, o3); x[7] = csub(e3, o3);
}

// cos/sin(2 pi k/16), k = 1
#define QLGPU_C1 0.92387953251128675613
#define QLGPU_S1 0.38268343236508977173
template <int M, int DIR>
__device__ __forceinline__ void dft(cplx* x) {
    if constexpr (M == 1) {
    } else if constexpr (M == 2) {
        dft2<DIR>(x[0], x[1]);
    } else if constexpr (M == 4) {
        dft4<DIR>(x[0], x[1], x[2], x[3]);
    } else {
        static_assert(M == 8, "register DFT size");
        dft8<DIR>(x);
    }
}

}  // namespace qlgpu
