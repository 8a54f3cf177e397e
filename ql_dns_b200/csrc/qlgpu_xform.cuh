// qlgpu_xform.cuh -- the z transforms with 8 points per thread (sm_100a).
//
// A group of T = NZ/8 threads (2 ... 32) holds one length-NZ column; thread t
// register r holds index t + T r in spectral AND in real space.  One routine
// (xform) computes the backward (FFTW_BACKWARD, fftwPlans.cpp:48-51) transform;
// the forward one is conj(xform(conj(x))), and the conjugations are folded into
// the pointwise code around it.  A transform is one register DFT-8, a twiddle,
// one shared-memory exchange and 8/T register DFT-T (T = 16 / 32: a radix-2 / 4
// step on the exchanged values and a DFT-8).
#pragma once
#include "qlgpu_fft.cuh"

namespace qlgpu {

// Asynchronous global -> shared copies (cp.async), 16 or 8 bytes each
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async8(void* smem, const void* gmem) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// Real-space / spectral register classes: index t + T r is in the dealiasing
// gap for every t (dead), stored for every t, or stored for some t.
template <class E>
__device__ __forceinline__ int sidx(int t, int r) {
    const int k = t + E::T * r;
    if (k <= E::H) return k;
    if (k >= E::NZ - E::H) return k - (E::NZ - E::nz);
    return -1;
}
template <class E>
__host__ __device__ constexpr bool rdead(int r) {
    return E::T * r > E::H && E::T * r + E::T - 1 < E::NZ - E::H;
}

// cos / sin (2 pi i / 16)
__device__ __forceinline__ constexpr double c16(int i) {
    return i == 0 ? 1.0 : i == 1 ? QLGPU_C1 : i == 2 ? QLGPU_RSQRT2 : i == 3 ? QLGPU_S1 : i == 4 ? 0.0
         : i == 5 ? -QLGPU_S1 : i == 6 ? -QLGPU_RSQRT2 : -QLGPU_C1;
}
__device__ __forceinline__ constexpr double s16(int i) {
    return i == 0 ? 0.0 : i == 1 ? QLGPU_S1 : i == 2 ? QLGPU_RSQRT2 : i == 3 ? QLGPU_C1 : i == 4 ? 1.0
         : i == 5 ? QLGPU_C1 : i == 6 ? QLGPU_RSQRT2 : QLGPU_S1;
}

// Exchange-buffer slot of (row q, column t) in group g's buffer (cplx units).  E::PAD: rows of
// T + 1, so every slot is the lane's base plus a constant (3 % of a stage); otherwise, and for
// groups of T < 8, whose padded rows would nearly double the buffer, rotated and permuted rows
// of T.  Either way the 8 lanes of a 128-byte access fall on different banks.
template <class E>
__device__ __forceinline__ int xslot(int g, int q, int t) {
    if constexpr (E::PAD) return (g * 8 + q) * (E::T + 1) + t;
    else return g * 8 * E::T + E::T * (q ^ (g & E::SWZ)) + ((t + q) & (E::T - 1));
}
// A warp's exchange buffer (cplx).
template <class E>
constexpr int XWARP = E::PAD ? 8 * (32 / E::T) * (E::T + 1) : 256;

// Backward DFT of one column: x[r] = X[t + T r] in, x[r] = y[t + T r] out,
// y[n] = sum_k X[k] exp(+2 pi i n k / NZ).  at(q, s) is the group's exchange slot of
// (row q < 8, column s < T), tw[q T + t] = exp(2 pi i q t / NZ).
// Warp-collective (every lane of the warp calls it together).
template <class E, class At>
__device__ __forceinline__ void xform_at(cplx (&x)[8], At&& at, const cplx* tw, int t) {
    constexpr int T = E::T;
    dft8<+1>(x);
#pragma unroll
    for (int q = 1; q < 8; ++q) x[q] = cmul(x[q], tw[q * T + t]);
#pragma unroll
    for (int q = 0; q < 8; ++q) at(q, t) = x[q];
    __syncwarp();
    if constexpr (T <= 8) {
        constexpr int J = 8 / T;
#pragma unroll
        for (int j = 0; j < J; ++j) {
            const int q = t + T * j;
            cplx v[T];
#pragma unroll
            for (int s = 0; s < T; ++s) v[s] = at(q, s);
            dft<T, +1>(v);
#pragma unroll
            for (int m = 0; m < T; ++m) x[j + J * m] = v[m];
        }
    } else if constexpr (T == 16) {
        // thread (q, h) = (t % 8, t / 8) takes the outputs of parity h of the 16-point
        // transforms over the columns of row q: a radix-2 step then a DFT-8.
        const int q = t & 7, h = t >> 3;
        const double sg = h ? -1.0 : 1.0;
#pragma unroll
        for (int s = 0; s < 8; ++s) {
            const cplx za = at(q, s);
            const cplx zb = at(q, s + 8);
            cplx w = mk(fma(sg, zb.x, za.x), fma(sg, zb.y, za.y));
            if (s != 0) w = cmul(w, mk(h ? c16(s) : 1.0, h ? s16(s) : 0.0));  // 3 % faster than the table
            x[s] = w;
        }
        dft8<+1>(x);
    } else {
        static_assert(T == 32, "8 points per thread, NZ <= 256");
        // thread (q, h) = (t % 8, t / 8) takes the outputs n = h + 4 m of the 32-point transforms
        // over the columns of row q: w_s = exp(2 pi i s h / 32) sum_j i^(j h) z[s + 8 j], then a DFT-8.
        const int q = t & 7, h = t >> 3;
        const double s1 = (h & 1) ? -1.0 : 1.0, s2 = (h & 2) ? -1.0 : 1.0;
#pragma unroll
        for (int s = 0; s < 8; ++s) {
            const cplx z0 = at(q, s), z1 = at(q, s + 8);
            const cplx z2 = at(q, s + 16), z3 = at(q, s + 24);
            const cplx a = mk(fma(s1, z2.x, z0.x), fma(s1, z2.y, z0.y));
            const cplx b = mk(fma(s1, z3.x, z1.x), fma(s1, z3.y, z1.y));
            const cplx ib = (h & 1) ? mk(-b.y, b.x) : b;  // i^h b up to the sign s2
            cplx w = mk(fma(s2, ib.x, a.x), fma(s2, ib.y, a.y));
            if (s != 0) w = cmul(w, tw[s * T + 8 * h]);  // exp(2 pi i 8 s h / 256)
            x[s] = w;
        }
        dft8<+1>(x);
    }
    __syncwarp();
}
// The same with the warp's exchange buffers xg, g = this thread's group in the warp.
template <class E>
__device__ __forceinline__ void xform(cplx (&x)[8], cplx* xg, const cplx* tw, int g, int t) {
    xform_at<E>(x, [&](int q, int s) -> cplx& { return xg[xslot<E>(g, q, s)]; }, tw, t);
}

}  // namespace qlgpu
