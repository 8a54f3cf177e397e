// qlgpu_stage.cuh -- what the kernels of the quasi-linear shearing-box step share
// (sm_100a): loads, wavenumbers, linear operators and the RK update.
//
// The fused RK3 stage (stage_body of qlgpu_wide.cuh, the chunks of qlgpu_ens.cuh)
// is one stage of RK3CN_Elin::Step (QL_DNS/Integrators/
// RK3CN_Elin.cpp:86-177) or RK3CN::Step (QL_DNS/Integrators/RK3CN.cpp:86-180)
// for every (kx,ky) mode, fused with the model right-hand side
// (MHD_BQlin::rhs, QL_DNS/Models/MHD_BQlin.cpp:117-284; MHD_FullQlin::rhs,
// QL_DNS/Models/MHD_FullQlin.cpp:171-427), the diagonal diffusion factor, the
// EMF / stress sum over modes that replaces the MPI_Allreduce
// (QL_DNS/Auxiliary/MPIdata.cpp:148-157), the mean-field update, and on the
// last stage the shearing-wave remap (MHD_BQlin.cpp:314-331) and the
// energy / stress / dissipation diagnostics (MHD_BQlin.cpp:337-488).
//
// Everything is FP64.
#pragma once
#include "qlgpu_debug.cuh"
#include "qlgpu_xform.cuh"
#include "qlgpu_types.h"

namespace qlgpu {

// ---------------------------------------------------------------------------
// Small helpers
// ---------------------------------------------------------------------------
// State loads (fields, previous right-hand sides) go through L2 (ld.global.cg):
// the persistent batch kernel rewrites these buffers while it runs, so the
// non-coherent read-only path must not cache them.
__device__ __forceinline__ cplx ldc(const cplx* p) {
    double2 v = __ldcg(reinterpret_cast<const double2*>(p));
    return mk(v.x, v.y);
}
__device__ __forceinline__ cplx ldc_cg(const cplx* p) {
    double2 v = __ldcg(reinterpret_cast<const double2*>(p));
    return mk(v.x, v.y);
}
__device__ __forceinline__ void stc(cplx* p, cplx v) {
    *reinterpret_cast<double2*>(p) = make_double2(v.x, v.y);
}
// i*s*a for real s
__device__ __forceinline__ cplx imul(cplx a, double s) { return mk(-a.y * s, a.x * s); }

// Asynchronous prefetch of a contiguous range into L2 (one bulk request, no
// registers or shared memory held; bytes a multiple of 16, address 16-aligned).
__device__ __forceinline__ void l2_prefetch(const void* p, unsigned bytes) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;\n" ::"l"(p), "r"(bytes) : "memory");
}

__device__ __forceinline__ unsigned long long gtimer() {
    unsigned long long v;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(v)::"memory");
    return v;
}

// kx(t) = kx0 + (q t) ky, evaluated with the reference's rounding order
// (MHD_BQlin.cpp:498: K->kx[i] + q_*t*kyctmp_)
__device__ __forceinline__ double kx_at(double kx0, double q, double t, double ky) {
    return __dadd_rn(kx0, __dmul_rn(__dmul_rn(q, t), ky));
}

// kz integer -> double wavenumber (Kdata.cpp:76-78: i*kzLfac)
__device__ __forceinline__ double kzval(int kzi, double kzL) { return __dmul_rn((double)kzi, kzL); }
// kz2 = (kz*kz).real() = -(c*c)  (Kdata.cpp:80)
__device__ __forceinline__ double kz2val(double c) { return -__dmul_rn(c, c); }
// lap2 = -ky*ky + kz2 with the ky=kz=0 fix (Kdata.cpp:105-113)
__device__ __forceinline__ double lap2val(double ky, double kz2, bool ky0kz0) {
    return ky0kz0 ? 0.0 : __dadd_rn(-__dmul_rn(ky, ky), kz2);
}
__device__ __forceinline__ double ilap2val(double lap2, bool ky0kz0) {
    return ky0kz0 ? 1.0 : __drcp_rn(lap2);
}

// Laplacian factor of the fluctuation linear operator at the stage end
// (MHD_BQlin.cpp:248-249: (-kx^2 - ky^2) + kz2; MHD_FullQlin.cpp:371-372:
// -|(-kx^2 - ky^2) + kz2|^(order/2)).  kxe = kx(t_s) + q dt_lin ky.
template <int MODEL>
__device__ __forceinline__ double lap_end(const DevParams& P, double kxe, double ky, double kz2) {
    double lap = __dadd_rn(__dsub_rn(-__dmul_rn(kxe, kxe), __dmul_rn(ky, ky)), kz2);
    if (MODEL == MODEL_BQLIN) return lap;
    double a = fabs(lap), r = 1.0;
    for (int i = 0; i < P.visc_half; ++i) r = __dmul_rn(r, a);
    return -r;
}
// linearOPs_Init form (MHD_BQlin.cpp:291, MHD_FullQlin.cpp:435): -kx^2 + lap2
template <int MODEL>
__device__ __forceinline__ double lap_init(const DevParams& P, double kx, double lap2) {
    double lapF = __dadd_rn(-__dmul_rn(kx, kx), lap2);
    if (MODEL == MODEL_BQLIN) return lapF;
    double a = fabs(lapF), r = 1.0;
    for (int i = 0; i < P.visc_half; ++i) r = __dmul_rn(r, a);
    return -r;
}
// L for field f (0 u, 1 zeta, 2 b, 3 eta) from the laplacian factor:
// BQlin L_u = nu lap, L_b = (eta/nu) L_u (MHD_BQlin.cpp:249-252);
// FullQlin L_u = nu lap, L_b = eta lap (MHD_FullQlin.cpp:373-376).
template <int MODEL>
__device__ __forceinline__ double linop_f(const DevParams& P, double lap, int f) {
    const double Lu = __dmul_rn(P.nu, lap);
    if (f < 2) return Lu;
    return MODEL == MODEL_BQLIN ? __dmul_rn(P.etanu, Lu) : __dmul_rn(P.eta, lap);
}

// RK3CN update of one coefficient: n1 d F + n2 d Fp + (1 + linC Lold) d u,
// d = 1/(1 - linC L) (RK3CN.cpp:105-107).
__device__ __forceinline__ cplx rk_update(const StageConst& S, double L, double Lold, cplx F, cplx Fp, cplx u,
                                          bool has_prev) {
    double d = __drcp_rn(__dsub_rn(1.0, __dmul_rn(S.linC, L)));
    double c1 = __dmul_rn(S.n1, d);
    double c3 = __dmul_rn(__dadd_rn(1.0, __dmul_rn(S.linC, Lold)), d);
    cplx r = cscale(F, c1);
    if (has_prev) r = cadd(r, cscale(Fp, __dmul_rn(S.n2, d)));
    return cadd(r, cscale(u, c3));
}

// CN: where the previous stage's operator was evaluated (RK3CN.cpp:119-122)
struct CnOld {
    double t_old, dtlin_old;
    int old_init;
};

}  // namespace qlgpu
