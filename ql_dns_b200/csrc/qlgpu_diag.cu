// Diagnostics of a state without stepping (the initial record, main.cpp:98-103,
// and the records of driven runs): Calc_Energy_AM_Diss (MHD_BQlin.cpp:337-488) of
// the fluctuations and the mean fields, one launch.
//
// The read of the state bounds it: one warp per mode, lanes along kz, over a
// cluster of 8 CTAs whose partial sums meet in the first CTA's shared memory, so
// there is neither scratch memory nor a second launch.  Sums run in a fixed order.
#include <cooperative_groups.h>

#include "qlgpu_host.h"
#include "qlgpu_kernel.cuh"

namespace qlgpu {

namespace {

constexpr int DIAG_CTAS = 8, DIAG_WARPS = 16;

__global__ void __cluster_dims__(DIAG_CTAS, 1, 1) __launch_bounds__(32 * DIAG_WARPS)
diag_kernel(const cplx* lin, const cplx* mf, const double* kx0, const double* ky, const int* kyi, DevParams P, double t,
            double* out) {
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    __shared__ double red[DIAG_WARPS][6];
    __shared__ double cta[6];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nz = P.nz, H = (nz - 1) / 2;
    double acc[6] = {0, 0, 0, 0, 0, 0};
    for (int m = blockIdx.x * DIAG_WARPS + warp; m < P.nxy; m += DIAG_CTAS * DIAG_WARPS) {
        const double b = ky[m], a = kx_at(kx0[m], P.q, t, b);
        const double ab = __dmul_rn(a, b), mult = b == 0.0 ? 1.0 : 2.0;
        const bool k0 = kyi[m] == 0;
        const cplx* u = lin + (size_t)m * 4 * nz;
        for (int s = lane; s < nz; s += 32) {
            const double c = kzval(s <= H ? s : s - nz, P.kzL);
            const bool z0 = k0 && s == 0;
            const double lap2 = lap2val(b, kz2val(c), z0);
            const double il2 = ilap2val(lap2, z0);
            const double lapF = __dadd_rn(-__dmul_rn(a, a), lap2);
            const double l2 = __dmul_rn(lapF, il2);
#pragma unroll
            for (int side = 0; side < 2; ++side) {
                const cplx p = ldc(u + 2 * side * nz + s), q = ldc(u + (2 * side + 1) * nz + s);
                const double e = l2 * (p.x * p.x + p.y * p.y) - il2 * (q.x * q.x + q.y * q.y);
                const cplx y = cscale(cadd(cscale(p, ab), imul(q, c)), il2);  // (MHD_BQlin.cpp:388-392)
                acc[side] += mult * e;
                acc[2 + side] += mult * (p.x * y.x + p.y * y.y);
                acc[4 + side] += mult * (side ? P.eta : P.nu) * (-lapF * e);
            }
        }
    }
#pragma unroll
    for (int q = 0; q < 6; ++q) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc[q] += __shfl_xor_sync(0xffffffffu, acc[q], o);
        if (lane == 0) red[warp][q] = acc[q];
    }
    __syncthreads();
    if (tid < 6) {
        double s = 0.0;
        for (int w = 0; w < DIAG_WARPS; ++w) s += red[w][tid];
        cta[tid] = s;
    }
    cl.sync();
    if (blockIdx.x == 0 && warp == 0) {
        double ds[6], v[6] = {0, 0, 0, 0, 0, 0};  // v: eMB, aMB, dMB, eMU, aMU, dMU
#pragma unroll
        for (int q = 0; q < 6; ++q) {
            ds[q] = 0.0;
            for (int r = 0; r < DIAG_CTAS; ++r) ds[q] += cl.map_shared_rank(cta, r)[q];
        }
        for (int s = lane; s < nz; s += 32) {
            const double kz2 = kz2val(kzval(s <= H ? s : s - nz, P.kzL));
            mf_sums(mf, mf + nz, s, kz2, v);
            if (P.nmf == 4) mf_sums(mf + 2 * nz, mf + 3 * nz, s, kz2, v + 3);
        }
#pragma unroll
        for (int q = 0; q < 6; ++q)
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
        if (lane == 0) put_record(P, ds, v, t, out);
    }
    cl.sync();  // the other CTAs' sums are read before they leave
}

}  // namespace

void launch_diag(const cplx* lin, const cplx* mf, const double* kx0, const double* ky, const int* kyi,
                 const DevParams& P, double t, double* out, cudaStream_t st) {
    diag_kernel<<<DIAG_CTAS, 32 * DIAG_WARPS, 0, st>>>(lin, mf, kx0, ky, kyi, P, t, out);
}

}  // namespace qlgpu
