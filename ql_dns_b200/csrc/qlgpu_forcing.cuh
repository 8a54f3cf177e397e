// qlgpu_forcing.cuh -- driving noise and the CFL time step of the QL models
// (sm_100a).
//
// noise_kernel: Model::DrivingNoise after a step of a single handle, one
// thread per (mode, kz) and the four fields (noise_value of qlgpu_noise.cuh).
// Modes that the step's remap zeroed (kx0 changed) are skipped: the reference
// adds their noise before the remap zeroes them (main.cpp:111-123).
//
// mf_absmax2_kernel: max over the NZ grid of |profile|^2 of each mean field, the
// real-space maxima Calculate_CFL reads (MHD_BQlin.cpp:540-552,
// MHD_FullQlin.cpp:769-780), by a direct sum over the stored kz.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "qlgpu_fft.cuh"
#include "qlgpu_noise.cuh"

namespace qlgpu {

struct NoiseArgs {
    cplx* lin;               // [nxy][4][nz]
    const double* kx0_prev;  // kx0 at the start of the step
    const double* kx0_now;   // after the step's remap
    const double* ky;
    const int* kxi;
    const int* kyi;
    int nxy, nz;
    double q, t, kzL;
    unsigned long long step;
    NoiseSpec ns;
};

__global__ void noise_kernel(NoiseArgs a) {
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= a.nxy * a.nz) return;
    const int i = idx / a.nz, k = idx % a.nz;
    const double kx0 = a.kx0_prev[i];
    if (a.kx0_now[i] != kx0) return;  // remapped: zeroed after its noise in the reference
    const double ky = a.ky[i];
    const int kxi = a.kxi[i], kyi = a.kyi[i];
#pragma unroll
    for (int v = 0; v < 4; ++v) {
        cplx n;
        if (!noise_value(a.ns, a.step, i, k, v, a.nz, kx0, ky, kxi, kyi, a.q, a.t, a.kzL, &n)) continue;
        cplx* p = a.lin + ((size_t)i * 4 + v) * a.nz + k;
        cplx u = *p;
        u.x = __dadd_rn(u.x, n.x);
        u.y = __dadd_rn(u.y, n.y);
        *p = u;
    }
}

// out[m] = max_z |sum_s fac mf[m][s] e^{+2 pi i kz_s z / NZ}|^2, one CTA per mean field.
// A chain of nz terms per z bounds it: MF_LANES lanes share a z, and the phase factors
// come from one table of the NZ-th roots of unity in shared memory (a sincospi per term
// and one thread per z took 21-31 us at NZ = 64, this 4 us).
constexpr int MF_THREADS = 512, MF_LANES = 8;

__global__ void __launch_bounds__(MF_THREADS) mf_absmax2_kernel(const cplx* mf, int nz, int NZ, double fac,
                                                                double* out) {
    __shared__ cplx w[256], f[2 * (256 / 3) + 1];
    __shared__ double red[MF_THREADS / 32];
    const int m = blockIdx.x, tid = threadIdx.x, H = (nz - 1) / 2;
    for (int i = tid; i < NZ; i += MF_THREADS) {
        double sn, cs;
        sincospi(2.0 * (double)i / (double)NZ, &sn, &cs);
        w[i] = mk(cs, sn);
    }
    for (int s = tid; s < nz; s += MF_THREADS) f[s] = mf[(size_t)m * nz + s];
    __syncthreads();
    const int part = tid % MF_LANES;
    double mx = 0.0;
    for (int z0 = 0; z0 < NZ; z0 += MF_THREADS / MF_LANES) {
        const int z = z0 + tid / MF_LANES;  // beyond NZ: a repeat of z mod NZ
        double re = 0.0, im = 0.0;
        for (int s = part; s < nz; s += MF_LANES) {
            const int kzi = s <= H ? s : s - nz;
            const cplx e = w[(kzi * z) & (NZ - 1)], v = f[s];
            re += fac * (v.x * e.x - v.y * e.y);
            im += fac * (v.x * e.y + v.y * e.x);
        }
#pragma unroll
        for (int o = MF_LANES / 2; o > 0; o >>= 1) {
            re += __shfl_xor_sync(0xffffffffu, re, o);
            im += __shfl_xor_sync(0xffffffffu, im, o);
        }
        mx = fmax(mx, re * re + im * im);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (tid % 32 == 0) red[tid / 32] = mx;
    __syncthreads();
    if (tid < 32) {
        mx = tid < MF_THREADS / 32 ? red[tid] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        if (tid == 0) out[m] = mx;
    }
}

}  // namespace qlgpu
