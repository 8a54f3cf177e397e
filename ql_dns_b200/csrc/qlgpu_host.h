// qlgpu_host.h -- host-side set-up shared by the single-case handle (qlgpu.cu)
// and the batch (qlgpu_batch_host.cu): parameter checks, the run constants of
// a case, the wavenumber / twiddle / 1/lap2 / integrating-factor tables, and
// the tables of compiled kernels.
#pragma once
#include <cuda_runtime.h>

#include <cmath>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <utility>
#include <vector>

#include "../../include/qlgpu.h"
#include "qlgpu_types.h"

namespace qlgpu {

struct cplx;

constexpr double kPI = 3.14159265358979323846;  // General_Definitions.h PI

typedef void (*stage_launch_fn)(const StageArgs&, const DevParams&, int grid, int block, size_t smem, cudaStream_t);
typedef cudaError_t (*run_launch_fn)(const RunArgs&, int grid, int block, size_t smem, cudaStream_t);
typedef size_t (*smem_fn)(int warps);
typedef const void* (*kptr_fn)();

// One compiled stage kernel (NZ x model x integrator).
struct Variant {
    stage_launch_fn launch;
    kptr_fn kernel;
    run_launch_fn run[2];  // many steps in one cooperative launch: plain, with noise and / or the CFL time step
    kptr_fn run_kernel[2];
    smem_fn smem;
    int PL;         // partial vector length (doubles)
    int max_warps;  // widest CTA the kernel is compiled for
};

// Defined in qlgpu_nz<NZ>.cu, one translation unit per NZ.
bool make_variant_nz16(int model, int integ, Variant* out);
bool make_variant_nz32(int model, int integ, Variant* out);
bool make_variant_nz64(int model, int integ, Variant* out);
bool make_variant_nz128(int model, int integ, Variant* out);
bool make_variant_nz256(int model, int integ, Variant* out);

inline bool pick_variant(int NZ, int model, int integ, Variant* out) {
    switch (NZ) {
        case 16: return make_variant_nz16(model, integ, out);
        case 32: return make_variant_nz32(model, integ, out);
        case 64: return make_variant_nz64(model, integ, out);
        case 128: return make_variant_nz128(model, integ, out);
        case 256: return make_variant_nz256(model, integ, out);
        default: return false;
    }
}

// The persistent batch kernel of one model x integrator (qlgpu_batch_<model>_<integ>.cu).
struct BatchKernel {
    cudaError_t (*launch)(const BatchLaunch& L, int grid, int block, size_t smem, cudaStream_t st);
    const void* (*kernel)();
    size_t (*smem)(int NZ, int warps);  // dynamic shared memory of one NZ class
    int max_warps;                      // widest CTA the build is compiled for
};
bool batch_kernel_bq_exp(BatchKernel* out);
bool batch_kernel_bq_cn(BatchKernel* out);
bool batch_kernel_fq_exp(BatchKernel* out);
bool batch_kernel_fq_cn(BatchKernel* out);

inline bool pick_batch_kernel(int model, int integ, BatchKernel* out) {
    if (model == MODEL_BQLIN)
        return integ == INTEG_EXP ? batch_kernel_bq_exp(out) : batch_kernel_bq_cn(out);
    return integ == INTEG_EXP ? batch_kernel_fq_exp(out) : batch_kernel_fq_cn(out);
}

// The dynamic shared memory limit is an attribute of the kernel function, shared
// by every handle, batch and no-allocation call of the process on a device: it
// is only ever raised, so a launch prepared by one of them is never invalidated
// by another that needs less.
inline cudaError_t ensure_smem_attr(const void* kernel, size_t bytes) {
    static std::mutex mu;
    static std::map<std::pair<int, const void*>, size_t> set;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lock(mu);
    size_t& cur = set[std::make_pair(dev, kernel)];
    if (bytes <= cur) return cudaSuccess;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e == cudaSuccess) cur = bytes;
    return e;
}

inline bool supported_nz(int NZ) { return NZ == 16 || NZ == 32 || NZ == 64 || NZ == 128 || NZ == 256; }

// Modes a team of the stage kernel steps at once and the teams of a CTA (qlgpu_wide.cuh WG).
inline int block_modes(int NZ) { return 256 / NZ; }
inline int stage_teams(int model, int warps) {
    const int n = warps / (model == MODEL_BQLIN ? 5 : 8);
    return n > 1 ? n : 1;
}

// CTA width and grid of a single case's stage kernel: one CTA per SM (sms: those left beside the
// CTAs of the mean-field side, run_kernel).  When every team can have its own SM, MHD_FullQlin and
// NZ >= 128 give a team as many warps as it has inverse transforms (one round of tasks).  MHD_BQlin
// below that has eight for its nine: the second round is short and runs under the wait for the mean
// field (a step of 32x32 x NZ=64 27.7 us, 28.0 with nine; 24x24 x NZ=128 33.5 and 32.3), and at 128
// registers two CTAs of eight warps fit an SM, of nine one, so that two handles step side by side (eight
// handles of 32x32 x NZ=64 on eight threads 124 us a step of all, 226 with nine).  Otherwise a CTA holds
// the teams that the case has blocks for.
struct StageGeom {
    int warps, grid;
};
inline StageGeom stage_geometry(int model, int NZ, int nxy, int sms, int max_grid, int max_warps) {
    const int blocks = (nxy + block_modes(NZ) - 1) / block_modes(NZ);
    const bool bq = model == MODEL_BQLIN;
    const int per_sm = (blocks + sms - 1) / sms;
    StageGeom g;
    g.warps = bq ? (per_sm <= 1 ? (NZ <= 64 ? 8 : 9) : per_sm == 2 ? 14 : max_warps) : (per_sm <= 1 ? 10 : 16);
    if (g.warps > max_warps) g.warps = max_warps;
    const int teams = stage_teams(model, g.warps);
    g.grid = (blocks + teams - 1) / teams;
    if (g.grid > sms) g.grid = sms;
    if (g.grid > max_grid) g.grid = max_grid;
    if (g.grid < 1) g.grid = 1;
    return g;
}

inline int stored_nz(int NZ) { return 1 + 2 * int(NZ / 3.0); }                   // Model.h:34
inline int mode_count(const qlgpu_params& p) { return (p.nx - 1) * (p.ny / 2); }  // Model.h:36
inline int mean_field_count(const qlgpu_params& p) { return p.model == QLGPU_MODEL_MHD_BQLIN ? 2 : 4; }

// Parameter checks of qlgpu_create; returns QLGPU_OK or an error code with *msg set.
inline int check_params(const qlgpu_params& p, std::string* msg) {
    if (p.model != QLGPU_MODEL_MHD_BQLIN && p.model != QLGPU_MODEL_MHD_FULLQLIN) {
        *msg = "unknown model (no matching model found, main.cpp:71-74)";
        return QLGPU_ERR_ARG;
    }
    if (p.integrator != QLGPU_INTEG_RK3CN_ELIN && p.integrator != QLGPU_INTEG_RK3CN) {
        *msg = "unknown integrator";
        return QLGPU_ERR_ARG;
    }
    if (p.nx < 2 || (p.nx % 2) || p.ny < 2 || (p.ny % 2)) {
        *msg = "nx and ny must be even and >= 2";
        return QLGPU_ERR_ARG;
    }
    if (!(p.dt > 0)) {
        *msg = "dt must be > 0 (variable CFL time step not supported)";
        return QLGPU_ERR_UNSUPPORTED;
    }
    if (!(p.L[0] > 0 && p.L[1] > 0 && p.L[2] > 0)) {
        *msg = "box lengths must be > 0";
        return QLGPU_ERR_ARG;
    }
    if (p.model == QLGPU_MODEL_MHD_BQLIN && p.nu == 0.0) {
        *msg = "MHD_BQlin divides by nu (MHD_BQlin.cpp:251); nu must be nonzero";
        return QLGPU_ERR_ARG;
    }
    if (!supported_nz(p.NZ)) {
        *msg = "unsupported NZ: must be a power of two in [16, 256]";
        return QLGPU_ERR_UNSUPPORTED;
    }
    return QLGPU_OK;
}

// Run constants of a case (MHD_BQlin.cpp:18-60, MHD_FullQlin.cpp:14-60).
inline DevParams make_devparams(const qlgpu_params& p) {
    DevParams d;
    std::memset(&d, 0, sizeof(d));
    d.nxy = mode_count(p);
    d.nz = stored_nz(p.NZ);
    d.NZ = p.NZ;
    d.nmf = mean_field_count(p);
    d.q = p.q;
    d.Omega = p.model == QLGPU_MODEL_MHD_BQLIN ? 2.0 / 3.0 * p.q : p.omega;
    d.nu = p.nu;
    d.eta = p.eta;
    d.etanu = p.model == QLGPU_MODEL_MHD_BQLIN ? p.eta / p.nu : p.eta;
    d.cb = p.model == QLGPU_MODEL_MHD_BQLIN ? (p.eta / p.nu) * p.nu : p.eta;
    // -|(-kx^2-ky^2)+kz2|^(order/2) is linear in kz2 only for order/2 == 1 (MHD_FullQlin.cpp:372)
    d.factored = (p.model == QLGPU_MODEL_MHD_BQLIN || p.viscosity_order / 2 == 1) ? 1 : 0;
    d.B0z = p.B0z;
    d.visc_half = p.viscosity_order / 2;
    d.ql = p.quasilinear ? 1 : 0;
    d.remap = p.remap ? 1 : 0;
    d.kzL = 2 * kPI / p.L[2];
    d.fac = 1.0 / p.NZ;
    const int Nx = p.nx, Ny = (p.ny / 2) * 2;
    d.rs_fac = 1.0 / (Ny * Nx) / (Ny * Nx);
    long totalN2 = (long)Nx * Ny * p.NZ;
    totalN2 = totalN2 * totalN2;
    d.divfac = p.L[2] / (double)totalN2;
    d.divMF = p.L[2] / ((double)p.NZ * p.NZ);
    const double kxLfac = 2 * kPI / p.L[0];
    const int nxm1 = Nx - 1;
    d.remap_thresh = nxm1 / 2.0 * kxLfac;
    d.remap_shift = nxm1 * kxLfac;
    d.dt = p.dt;
    d.tv_interval = 0.0;
    d.kzmax = 2 * kPI / p.L[2] * (p.NZ / 3);
    return d;
}

// Kdata tables (QL_DNS/Auxiliary/Kdata.cpp:24-46)
inline void ktables(const qlgpu_params& p, std::vector<double>& kx, std::vector<double>& ky, std::vector<int>& kxi,
                    std::vector<int>& kyi) {
    const double kxL = 2 * kPI / p.L[0], kyL = 2 * kPI / p.L[1];
    const int ny = ((p.ny / 2) * 2) / 2, nx = p.nx / 2;
    const int nxy = (p.nx - 1) * (p.ny / 2);
    kx.assign(nxy, 0.0);
    ky.assign(nxy, 0.0);
    kxi.assign(nxy, 0);
    kyi.assign(nxy, 0);
    for (int i = 0; i < nx; ++i)
        for (int j = 0; j < ny; ++j) {
            kx[j + ny * i] = i * kxL;
            ky[j + ny * i] = j * kyL;
            kxi[j + ny * i] = i;
            kyi[j + ny * i] = j;
        }
    for (int i = nx + 1; i < 2 * nx; ++i)
        for (int j = 0; j < ny; ++j) {
            kx[j + ny * (i - 1)] = (-2 * nx + i) * kxL;
            ky[j + ny * (i - 1)] = j * kyL;
            kxi[j + ny * (i - 1)] = -2 * nx + i;
            kyi[j + ny * (i - 1)] = j;
        }
}

// Twiddles of the 8-points-per-thread transforms: tw[q T + t] = exp(+2 pi i q t / NZ), q < 8,
// T = NZ / 8, as (re, im) pairs.
inline std::vector<double> twiddles(int NZ) {
    std::vector<double> tw(2 * (size_t)NZ);
    const int T = NZ / 8;
    for (int q = 0; q < 8; ++q)
        for (int t = 0; t < T; ++t) {
            const double ang = 2.0 * kPI * (double)(q * t % NZ) / (double)NZ;
            tw[2 * (q * T + t)] = std::cos(ang);
            tw[2 * (q * T + t) + 1] = std::sin(ang);
        }
    return tw;
}
// Diagnostics of a state in one launch (qlgpu_diag.cu): the 15-column record at time t into out.
void launch_diag(const cplx* lin, const cplx* mf, const double* kx0, const double* ky, const int* kyi,
                 const DevParams& P, double t, double* out, cudaStream_t st);

// 1/lap2 per (ky index, stored kz), Kdata.cpp:100-119
inline std::vector<double> ilap2_table(const qlgpu_params& p, int nz) {
    std::vector<double> il2((size_t)(p.ny / 2) * nz, 0.0);
    const double kyL = 2 * kPI / p.L[1], kzL = 2 * kPI / p.L[2];
    const int nzl = (nz - 1) / 2;
    for (int j = 0; j < p.ny / 2; ++j) {
        const double kyr = j * kyL;
        for (int s = 0; s < nz; ++s) {
            const int kzi = s <= nzl ? s : (-2 * nzl + s - 1);
            const double c = kzi * kzL;
            const double kz2 = 0.0 * 0.0 - c * c;
            double l2 = -kyr * kyr + kz2;
            double v = 1 / l2;
            if (kyr == 0 && s == 0) v = 1;
            il2[(size_t)j * nz + s] = v;
        }
    }
    return il2;
}

// exp(linC nu kz2), exp(linC cb kz2) per stage, [3][2][nz] (RK3CN_Elin.cpp:89,122,155)
inline std::vector<double> ekz_table(const qlgpu_params& p, const DevParams& d) {
    const int nz = d.nz;
    const double dt = p.dt;
    const double linC[3] = {dt * (a0_), dt * (a1_ + b1_), dt * (a2_ + b2_)};
    const double kzL = 2 * kPI / p.L[2];
    const int nzl = (nz - 1) / 2;
    std::vector<double> e((size_t)6 * nz, 1.0);
    for (int st = 0; st < 3; ++st)
        for (int s = 0; s < nz; ++s) {
            const int kzi = s <= nzl ? s : s - nz;
            const double c = kzi * kzL;
            const double kz2 = -(c * c);
            e[(size_t)(st * 2) * nz + s] = std::exp(linC[st] * d.nu * kz2);
            e[(size_t)(st * 2 + 1) * nz + s] = std::exp(linC[st] * d.cb * kz2);
        }
    return e;
}

// Noise constants of a case stepping with dt (MHD_FullQlin.cpp:45-66,804;
// MHD_BQlin.cpp:23-36,563): ky = 0 pairs are driven by MHD_FullQlin only.
inline NoiseSpec noise_spec(const qlgpu_params& p, int NZ, double dt, double f_noise, double k_low, double k_high,
                            unsigned long long seed, int only_velocity, int only_magnetic) {
    NoiseSpec n;
    std::memset(&n, 0, sizeof(n));
    const int Ny = (p.ny / 2) * 2;
    const double tot = (double)p.nx * (double)Ny * (double)NZ;
    n.lo2 = k_low * k_low;
    n.hi2 = k_high * k_high;
    n.tot2 = tot * tot;
    n.multfac = noise_factor(dt, n.tot2);
    n.sd = f_noise / std::sqrt(2.0);
    n.seed = seed;
    n.pair_ky0 = p.model == QLGPU_MODEL_MHD_FULLQLIN;
    n.drive_u = !only_magnetic;
    n.drive_b = !only_velocity;
    n.nxh = p.nx / 2;
    n.nyh = Ny / 2;
    return n;
}

// Stage constants of a case at its fixed time step.
inline StageConst stage_const(const qlgpu_params& p, int s) {
    return stage_const(p.dt, p.integrator == QLGPU_INTEG_RK3CN, s);
}

}  // namespace qlgpu
