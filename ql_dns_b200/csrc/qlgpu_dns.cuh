// qlgpu_dns.cuh -- FP64 kernels of the full 3-D shearing-box MHD DNS (sm_100a).
//
// One right-hand side is four launches over data that stays in L2:
//   A  dns_inv_zx<NZ,MX>  grid (ky, field):   per ky plane, the z inverse of every
//                         column (padded from nz) and the x inverse of every z row
//                         (bins kx0 mod Mx) -> X[f][ky][x][z]
//   B  dns_phys<MY>       grid (x, z chunk):  y inverse of u and b (two real fields per
//                         complex transform, Hermitian in ky), the nine products
//                         T_ij = u_i u_j - b_i b_j and E = u x b in shared memory, and
//                         their y forward transforms -> P[p][ky][x][z]
//   C  dns_fwd_xz<MX,NZ>  grid (ky, product): x forward of every z row, gather of the
//                         plane's columns, z forward and truncation -> T[p][mode][kz]
//   D  dns_update         one thread per (mode, kz): the rhs (projection, shear,
//                         rotation, B0z, the i k.T and i k x E terms), the RK3 update
//                         (RK3CN_Elin exponential or RK3CN Crank-Nicolson), the 2/3
//                         mask in x at the next stage time, the divergence correction
//                         and, at the last stage, the remap zeroing.
// Transforms are the 8-points-per-thread ones of qlgpu_xform.cuh: a warp transforms
// GPW = 256/N rows of length N at once, lane (g, t) register r holding index t + T r of
// row g before and after.  Sign and scale: backward exp(+), forward exp(-) as
// conj(xform(conj)), both unnormalised; 1/(Mx My NZ) is applied when the state is loaded.
#pragma once
#include <cuda_runtime.h>

#include "qlgpu_debug.cuh"
#include "qlgpu_xform.cuh"

namespace qlgpu {
namespace dns {

constexpr int BLOCK = 128;  // dns_update: 5 CTAs per SM, one wave at 64 x 128 x 64
constexpr int NPROD = 9;

struct DnsArgs {
    int nxy, nz, ncol, Kyn, nx;  // columns, stored kz, columns per ky, ky count, QL nx
    int Mx, My, NZ;
    int order_half, remap, integ;
    double dkx, q, omega, nu, eta, B0z, scale, kmask, dt;
    double remap_thresh, remap_shift;  // (nx-1)/2 dkx and (nx-1) dkx (MHD_FullQlin.cpp:472-474)
    const double* ky;  // [nxy]
    const double* kz;  // [nz]
    const cplx* twz;
    const cplx* twx;
    const cplx* twy;
    cplx* lin;      // [nxy][6][nz]
    double* kx0;    // [nxy]
    cplx* X;        // [6][Kyn][Mx][NZ]
    cplx* P;        // [9][Kyn][Mx][NZ]
    cplx* T;        // [9][nxy][nz]
    cplx* F[2];     // [nxy][6][nz]
    double* clock;  // [0] = t at the start of the step
    int* status;
};

struct DnsStage {
    double t_off, dt_lin, linC, n1, n2, tn_off;  // stage time t + t_off, next evaluation at t + tn_off
    int cur, prev, has_prev, last, rhs_only;     // F buffers, flags
    double t_abs;                                 // rhs_only: absolute time
};

// Programmatic dependent launch (the step's kernels are launched with it): a
// kernel lets the next one be scheduled as soon as all its CTAs have started, and
// waits for the previous kernel to complete (and its memory to be visible) before
// it touches global memory.  Without the launch attribute both are no-ops.
__device__ __forceinline__ void pdl_start() {
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
}

// Rows of length N: T lanes each, GPW rows per warp.
template <int N>
struct XG {
    static constexpr int NZ = N;
    static constexpr int T = N / 8;
    static constexpr int GPW = 32 / T;
    static constexpr bool PAD = false;  // rows of T + 1 cost the y pass 3 %
    static constexpr int SWZ = T == 4 ? 1 : (T == 2 ? 3 : 0);
};
// stored kz index of spectral slot k of an NZ-point row (fftwPlans.h:66-97), -1 in the gap
template <int NZ>
__device__ __forceinline__ int zstored(int k) {
    constexpr int H = NZ / 3;
    return k <= H ? k : (k >= NZ - H ? k - (NZ - 2 * H - 1) : -1);
}

// kx(t) = kx0 + (q t) ky, rounded as the host restatement does (no contraction)
__device__ __forceinline__ double kx_at(double kx0, double q, double t, double ky) {
    return __dadd_rn(kx0, __dmul_rn(__dmul_rn(q, t), ky));
}

__device__ __forceinline__ int xbin(double kx0, double dkx, int M) {
    long long m = llrint(kx0 / dkx);
    int b = (int)(m % M);
    return b < 0 ? b + M : b;
}

// ---------------------------------------------------------------------------
// The ky plane of A and C in shared memory, [x][z] with the 16-byte entries of a row
// permuted within 128 bytes by its x, so that the lanes of a transform along x or z read
// different banks.  The transforms exchange in place, in the entries they transform, so
// a 64 x 64 plane is 64 KB: three CTAs of 8 warps per SM, and every plane of
// 64 x 128 x 64 (258 in A, 387 in C) is resident at once.
// ---------------------------------------------------------------------------
constexpr int ZX_WARPS = 8;

template <int NZ, int MX>
struct PlaneZX {
    static constexpr size_t BYTES = sizeof(cplx) * ((size_t)NZ * MX + NZ + MX) + sizeof(int) * MX;
};
template <int NZ>
__device__ __forceinline__ int plane_at(int x, int z) {
    return x * NZ + (z ^ (x & 7));
}
// x bin of every column of the plane (bin2col[b] = column or -1)
template <int MX>
__device__ __forceinline__ void plane_bins(const DnsArgs& a, int ky, int* bin2col) {
    for (int c = threadIdx.x; c < a.ncol; c += blockDim.x)
        bin2col[QLGPU_CHECK_INDEX(xbin(a.kx0[QLGPU_CHECK_INDEX(ky + a.Kyn * c, a.nxy, a.status)], a.dkx, MX), MX,
                                  a.status)] = c;
}

// ---------------------------------------------------------------------------
// A: z inverse + x inverse of one field on one ky plane
// ---------------------------------------------------------------------------
template <int NZ, int MX>
__global__ void __launch_bounds__(32 * ZX_WARPS, 3) dns_inv_zx(const __grid_constant__ DnsArgs a) {
    using GZ = XG<NZ>;
    using GX = XG<MX>;
    extern __shared__ __align__(16) unsigned char smraw[];
    cplx* S = reinterpret_cast<cplx*>(smraw);
    cplx* twz = S + NZ * MX;
    cplx* twx = twz + NZ;
    int* bin2col = reinterpret_cast<int*>(twx + MX);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nth = blockDim.x;
    const int ky = blockIdx.x, f = blockIdx.y;
    for (int i = tid; i < NZ; i += nth) twz[i] = a.twz[i];
    for (int i = tid; i < MX; i += nth) twx[i] = a.twx[i];
    for (int b = tid; b < MX; b += nth) bin2col[b] = -1;
    __syncthreads();
    pdl_start();
    plane_bins<MX>(a, ky, bin2col);
    __syncthreads();
    {  // z inverse of every x row (zero where no column has the bin)
        constexpr int T = GZ::T;
        const int g = lane / T, t = lane % T;
        for (int x0 = warp * GZ::GPW; x0 < MX; x0 += ZX_WARPS * GZ::GPW) {
            const int xr = x0 + g, c = bin2col[xr];
            cplx x[8];
#pragma unroll
            for (int r = 0; r < 8; ++r) x[r] = mk(0.0, 0.0);
            if (c >= 0) {
                const cplx* src =
                    a.lin + ((size_t)QLGPU_CHECK_INDEX(ky + a.Kyn * c, a.nxy, a.status) * 6 + f) * a.nz;
#pragma unroll
                for (int r = 0; r < 8; ++r) {
                    const int s = QLGPU_CHECK_STORED(zstored<NZ>(t + T * r), a.nz, a.status);
                    if (s >= 0) x[r] = cscale(src[s], a.scale);
                }
            }
            xform_at<GZ>(
                x, [&](int q, int s) -> cplx& { return S[plane_at<NZ>(xr, q * T + ((s + q) & (T - 1)))]; }, twz, t);
#pragma unroll
            for (int r = 0; r < 8; ++r) S[plane_at<NZ>(xr, t + T * r)] = x[r];
        }
    }
    __syncthreads();
    {  // x inverse of every z column
        constexpr int T = GX::T;
        const int g = lane / T, t = lane % T;
        for (int z0 = warp * GX::GPW; z0 < NZ; z0 += ZX_WARPS * GX::GPW) {
            const int z = z0 + g;
            cplx x[8];
#pragma unroll
            for (int r = 0; r < 8; ++r) x[r] = S[plane_at<NZ>(t + T * r, z)];
            __syncwarp();
            xform_at<GX>(
                x, [&](int q, int s) -> cplx& { return S[plane_at<NZ>(q * T + ((s + q) & (T - 1)), z)]; }, twx, t);
#pragma unroll
            for (int r = 0; r < 8; ++r) S[plane_at<NZ>(t + T * r, z)] = x[r];
        }
    }
    __syncthreads();
    cplx* dst = a.X + ((size_t)f * a.Kyn + ky) * MX * NZ;
    for (int i = tid; i < MX * NZ; i += nth) dst[i] = S[plane_at<NZ>(i / NZ, i % NZ)];
}

// ---------------------------------------------------------------------------
// B: y transforms and the products, per (x, chunk of ZC z lines).
//
// Its chain of loads, transforms and stores bounds it, and the bytes: 17 MB in, 25 MB out
// at 64 x 128 x 64.  The chunk's spectra come in as one tile of contiguous ZC-line rows
// (each entry is used twice, for k and for its conjugate My - k) and the products' spectra
// leave the same way; the two real fields of a complex transform stay in the buffer it was
// exchanged in, where the products read them at the same lane and register.  82 KB and 8
// warps: two CTAs per SM.
// ---------------------------------------------------------------------------
template <int MY>
struct Phys {
    using G = XG<MY>;
    static constexpr int ZC = MY >= 256 ? 4 : (MY == 16 ? 16 : 8);
    static constexpr int LT = ZC / G::GPW;              // warp-tasks per field pair
    static constexpr int BUF = XWARP<G>;                // a warp-task's result / exchange buffer
    static constexpr int WARPS = MY >= 128 ? 8 : (MY == 64 ? 6 : 5);
    static constexpr int THREADS = 32 * WARPS;
    static constexpr int KYN = MY / 3 + 1;              // ky of the mode set
    static constexpr int PPR = (WARPS + LT - 1) / LT;   // product pairs per round of the forward tasks
    static_assert(WARPS % LT == 0, "a round of forward tasks holds whole pairs");
    static constexpr size_t TILE = (size_t)6 * KYN * ZC, XCH = (size_t)BUF * WARPS;
    static constexpr size_t OUT = (size_t)2 * PPR * KYN * ZC;
    static constexpr size_t WORK = TILE > XCH ? (TILE > OUT ? TILE : OUT) : (XCH > OUT ? XCH : OUT);
    static_assert(THREADS % ZC == 0, "whole tile rows per pass");
    static size_t smem() { return sizeof(cplx) * ((size_t)3 * LT * BUF + WORK + MY); }
};
// tile row (field or product, k), line l: 16-byte entries permuted within 128 bytes, so that a
// transform's lanes (consecutive k, one line) read different banks
template <int ZC>
__device__ __forceinline__ int tile_at(int row, int l) {
    return row * ZC + (l ^ (row & (ZC - 1) & 7));
}

__device__ __forceinline__ double product(int p, const double* v) {
    // v = ux, uy, uz, bx, by, bz
    switch (p) {
        case 0: return v[0] * v[0] - v[3] * v[3];
        case 1: return v[1] * v[1] - v[4] * v[4];
        case 2: return v[2] * v[2] - v[5] * v[5];
        case 3: return v[0] * v[1] - v[3] * v[4];
        case 4: return v[0] * v[2] - v[3] * v[5];
        case 5: return v[1] * v[2] - v[4] * v[5];
        case 6: return v[1] * v[5] - v[2] * v[4];
        case 7: return v[2] * v[3] - v[0] * v[5];
        case 8: return v[0] * v[4] - v[1] * v[3];
        default: return 0.0;
    }
}

// conj of products 2 PP and 2 PP + 1 as one complex row, from the three field pairs of the lane
template <int PP, int LT, int BUF>
__device__ __forceinline__ void product_pair(cplx (&x)[8], const cplx* ph) {
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        double f6[6];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const cplx v = ph[BUF * q * LT + 32 * r];
            f6[2 * q] = v.x;
            f6[2 * q + 1] = v.y;
        }
        x[r] = mk(product(2 * PP, f6), 2 * PP + 1 < NPROD ? -product(2 * PP + 1, f6) : 0.0);
    }
}

template <int MY>
__global__ void __launch_bounds__(Phys<MY>::THREADS, 2) dns_phys(const __grid_constant__ DnsArgs a) {
    using K = Phys<MY>;
    using G = typename K::G;
    constexpr int T = G::T, GPW = G::GPW, ZC = K::ZC, LT = K::LT, KYN = K::KYN, BUF = K::BUF;
    extern __shared__ __align__(16) unsigned char smraw[];
    cplx* Ph = reinterpret_cast<cplx*>(smraw);   // [3 LT warp-tasks][BUF], [8][32] each: the pairs (ux,uy), (uz,bx), (by,bz)
    cplx* work = Ph + (size_t)3 * LT * BUF;       // input tile; then exchange buffers / output tile
    cplx* tw = work + K::WORK;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nth = blockDim.x;
    const int g = lane / T, t = lane % T;
    const int x0 = blockIdx.x, z0 = blockIdx.y * ZC;
    const size_t plane = (size_t)a.Mx * a.NZ;
    const size_t off = (size_t)x0 * a.NZ + z0;
    for (int i = tid; i < MY; i += nth) tw[i] = a.twy[i];
    pdl_start();
    for (int row = tid / ZC, l = tid % ZC; row < 6 * KYN; row += K::THREADS / ZC)
        cp_async16(work + tile_at<ZC>(row, l), a.X + (size_t)row * plane + off + l);
    cp_async_commit();
    cp_async_wait_all();
    __syncthreads();
    // inverse: three complex transforms per line, c(k) = A + i B, c(My - k) = conj(A) + i conj(B)
    for (int task = warp; task < 3 * LT; task += K::WARPS) {
        const int pr = task / LT, l = (task % LT) * GPW + g;
        const int ra = 2 * pr * KYN, rb = ra + KYN;  // the fields' first tile rows
        cplx x[8];
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const int k = t + T * r;
            cplx c = mk(0.0, 0.0);
            if (k < KYN) {
                cplx A = work[tile_at<ZC>(ra + k, l)], B = work[tile_at<ZC>(rb + k, l)];
                if (k == 0) { A.y = 0.0; B.y = 0.0; }
                c = mk(A.x - B.y, A.y + B.x);
            } else if (k > MY - KYN) {
                const int kk = MY - k;
                const cplx A = work[tile_at<ZC>(ra + kk, l)], B = work[tile_at<ZC>(rb + kk, l)];
                c = mk(A.x + B.y, B.x - A.y);
            }
            x[r] = c;
        }
        cplx* xb = Ph + BUF * task;
        xform<G>(x, xb, tw, g, t);
#pragma unroll
        for (int r = 0; r < 8; ++r) xb[32 * r + lane] = x[r];
    }
    __syncthreads();
    // products and their forward transforms, two per complex transform: pair pp of the lines of
    // warp-task lt is task pp LT + lt
#pragma unroll 1
    for (int base = 0; base < 5 * LT; base += K::WARPS) {
        const int task = base + warp;
        const bool on = task < 5 * LT;
        const int pp = task / LT, lt = task % LT, l = lt * GPW + g;
        cplx x[8];
        if (on) {
            const cplx* ph = Ph + BUF * lt + lane;
            switch (pp) {
                case 0: product_pair<0, LT, BUF>(x, ph); break;
                case 1: product_pair<1, LT, BUF>(x, ph); break;
                case 2: product_pair<2, LT, BUF>(x, ph); break;
                case 3: product_pair<3, LT, BUF>(x, ph); break;
                default: product_pair<4, LT, BUF>(x, ph); break;
            }
            xform<G>(x, work + BUF * warp, tw, g, t);
        }
        __syncthreads();  // the exchange buffers become the output tile
        if (on) {
            const int ra = 2 * (pp - base / LT) * KYN, rb = ra + KYN;
            const int lm = g * T + ((T - t) & (T - 1));  // the lane of My - k
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                if (T * r >= KYN) break;
                // c(k) and c(My - k): register 8 - r of this lane for t = 0, 7 - r of lane T - t
                const cplx c = conjc(x[r]);
                cplx m = mk(__shfl_sync(0xffffffffu, x[7 - r].x, lm), __shfl_sync(0xffffffffu, x[7 - r].y, lm));
                if (t == 0) m = x[(8 - r) & 7];
                m.y = -m.y;
                const int k = t + T * r;
                if (k < KYN) {
                    work[tile_at<ZC>(ra + k, l)] = mk(0.5 * (c.x + m.x), 0.5 * (c.y - m.y));
                    work[tile_at<ZC>(rb + k, l)] = mk(0.5 * (c.y + m.y), -0.5 * (c.x - m.x));
                }
            }
        }
        __syncthreads();
        // the round's products, whole rows of ZC lines
        const int p0 = 2 * (base / LT), np = min(2 * K::PPR, NPROD - p0);
        for (int row = tid / ZC, l2 = tid % ZC; row < np * KYN; row += K::THREADS / ZC)
            a.P[((size_t)p0 * KYN + row) * plane + off + l2] = work[tile_at<ZC>(row, l2)];
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// C: x forward + z forward of one product on one ky plane
// ---------------------------------------------------------------------------
template <int MX, int NZ>
__global__ void __launch_bounds__(32 * ZX_WARPS, 3) dns_fwd_xz(const __grid_constant__ DnsArgs a) {
    using GZ = XG<NZ>;
    using GX = XG<MX>;
    extern __shared__ __align__(16) unsigned char smraw[];
    cplx* S = reinterpret_cast<cplx*>(smraw);
    cplx* twz = S + NZ * MX;
    cplx* twx = twz + NZ;
    int* bin2col = reinterpret_cast<int*>(twx + MX);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nth = blockDim.x;
    const int ky = blockIdx.x, p = blockIdx.y;
    for (int i = tid; i < NZ; i += nth) twz[i] = a.twz[i];
    for (int i = tid; i < MX; i += nth) twx[i] = a.twx[i];
    for (int b = tid; b < MX; b += nth) bin2col[b] = -1;
    __syncthreads();
    pdl_start();
    const cplx* src = a.P + ((size_t)p * a.Kyn + ky) * MX * NZ;
    for (int i = tid; i < MX * NZ; i += nth) cp_async16(S + plane_at<NZ>(i / NZ, i % NZ), src + i);
    cp_async_commit();
    plane_bins<MX>(a, ky, bin2col);
    cp_async_wait_all();
    __syncthreads();
    {  // x forward of every z column (the conjugates are kept: the z transform takes them)
        constexpr int T = GX::T;
        const int g = lane / T, t = lane % T;
        for (int z0 = warp * GX::GPW; z0 < NZ; z0 += ZX_WARPS * GX::GPW) {
            const int z = z0 + g;
            cplx x[8];
#pragma unroll
            for (int r = 0; r < 8; ++r) x[r] = conjc(S[plane_at<NZ>(t + T * r, z)]);
            __syncwarp();
            xform_at<GX>(
                x, [&](int q, int s) -> cplx& { return S[plane_at<NZ>(q * T + ((s + q) & (T - 1)), z)]; }, twx, t);
#pragma unroll
            for (int r = 0; r < 8; ++r) S[plane_at<NZ>(t + T * r, z)] = x[r];
        }
    }
    __syncthreads();
    {  // z forward of every x row that is a column's bin, truncated to the stored kz
        constexpr int T = GZ::T;
        const int g = lane / T, t = lane % T;
        for (int x0 = warp * GZ::GPW; x0 < MX; x0 += ZX_WARPS * GZ::GPW) {
            const int xr = x0 + g, c = bin2col[xr];
            cplx x[8];
#pragma unroll
            for (int r = 0; r < 8; ++r) x[r] = S[plane_at<NZ>(xr, t + T * r)];
            __syncwarp();
            xform_at<GZ>(
                x, [&](int q, int s) -> cplx& { return S[plane_at<NZ>(xr, q * T + ((s + q) & (T - 1)))]; }, twz, t);
            if (c >= 0) {
                cplx* dst = a.T + ((size_t)p * a.nxy + QLGPU_CHECK_INDEX(ky + a.Kyn * c, a.nxy, a.status)) * a.nz;
#pragma unroll
                for (int r = 0; r < 8; ++r) {
                    const int s = QLGPU_CHECK_STORED(zstored<NZ>(t + T * r), a.nz, a.status);
                    if (s >= 0) dst[s] = conjc(x[r]);
                }
            }
        }
    }
}

// ---------------------------------------------------------------------------
// D: right-hand side, RK3 update, mask, divergence correction, remap zeroing
// ---------------------------------------------------------------------------
__device__ __forceinline__ double ipow(double x, int n) {
    double r = 1.0;
    for (int i = 0; i < n; ++i) r *= x;
    return r;
}

// -|k|^(2 order_half) at kx = kx0 + q t ky (+ q dt_lin ky), MHD_FullQlin.cpp:371-376
__device__ __forceinline__ double lap_order(const DnsArgs& a, double kx0, double ky, double kz, double t,
                                            double dt_lin) {
    double kxt = kx_at(kx0, a.q, t, ky);
    kxt = kx_at(kxt, a.q, dt_lin, ky);
    const double kz2 = -__dmul_rn(kz, kz);
    return -ipow(fabs(__dadd_rn(__dsub_rn(-__dmul_rn(kxt, kxt), __dmul_rn(ky, ky)), kz2)), a.order_half);
}

__device__ __forceinline__ cplx cmuli(cplx a) { return mk(-a.y, a.x); }  // i a

__global__ void __launch_bounds__(BLOCK, 5)
    dns_update(const __grid_constant__ DnsArgs a, const __grid_constant__ DnsStage st) {
    pdl_start();
    const int idx = blockIdx.x * BLOCK + threadIdx.x;
    if (idx >= a.nxy * a.nz) return;
    const int mode = idx / a.nz, s = idx % a.nz;
    const double t0 = st.rhs_only ? st.t_abs : a.clock[0];
    const double ts = st.rhs_only ? st.t_abs : t0 + st.t_off;
    const double kx0 = a.kx0[mode], ky = a.ky[mode], kz = a.kz[s];
    const double Kx = kx_at(kx0, a.q, ts, ky);
    cplx u[6];
#pragma unroll
    for (int c = 0; c < 6; ++c) u[c] = a.lin[((size_t)mode * 6 + c) * a.nz + s];
    cplx Tm[NPROD];
#pragma unroll
    for (int p = 0; p < NPROD; ++p) Tm[p] = a.T[((size_t)p * a.nxy + mode) * a.nz + s];
    const double om = a.omega, q = a.q, B0z = a.B0z;
    // A = -i k.T + (2 Om u_y, (q - 2 Om) u_x, 0) + i kz B0z b
    cplx kT[3];
    kT[0] = mk(Kx * Tm[0].x + ky * Tm[3].x + kz * Tm[4].x, Kx * Tm[0].y + ky * Tm[3].y + kz * Tm[4].y);
    kT[1] = mk(Kx * Tm[3].x + ky * Tm[1].x + kz * Tm[5].x, Kx * Tm[3].y + ky * Tm[1].y + kz * Tm[5].y);
    kT[2] = mk(Kx * Tm[4].x + ky * Tm[5].x + kz * Tm[2].x, Kx * Tm[4].y + ky * Tm[5].y + kz * Tm[2].y);
    cplx A[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const cplx mi = mk(kT[c].y, -kT[c].x);           // -i kT
        const cplx bz = cmuli(cscale(u[3 + c], kz * B0z));  // i kz B0z b
        A[c] = cadd(mi, bz);
    }
    A[0] = cadd(A[0], cscale(u[1], 2 * om));
    A[1] = cadd(A[1], cscale(u[0], q - 2 * om));
    const double K2 = Kx * Kx + ky * ky + kz * kz;
    const double iK2 = K2 > 0 ? 1.0 / K2 : 0.0;
    cplx sdot = cadd(cadd(cscale(A[0], Kx), cscale(A[1], ky)), cadd(cscale(A[2], kz), cscale(u[0], q * ky)));
    sdot = cscale(sdot, iK2);
    cplx F[6];
    F[0] = csub(A[0], cscale(sdot, Kx));
    F[1] = csub(A[1], cscale(sdot, ky));
    F[2] = csub(A[2], cscale(sdot, kz));
    // i k x E + (0, -q b_x, 0) + i kz B0z u
    const cplx Ex = Tm[6], Ey = Tm[7], Ez = Tm[8];
    F[3] = cadd(cmuli(csub(cscale(Ez, ky), cscale(Ey, kz))), cmuli(cscale(u[0], kz * B0z)));
    F[4] = cadd(csub(cmuli(csub(cscale(Ex, kz), cscale(Ez, Kx))), cscale(u[3], q)), cmuli(cscale(u[1], kz * B0z)));
    F[5] = cadd(cmuli(csub(cscale(Ey, Kx), cscale(Ex, ky))), cmuli(cscale(u[2], kz * B0z)));
    const bool keep_s = fabs(Kx) <= a.kmask;
    if (!keep_s) {
#pragma unroll
        for (int c = 0; c < 6; ++c) F[c] = mk(0.0, 0.0);
    }
    cplx* Fc = a.F[st.cur];
#pragma unroll
    for (int c = 0; c < 6; ++c) Fc[((size_t)mode * 6 + c) * a.nz + s] = F[c];
    if (st.rhs_only) return;
    // update (RK3CN_Elin.cpp:102-104 / RK3CN.cpp:105-107), operator at t_s + dt_lin
    // the kx = ky = 0 column (the means) has ordinary diffusion at every order, as the
    // mean-field operator of MHD_FullQlin (linOpMF = coef kz2, MHD_FullQlin.cpp:449-455)
    const bool mean_col = (mode == 0);
    const double kz2m = -__dmul_rn(kz, kz);
    const double Lu = mean_col ? a.nu * kz2m : a.nu * lap_order(a, kx0, ky, kz, ts, st.dt_lin);
    const double Lb = mean_col ? a.eta * kz2m : a.eta * lap_order(a, kx0, ky, kz, ts, st.dt_lin);
    const cplx* Fp = a.F[st.prev];
    cplx nw[6];
    if (a.integ == 0) {
        const double eu = exp(st.linC * Lu), eb = exp(st.linC * Lb);
#pragma unroll
        for (int c = 0; c < 6; ++c) {
            cplx acc = cscale(F[c], st.n1);
            if (st.has_prev) acc = cadd(acc, cscale(Fp[((size_t)mode * 6 + c) * a.nz + s], st.n2));
            nw[c] = cscale(cadd(acc, u[c]), c < 3 ? eu : eb);
        }
    } else {
        const double Lou = mean_col ? Lu : a.nu * lap_order(a, kx0, ky, kz, ts, 0.0);
        const double Lob = mean_col ? Lb : a.eta * lap_order(a, kx0, ky, kz, ts, 0.0);
#pragma unroll
        for (int c = 0; c < 6; ++c) {
            const double L = c < 3 ? Lu : Lb, Lo = c < 3 ? Lou : Lob;
            cplx acc = cscale(F[c], st.n1);
            if (st.has_prev) acc = cadd(acc, cscale(Fp[((size_t)mode * 6 + c) * a.nz + s], st.n2));
            acc = cadd(acc, cscale(u[c], 1 + st.linC * Lo));
            nw[c] = cscale(acc, 1.0 / (1.0 - st.linC * L));
        }
    }
    // 2/3 mask in x and divergence correction at the next evaluation time
    const double tn = t0 + st.tn_off;
    const double Kxn = kx_at(kx0, q, tn, ky);
    bool zero = fabs(Kxn) > a.kmask;
    if (st.last && a.remap) zero = zero || (Kxn > a.remap_thresh);
    if (zero) {
#pragma unroll
        for (int c = 0; c < 6; ++c) nw[c] = mk(0.0, 0.0);
    } else {
        const double kp2 = ky * ky + kz * kz;
        const double ikp = kp2 > 0 ? 1.0 / kp2 : 0.0;
#pragma unroll
        for (int b = 0; b < 6; b += 3) {
            const cplx D = cadd(cadd(cscale(nw[b], Kxn), cscale(nw[b + 1], ky)), cscale(nw[b + 2], kz));
            if (kp2 > 0) {
                nw[b + 1] = csub(nw[b + 1], cscale(cscale(D, ky), ikp));
                nw[b + 2] = csub(nw[b + 2], cscale(cscale(D, kz), ikp));
            } else if (Kxn != 0.0) {
                nw[b] = mk(0.0, 0.0);
            } else {
                nw[b + 2] = mk(0.0, 0.0);
            }
        }
    }
    bool bad = false;
#pragma unroll
    for (int c = 0; c < 6; ++c) {
        bad = bad || !isfinite(nw[c].x) || !isfinite(nw[c].y);
        a.lin[((size_t)mode * 6 + c) * a.nz + s] = nw[c];
    }
    if (bad) atomicOr(a.status, 1);
}

// After the last stage, one CTA: shift kx0 of the columns that left the box (their
// fields were zeroed by dns_update), MHD_FullQlin.cpp:464-481, and the clock.
__global__ void __launch_bounds__(1024) dns_end_step(const __grid_constant__ DnsArgs a) {
    pdl_start();
    const double tn = a.clock[0] + a.dt;
    __syncthreads();
    if (threadIdx.x == 0) a.clock[0] = tn;
    if (!a.remap) return;
    for (int i = threadIdx.x; i < a.nxy; i += blockDim.x) {
        const double kxt = kx_at(a.kx0[i], a.q, tn, a.ky[i]);
        if (kxt > a.remap_thresh) a.kx0[i] = __dsub_rn(a.kx0[i], a.remap_shift);
    }
}

// ---------------------------------------------------------------------------
// Diagnostics: one warp per column, then one block in fixed order
// ---------------------------------------------------------------------------
__global__ void dns_diag_modes(DnsArgs a, double* part) {
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (w >= a.nxy) return;
    const double t = a.clock[0];
    const double Kx = kx_at(a.kx0[w], a.q, t, a.ky[w]), ky = a.ky[w];
    double acc[6] = {0, 0, 0, 0, 0, 0};
    for (int s = lane; s < a.nz; s += 32) {
        const cplx* c = a.lin + (size_t)w * 6 * a.nz + s;
        const cplx ux = c[0], uy = c[a.nz], uz = c[2 * a.nz];
        const cplx bx = c[3 * a.nz], by = c[4 * a.nz], bz = c[5 * a.nz];
        const double kz = a.kz[s];
        if (w == 0) {  // means: energy, stress, dissipation of (Ux, Uy) and (Bx, By)
            const double eu = ux.x * ux.x + ux.y * ux.y + uy.x * uy.x + uy.y * uy.y;
            const double eb = bx.x * bx.x + bx.y * bx.y + by.x * by.x + by.y * by.y;
            acc[0] += eu;
            acc[1] += eb;
            acc[2] += ux.x * uy.x + ux.y * uy.y;
            acc[3] += bx.x * by.x + bx.y * by.y;
            acc[4] += kz * kz * eu;
            acc[5] += kz * kz * eb;
        } else {
            const double eu = ux.x * ux.x + ux.y * ux.y + uy.x * uy.x + uy.y * uy.y + uz.x * uz.x + uz.y * uz.y;
            const double eb = bx.x * bx.x + bx.y * bx.y + by.x * by.x + by.y * by.y + bz.x * bz.x + bz.y * bz.y;
            const double K2 = Kx * Kx + ky * ky + kz * kz;
            acc[0] += eu;
            acc[1] += eb;
            acc[2] += ux.x * uy.x + ux.y * uy.y;
            acc[3] += bx.x * by.x + bx.y * by.y;
            acc[4] += K2 * eu;
            acc[5] += K2 * eb;
        }
    }
#pragma unroll
    for (int k = 0; k < 6; ++k)
        for (int o = 16; o > 0; o >>= 1) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], o);
    if (lane == 0) {
        const double wgt = (w != 0 && ky != 0.0) ? 2.0 : 1.0;  // conjugate column counted
#pragma unroll
        for (int k = 0; k < 6; ++k) part[(size_t)w * 6 + k] = acc[k] * wgt;
    }
}

__global__ void __launch_bounds__(256) dns_diag_final(DnsArgs a, const double* part, double divf, double kzmax,
                                                      double* out) {
    __shared__ double sh[256][6];
    const int tid = threadIdx.x;
    double acc[6] = {0, 0, 0, 0, 0, 0};
    for (int m = 1 + tid; m < a.nxy; m += 256)
        for (int k = 0; k < 6; ++k) acc[k] += part[(size_t)m * 6 + k];
    for (int k = 0; k < 6; ++k) sh[tid][k] = acc[k];
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if (tid < o)
            for (int k = 0; k < 6; ++k) sh[tid][k] += sh[tid + o][k];
        __syncthreads();
    }
    if (tid == 0) {
        const double Eu = sh[0][0] * divf, Eb = sh[0][1] * divf;
        const double AMu = sh[0][2] * divf, AMb = sh[0][3] * divf;
        const double Du = a.nu * sh[0][4] * divf, Db = a.eta * sh[0][5] * divf;
        const double eMU = part[0] * divf, eMB = part[1] * divf, aMU = part[2] * divf, aMB = part[3] * divf;
        const double dMU = a.nu * part[4] * divf, dMB = a.eta * part[5] * divf;
        out[0] = a.clock[0];
        out[1] = eMU / 2; out[2] = eMB / 2; out[3] = Eu / 2; out[4] = Eb / 2;
        out[5] = aMU; out[6] = aMB; out[7] = AMu; out[8] = AMb;
        out[9] = dMU; out[10] = dMB; out[11] = Du; out[12] = Db;
        out[13] = pow(a.nu * a.nu * a.nu / (dMU + Du), 0.25) * kzmax;
        out[14] = pow(a.eta * a.eta * a.eta / (dMB + Db), 0.25) * kzmax;
    }
}

}  // namespace dns
}  // namespace qlgpu
