// qlgpu_adjoint.cuh -- discrete adjoint of one RK3CN_Elin or RK3CN stage of
// MHD_BQlin (sm_100a kernels).  No counterpart in the reference.
//
// Forward stage (QL_DNS/Integrators/RK3CN_Elin.cpp:86-177 with
// QL_DNS/Models/MHD_BQlin.cpp:117-284), per mode, with R_f = P(fac f) the
// padded inverse transform and T the truncated forward transform (P^H = T):
//   F_b   = T(i b By R_u)
//   F_zeta= T(-i a dBy R_b + ddBy R_bz + i b By R_eta) + (q - 2 Omega) i c u
//   F_eta = T(-i a dBy R_u + i b By R_zeta - 2 dBy R_{i c uz} - ddBy R_uz) - q i c b
//   F_u   = T(i b By R_b) + ilapF (T(2 a b dBy R_bz) + 2 a b q u + 2 Omega i c zeta)
//   u' = E (n1 F + n2 Fprev + u),   E = exp(linC L)            (RK3CN_Elin.cpp:102-104)
//   u' = D (n1 F + n2 Fprev) + C u,  D = 1/(1 - linC L), C = (1 + linC Lold) D
//                                                              (RK3CN.cpp:105-107, Lold the
//                                                               previous stage's operator)
// and for the mean field G_Bx = EMF_x, G_By = -q Bx + EMF_y with the real
// stress profiles  Ex = sum_modes mult (Re(R_bz R_u*) - Re(R_uz R_b*)),
// Ey = sum_modes mult (Re(R_bz R_uy*) - Re(R_uz R_by*)), EMF = rs_fac i kz T(E)
// (half spectrum mirrored), B' = E_B (n1 G + n2 Gprev + B).
//
// The adjoint of a stage maps (lamU', lamB', lamF_out, lamG_out) to
// (lamU, lamB, lamFprev, lamGprev) with the real inner product
// <x, y> = Re sum conj(x) y:  mu = E lamU', lamF = n1 mu + lamF_out,
// lamU = mu + (dR/dU)^H lamF + (dEMF/dU)^H lamG, lamFprev = n2 mu, and the
// mean-field part likewise (Crank-Nicolson: mu = D lamU' and the direct term
// C lamU' in place of mu).
//
// Two kernels per stage, for one seed or many (seed = blockIdx.y):
//   adj_modes_kernel  a team of warps (one CTA) per chunk of modes: 14 inverse transforms
//                     (the nine forward real-space fields and five back-propagated rhs
//                     fields W = P(lamF)), the pointwise adjoints formed as inputs of nine
//                     forward transforms, and the spectral chain back to (u, zeta, b, eta);
//                     the chunk's sum of the adjoint of the mean-field profiles.
//   adj_mf_kernel     one CTA per seed: the sum of those over the chunks, the rest of the
//                     mean-field adjoint of the stage, and the profiles of the next one.
// Both are launched with programmatic dependent launch: a chunk's inverse transforms need
// only the mode kernel before the running mean-field kernel, and the mean-field kernel's
// forward profiles need neither, so each kernel's first half runs under the other.
#pragma once
#include "qlgpu_debug.cuh"
#include "qlgpu_stage.cuh"
#include "qlgpu_xform.cuh"

namespace qlgpu {

// Per-seed buffers of the reverse sweep (a device table).
struct AdjSeedBufs {
    const CnRec* cn_pre;   // [C][3] RK3CN old-operator fields at every stage start (null: RK3CN_Elin)
    const cplx* stU;       // [C][3] recorded stage inputs
    const cplx* stB;       // [C][3] recorded stage mean fields
    const cplx* postU;     // the window's end state
    const double* kx_pre;  // [C] kx0 at every step start
    const double* kx_post; // kx0 at the window end
    const double* t_pre;   // [C + 1] step start times
    cplx* lamU[2];
    cplx* lamB[2];
    cplx* lamF[2];
    cplx* lamG[2];
    double* prof;          // [5][NZ]: By, dBy, ddBy, px, py (real space)
    double* bpart;         // [nchunk][3][NZ] chunk sums of the adjoint of the mean-field profiles
};

// Tables and parameters the seeds share.
struct AdjShared {
    const AdjSeedBufs* seeds;
    const double* ky;
    const int* kxi;
    const int* kyi;
    const double* ilap2;   // [Ny/2][nz]
    const cplx* tw8;       // transform twiddles [8][NZ/8]
    int* status;           // the first handle's status word (debug-build index checks)
    long long nlin, nmfe;
    int nchunk, cblocks;   // chunks per seed, blocks of 256/NZ modes per chunk
    int integ;             // INTEG_EXP or INTEG_CN
    int pad;
    double weight;         // of AM_b in J
};

// Position in the sweep: stage s of step n of a window of `steps` steps.
struct AdjPos {
    int n, steps, s;
    int par;  // stages already reversed, mod 2: lamU[par] is the current adjoint state
    StageConst sc;
};

// The programmatic-launch pair: the next kernel may start / the kernels before are complete.
__device__ __forceinline__ void pdl_next() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }

// Geometry of the team kernels: T = NZ/8 lanes per transform, GPW modes per block.
template <int NZ_>
struct AG {
    static constexpr int NZ = NZ_;
    static constexpr int T = NZ_ / 8;
    static constexpr int nz = 1 + 2 * (NZ_ / 3);
    static constexpr int H = (nz - 1) / 2;
    static constexpr int GPW = 32 / T;
    static constexpr int SWZ = T == 4 ? 1 : (T == 2 ? 3 : 0);
    static constexpr int NZE = (nz + 1) & ~1;
    static constexpr int NR = 16;  // 14 inverse results, 2 exchange buffers
    static constexpr bool PAD = T >= 8;
    static constexpr int XW = PAD ? 8 * GPW * (T + 1) : 256;  // one of them (cplx)
    static constexpr size_t o_tw = 0;                                    // [8][T] cplx
    static constexpr size_t o_prof = o_tw + 16 * (size_t)NZ_;           // [5][NZ]
    static constexpr size_t o_kz = o_prof + 8 * 5 * (size_t)NZ_;        // kz per spectral slot
    static constexpr size_t o_e = o_kz + 8 * (size_t)NZ_;               // [GPW][2][NZE] E or D of the block's modes
    static constexpr size_t o_acc = o_e + 16 * (size_t)GPW * NZE;       // [3][8][32] profile sums
    static constexpr size_t o_R = o_acc + 8 * 3 * 256;                  // [NR][XW] cplx, a result at [8][32]
    static constexpr size_t o_stg = o_R + 16 * XW * (size_t)NR;        // [GPW][4][nz] cplx: U
    static constexpr size_t o_lf = o_stg + 16 * (size_t)GPW * 4 * nz;   // [GPW][4][nz] cplx: lamF
    static constexpr size_t o_il2 = o_lf + 16 * (size_t)GPW * 4 * nz;   // [GPW][nz] 1/lap2
    static constexpr size_t BYTES = o_il2 + 8 * (size_t)GPW * nz;
};
inline int adj_block_modes(int NZ) { return 256 / NZ; }

enum { A_RU = 0, A_RZ, A_RB, A_RE, A_RUZ, A_RBZ, A_RIK, A_RUY, A_RBY, A_WB, A_WZ, A_WE, A_WS, A_WU2, A_X0, A_X1 };

// One lane's mode in the stage being reversed.
struct AdjLane {
    int m, kyi, kxi;
    bool valid;
    double a, b, kxo, mult;
    int old_init;
};

// E = exp(linC L) (RK3CN_Elin.cpp:102-104) or D = 1/(1 - linC L) (RK3CN.cpp:105) of (u, zeta), side 0,
// or (b, eta), side 1, at stored index s; kxe: kx at the stage end.  One exp: a
// product of the mode's and kz's factors, as the forward stage takes it, has three roundings, the same at
// every stage (gradient of 32x32 x NZ=64 over 100 steps 3.4e-15 from the 64-bit restatement, 1.9e-15 so).
__device__ __forceinline__ double adj_e(const DevParams& P, const StageConst& S, double kxe, double ky, double kz2,
                                        int side, int integ) {
    const double L = linop_f<MODEL_BQLIN>(P, lap_end<MODEL_BQLIN>(P, kxe, ky, kz2), 2 * side);
    return integ == INTEG_CN ? __drcp_rn(__dsub_rn(1.0, __dmul_rn(S.linC, L))) : exp(__dmul_rn(S.linC, L));
}

// The stage adjoint of the chunk's modes.  What bounds it: the transforms' chain of a block
// (two deep) at one seed, the instruction and barrier latency at many.  Eight warps at 128
// registers leave room for a second CTA per SM, whose transforms run under the barriers of the
// first (nine, one round of the forward transforms, would have 96 registers and spill); with at most one chunk per SM a CTA has 16 warps, one
// round of the 14 inverse transforms too.
constexpr int ADJ_FEW = 512, ADJ_MANY = 256;  // threads

template <int NZ, int THREADS>
__global__ void __launch_bounds__(THREADS, THREADS == ADJ_MANY ? 2 : 1)
    adj_modes_kernel(const __grid_constant__ AdjShared H, const __grid_constant__ DevParams P,
                     const __grid_constant__ AdjPos X) {
    using W = AG<NZ>;
    constexpr int T = W::T, nzd = W::nz, GPW = W::GPW;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cplx* tw = reinterpret_cast<cplx*>(smem_raw + W::o_tw);
    double* prof = reinterpret_cast<double*>(smem_raw + W::o_prof);
    double* kzc = reinterpret_cast<double*>(smem_raw + W::o_kz);
    double* e_all = reinterpret_cast<double*>(smem_raw + W::o_e);
    double* acc = reinterpret_cast<double*>(smem_raw + W::o_acc);
    cplx* R = reinterpret_cast<cplx*>(smem_raw + W::o_R);
    cplx* stg_all = reinterpret_cast<cplx*>(smem_raw + W::o_stg);
    cplx* lf_s = reinterpret_cast<cplx*>(smem_raw + W::o_lf);
    double* il2_all = reinterpret_cast<double*>(smem_raw + W::o_il2);
    constexpr int warps = THREADS / 32, nth = THREADS;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane / T, t = lane % T;
    const AdjSeedBufs& B = H.seeds[blockIdx.y];
    const StageConst& S = X.sc;
    const int par = X.par;
    const cplx* U = B.stU + (size_t)(3 * X.n + X.s) * H.nlin;
    const cplx* lo_all = B.lamU[par];
    const cplx* lf_all = X.s == 2 ? nullptr : B.lamF[par];
    cplx* lu_all = B.lamU[par ^ 1];
    cplx* lp_all = X.s == 0 ? nullptr : B.lamF[par ^ 1];
    const double* kx0 = B.kx_pre + (size_t)X.n * P.nxy;
    const int first = (int)blockIdx.x * H.cblocks * GPW;
    const int end = min(P.nxy, first + H.cblocks * GPW);
    auto stage_block = [&](int base) {
        const int n = min(GPW, P.nxy - base) * 4 * nzd;
        for (int i = tid; i < n; i += nth) cp_async16(stg_all + i, U + (size_t)base * 4 * nzd + i);
        for (int i = tid; i < n / 4; i += nth)
            cp_async8(il2_all + i, H.ilap2 + (size_t)__ldg(H.kyi + base + i / nzd) * nzd + i % nzd);
        cp_async_commit();
    };
    stage_block(first);
    for (int i = tid; i < NZ; i += nth) {
        tw[i] = ldc_cg(H.tw8 + i);
        kzc[i] = kzval(i <= W::H ? i : i - NZ, P.kzL);
    }
    for (int i = tid; i < 3 * 256; i += nth) acc[i] = 0.0;
    const double tclock = B.t_pre[X.n];
    const double ts = __dadd_rn(tclock, S.t_off);
    auto buf = [&](int i) { return R + i * W::XW; };
    const double Om2 = __dmul_rn(2.0, P.Omega), fac = P.fac;

    for (int base = first; base < end; base += GPW) {
        const int nv = min(GPW, end - base);
        AdjLane M;
        M.valid = g < nv;
        M.m = QLGPU_CHECK_INDEX(base + min(g, nv - 1), P.nxy, H.status);
        const cplx* stg = stg_all + (size_t)min(g, nv - 1) * 4 * nzd;
        M.b = __ldg(H.ky + M.m);
        M.kyi = __ldg(H.kyi + M.m);
        M.kxi = __ldg(H.kxi + M.m);
        const double k0 = kx0[M.m];
        M.a = kx_at(k0, P.q, ts, M.b);
        M.mult = M.valid ? (M.b == 0.0 ? 1.0 : 2.0) : 0.0;
        M.kxo = 0.0;
        M.old_init = 0;
        if (H.integ == INTEG_CN) {
            // kx where the previous stage's operator was evaluated (RK3CN.cpp:119-122; the init form
            // at the run's start, RK3CN.cpp:57), as the forward stage computes it
            const CnRec* cn = B.cn_pre + (size_t)3 * X.n + X.s;
            M.old_init = cn->old_init;
            if (M.old_init) M.kxo = kx_at(k0, P.q, tclock, M.b);
            else M.kxo = __dadd_rn(kx_at(k0, P.q, cn->t_old, M.b), __dmul_rn(__dmul_rn(P.q, cn->dtlin_old), M.b));
        }
        const double a = M.a, b = M.b, ab = __dmul_rn(a, b);
        const double* il2row = il2_all + min(g, nv - 1) * nzd;
        const double* e = e_all + (size_t)min(g, nv - 1) * 2 * W::NZE;  // this mode's E or D
        cplx* lfm = lf_s + (size_t)min(g, nv - 1) * 4 * nzd;  // this mode's lamF
        const cplx* lo = lo_all + (size_t)M.m * 4 * nzd;
        const cplx* lf = lf_all ? lf_all + (size_t)M.m * 4 * nzd : nullptr;
        // lamF of field f at stored index s: n1 E lamU' + lamF_out
        auto lam_F = [&](int f, int s) -> cplx {
            cplx r = cscale(ldc(lo + f * nzd + s), __dmul_rn(S.n1, e[(f >> 1) * W::NZE + s]));
            if (lf) r = cadd(r, ldc(lf + f * nzd + s));
            return r;
        };
        if (base != first) stage_block(base);
        // E of the block's modes, while the fields are on their way
        for (int i = tid; i < 2 * nv * nzd; i += nth) {
            const int q = i / nzd, s = i - q * nzd, m = base + (q >> 1);
            const double ky = __ldg(H.ky + m);
            const double kxe = __dadd_rn(kx_at(kx0[m], P.q, ts, ky), __dmul_rn(__dmul_rn(P.q, S.dt_lin), ky));
            e_all[q * W::NZE + s] = adj_e(P, S, kxe, ky, kz2val(kzval(s <= W::H ? s : s - nzd, P.kzL)), q & 1, H.integ);
        }
        cp_async_wait_all();
        __syncthreads();
        // ---- fourteen inverse transforms
#pragma unroll 1
        for (int task = warp; task < 14; task += warps) {
            cplx x[8];
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                const int s = rdead<W>(r) ? -1 : QLGPU_CHECK_STORED(sidx<W>(t, r), nzd, H.status);
                cplx v = mk(0.0, 0.0);
                if (s >= 0) {
                    const double c = kzc[t + T * r], kz2 = kz2val(c);
                    if (task < 4) {
                        v = cscale(stg[task * nzd + s], fac);  // R_u, R_zeta, R_b, R_eta
                    } else if (task < 9) {
                        const int f0 = (task == A_RBZ || task == A_RBY) ? 2 : 0;
                        const cplx g0 = stg[f0 * nzd + s], g1 = stg[(f0 + 1) * nzd + s];
                        const double sc = il2row[s] * fac;
                        const bool y = task >= A_RUY;
                        // y: (a b) u + i c z;  z: (a c) u - i b z
                        const double p = y ? ab : __dmul_rn(a, c), q = y ? c : -b;
                        v = mk(fma(p, g0.x, -q * g1.y), fma(p, g0.y, q * g1.x));
                        v = task == A_RIK ? imul(v, sc * c) : cscale(v, sc);
                    } else {
                        const int f = task == A_WB ? 2 : task == A_WZ ? 1 : task == A_WE ? 3 : 0;
                        v = lam_F(f, s);
                        if (task != A_WU2) {
                            if (M.valid) lfm[f * nzd + s] = v;  // kept for the spectral chain
                        } else {
                            const bool z0 = (M.kyi == 0 && s == 0);
                            const double lapF = __dadd_rn(-__dmul_rn(a, a), lap2val(b, kz2, z0));
                            v = cscale(v, (z0 && M.kxi == 0) ? 1.0 : __drcp_rn(lapF));
                        }
                    }
                }
                x[r] = v;
            }
            xform<W>(x, buf(task), tw, g, t);
#pragma unroll
            for (int r = 0; r < 8; ++r) buf(task)[32 * r + lane] = x[r];
        }
        if (base == first) {
            pdl_wait();  // the mean-field kernel of the stage
            for (int i = tid; i < 5 * NZ; i += nth) prof[i] = __ldcg(B.prof + i);
            pdl_next();
        }
        __syncthreads();
        // ---- pointwise adjoints as inputs of nine forward transforms.  Inputs 0-6 are held in
        // registers until every warp has read its own (and the profile adjoints are formed); then
        // every result has a buffer of its own: 0-3 and 6 theirs, 4 and 5 the two spare ones, and 7
        // and 8 transform in place of the R_bz and R_uz they are made of.
        auto res = [&](int k) { return buf(k == 4 ? A_X1 : k == 5 ? A_X0 : k == 7 ? A_RBZ : k == 8 ? A_RUZ : k); };
        const double *By = prof, *dBy = prof + NZ, *ddBy = prof + 2 * NZ, *px = prof + 3 * NZ, *py = prof + 4 * NZ;
        auto rd = [&](int i, int r) { return R[i * W::XW + 32 * r + lane]; };
        cplx x[8];
        if (warp < 7) {
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                const int z = t + T * r;
                const double bBy = b * By[z], adBy = a * dBy[z];
                const double mx = M.mult * px[z], my = M.mult * py[z];
                cplx o;
                switch (warp) {
                    case 0: o = cadd(cadd(imul(rd(A_WB, r), -bBy), imul(rd(A_WE, r), adBy)), cscale(rd(A_RBZ, r), mx)); break;
                    case 1: o = imul(rd(A_WE, r), -bBy); break;
                    case 2: o = csub(cadd(imul(rd(A_WZ, r), adBy), imul(rd(A_WS, r), -bBy)), cscale(rd(A_RUZ, r), mx)); break;
                    case 3: o = imul(rd(A_WZ, r), -bBy); break;
                    case 4:
                        o = csub(csub(cscale(rd(A_WE, r), -ddBy[z]), cscale(rd(A_RB, r), mx)), cscale(rd(A_RBY, r), my));
                        break;
                    case 5:
                        o = cadd(cadd(cscale(rd(A_WZ, r), ddBy[z]), cscale(rd(A_WU2, r), 2.0 * ab * dBy[z])),
                                 cadd(cscale(rd(A_RU, r), mx), cscale(rd(A_RUY, r), my)));
                        break;
                    default: o = cscale(rd(A_WE, r), -2.0 * dBy[z]); break;
                }
                x[r] = conjc(o);
            }
        } else if (warp == (warps > 9 ? 9 : 7) && M.valid) {
            // adjoint of the mean-field profiles: Re(conj(multiplier * R) W) per term
            auto re_cw = [](cplx p, cplx w) { return p.x * w.x + p.y * w.y; };   // Re(conj(p) w)
            auto re_icw = [](cplx p, cplx w) { return p.y * w.x - p.x * w.y; };  // Re(i conj(p) w)
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                const cplx Wb = rd(A_WB, r), Wz = rd(A_WZ, r), We = rd(A_WE, r), WS = rd(A_WS, r);
                const cplx Ru = rd(A_RU, r), Rb = rd(A_RB, r), Rbz = rd(A_RBZ, r);
                double* ac = acc + 32 * r + lane;
                ac[0] += -b * (re_icw(Ru, Wb) + re_icw(rd(A_RE, r), Wz) + re_icw(rd(A_RZ, r), We) + re_icw(Rb, WS));
                ac[256] += a * (re_icw(Rb, Wz) + re_icw(Ru, We)) - 2.0 * re_cw(rd(A_RIK, r), We) +
                           2.0 * ab * re_cw(Rbz, rd(A_WU2, r));
                ac[512] += re_cw(Rbz, Wz) - re_cw(rd(A_RUZ, r), We);
            }
        }
        __syncthreads();
        // with eight warps the one that formed the profile adjoints takes both of 7 and 8
#pragma unroll 1
        for (int k = warp; k < 9; k += warps > 8 ? warps : (warp == 7 ? 1 : 9)) {
            if (k >= 7) {  // 7: mult py R_bz, 8: -mult py R_uz
#pragma unroll
                for (int r = 0; r < 8; ++r) {
                    const double my = M.mult * py[t + T * r];
                    x[r] = conjc(k == 7 ? cscale(rd(A_RBZ, r), my) : cscale(rd(A_RUZ, r), -my));
                }
                __syncwarp();
            }
            cplx* xb = res(k);
            xform<W>(x, xb, tw, g, t);
#pragma unroll
            for (int r = 0; r < 8; ++r) xb[32 * r + lane] = conjc(x[r]);
        }
        __syncthreads();
        // ---- spectral chain to (u, zeta, b, eta), linear terms, RK adjoint: field f, half of the
        // registers per task
#pragma unroll 1
        for (int task = warp; task < 8; task += warps) {
            const int f = task >> 1, h = task & 1;
            if (!M.valid) continue;
            const size_t at = ((size_t)M.m * 4 + f) * nzd;
            cplx lov[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int s = sidx<W>(t, 4 * h + i);
                lov[i] = s >= 0 ? ldc(lo + f * nzd + s) : mk(0.0, 0.0);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int r = 4 * h + i;
                const int s = QLGPU_CHECK_STORED(sidx<W>(t, r), nzd, H.status);
                if (s < 0) continue;
                const int rl = 32 * r + lane;
                const double c = kzc[t + T * r], kz2 = kz2val(c);
                const bool z0 = (M.kyi == 0 && s == 0);
                const double il2 = il2row[s];
                const cplx mu = cscale(lov[i], e[(f >> 1) * W::NZE + s]);
                cplx v = mu;
                if (H.integ == INTEG_CN) {
                    // the direct term (1 + linC Lold) D lamU' (RK3CN.cpp:107)
                    const double lo_lap = M.old_init ? lap_init<MODEL_BQLIN>(P, M.kxo, lap2val(b, kz2, z0))
                                                     : lap_end<MODEL_BQLIN>(P, M.kxo, b, kz2);
                    v = cscale(mu, __dadd_rn(1.0, __dmul_rn(S.linC, linop_f<MODEL_BQLIN>(P, lo_lap, f))));
                }
                v = cadd(v, cscale(res(f)[rl], fac));
                // uz = (a c u - i b zeta) il2, i c uz, uy = (a b u + i c zeta) il2 (b, eta likewise)
                const cplx lz = f < 2 ? cscale(csub(res(4)[rl], imul(res(6)[rl], c)), fac) : cscale(res(5)[rl], fac);
                const cplx ly = cscale(res(f < 2 ? 7 : 8)[rl], fac);
                if (f == 0 || f == 2) {
                    v = cadd(v, cscale(lz, __dmul_rn(a, c) * il2));
                    v = cadd(v, cscale(ly, ab * il2));
                } else {
                    v = cadd(v, imul(lz, b * il2));
                    v = cadd(v, imul(ly, -c * il2));
                }
                if (f < 2) {
                    const double lapF = __dadd_rn(-__dmul_rn(a, a), lap2val(b, kz2, z0));
                    const double ilapF = (z0 && M.kxi == 0) ? 1.0 : __drcp_rn(lapF);
                    const cplx l0 = lfm[s];
                    if (f == 0) {
                        // linear terms of F_zeta ((q - 2 Omega) i c u) and F_u (ilapF 2 a b q u)
                        v = cadd(v, imul(lfm[nzd + s], -(P.q - Om2) * c));
                        v = cadd(v, cscale(l0, ilapF * 2.0 * ab * P.q));
                    } else {
                        v = cadd(v, imul(l0, -Om2 * c * ilapF));  // linear term of F_u: ilapF 2 Omega i c zeta
                    }
                } else if (f == 2) {
                    v = cadd(v, imul(lfm[3 * nzd + s], P.q * c));  // linear term of F_eta: -q i c b
                }
                if (X.s == 0 && X.n > 0) {
                    // this stage's input is the post-step state of step n - 1: the remap's adjoint (the
                    // fields of a remapped mode were set to zero, MHD_BQlin.cpp:319-329) and J's gradient
                    // there, d/db = 2 a b_y il2 b + i c il2 eta, d/deta = -i c il2 b (MHD_BQlin.cpp:388-392,424)
                    const bool remapped = B.kx_pre[(size_t)(X.n - 1) * P.nxy + M.m] != kx0[M.m];
                    const double w = H.weight * P.divfac * M.mult;
                    if (f == 2)
                        v = cadd(v, cscale(cadd(cscale(stg[2 * nzd + s], 2.0 * ab * il2),
                                                imul(stg[3 * nzd + s], c * il2)), w));
                    if (f == 3) v = cadd(v, cscale(imul(stg[2 * nzd + s], -c * il2), w));
                    if (remapped) v = mk(0.0, 0.0);
                }
                stc(lu_all + at + s, v);
                if (lp_all) stc(lp_all + at + s, cscale(mu, S.n2));
            }
        }
        __syncthreads();
    }
    // ---- the chunk's sum of the profile adjoints (modes of a block in order, then blocks)
    double* out = B.bpart + (size_t)blockIdx.x * 3 * NZ;
    for (int i = tid; i < 3 * NZ; i += nth) {
        const int e = i / NZ, z = i % NZ;
        double s = 0.0;
#pragma unroll
        for (int q = 0; q < GPW; ++q) s += acc[256 * e + 32 * (z / T) + q * T + z % T];
        out[i] = s;
    }
}

// Mean-field side of the adjoint, one CTA per seed.  post (the stage X just reversed):
// lamB_y += fac (T(pBy) - i c T(pdBy) - c^2 T(pddBy)), the adjoint of the stage's
// mean-field profiles (MHD_BQlin.cpp:122-127).  pre (the next stage Y): the forward
// profiles By, dBy, ddBy of its input and the RK / mean-field-rhs adjoint of B:
//   muB = E_B lamB', lamG = n1 muB + lamG_out, lamB = muB - q lamG_y e_x,
//   lamGp = n2 muB,  p(z) = Re sum_{s=1..H} h_s e^{+i k_s z},
//   h_s = rs_fac (-i kz_s) (lamEMF[s] + conj(lamEMF[nz-s])).
constexpr int ADJ_MF_THREADS = 512;

template <int NZ>
__global__ void __launch_bounds__(ADJ_MF_THREADS, 1)
    adj_mf_kernel(const __grid_constant__ AdjShared H, const __grid_constant__ DevParams P,
                  const __grid_constant__ AdjPos X, const __grid_constant__ AdjPos Y, int post, int pre) {
    using W = AG<NZ>;
    constexpr int T = W::T, nzd = W::nz;
    constexpr int SPLIT = NZ <= 128 ? 4 : 2;  // threads that share a sum over the chunks
    __shared__ __align__(16) cplx tw[NZ];
    __shared__ __align__(16) cplx xch[3][W::XW];
    __shared__ __align__(16) cplx lamB[2][nzd], lamG[2][nzd];
    __shared__ double tot[3 * NZ];
    __shared__ __align__(16) double psum[SPLIT][3 * NZ];  // then the spectra of the sums
    static_assert(SPLIT >= 2, "the spectra take two doubles per value");
    cplx(*spec)[NZ] = reinterpret_cast<cplx(*)[NZ]>(&psum[0][0]);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nth = blockDim.x;
    const int g = lane / T, t = lane % T;
    const AdjSeedBufs& B = H.seeds[blockIdx.y];
    const int pp = post ? X.par ^ 1 : Y.par;  // the buffers the pre part reads
    cplx* lamBg = B.lamB[pp];
    for (int i = tid; i < NZ; i += nth) tw[i] = ldc_cg(H.tw8 + i);
    for (int i = tid; i < 2 * nzd; i += nth) lamB[i / nzd][i % nzd] = ldc(lamBg + i);
    __syncthreads();
    // forward profiles of the next stage's input: warp w transforms profiles w GPW ... (they
    // do not depend on the stage being reversed)
    constexpr int PW = (3 + W::GPW - 1) / W::GPW;  // warps of the three profiles
    cplx x[8];
    const int arr = warp * W::GPW + g;
    if (pre && warp < PW) {
        const cplx* By = B.stB + (size_t)(3 * Y.n + Y.s) * H.nmfe + nzd;
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const int s = rdead<W>(r) ? -1 : sidx<W>(t, r);
            cplx v = mk(0.0, 0.0);
            if (s >= 0 && arr < 3) {
                const int k = t + T * r;
                const double c = kzval(k <= W::H ? k : k - NZ, P.kzL);
                v = cscale(ldc(By + s), P.fac);
                if (arr == 1) v = imul(v, c);
                if (arr == 2) v = cscale(v, kz2val(c));
            }
            x[r] = v;
        }
        xform<W>(x, xch[warp], tw, g, t);
    }
    pdl_wait();
    pdl_next();
    if (pre && warp < PW && arr < 3) {
#pragma unroll
        for (int r = 0; r < 8; ++r) B.prof[arr * NZ + t + T * r] = x[r].x;
    }
    if (post) {
        // chunk sums: SPLIT runs of consecutive chunks per value, each in order, then the runs
        const int len = (H.nchunk + SPLIT - 1) / SPLIT;
        for (int i = tid; i < 3 * NZ * SPLIT; i += nth) {
            const int j = i / (3 * NZ), idx = i - j * (3 * NZ);
            const int c0 = j * len, c1 = min(H.nchunk, c0 + len);
            double s = 0.0;
            for (int c = c0; c < c1; c += 16) {
                double v[16];
#pragma unroll
                for (int u = 0; u < 16; ++u) v[u] = c + u < c1 ? __ldcg(B.bpart + (size_t)(c + u) * 3 * NZ + idx) : 0.0;
#pragma unroll
                for (int u = 0; u < 16; ++u) s += v[u];
            }
            psum[j][idx] = s;
        }
        __syncthreads();
        for (int i = tid; i < 3 * NZ; i += nth) {
            double s = 0.0;
#pragma unroll
            for (int j = 0; j < SPLIT; ++j) s += psum[j][i];
            tot[i] = s;
        }
        __syncthreads();
        if (warp < PW) {
            cplx y[8];
#pragma unroll
            for (int r = 0; r < 8; ++r) y[r] = mk(arr < 3 ? tot[arr * NZ + t + T * r] : 0.0, 0.0);
            xform<W>(y, xch[warp], tw, g, t);
            if (arr < 3) {
#pragma unroll
                for (int r = 0; r < 8; ++r) spec[arr][t + T * r] = conjc(y[r]);
            }
        }
        __syncthreads();
        for (int s = tid; s < nzd; s += nth) {
            const int k = s <= W::H ? s : s + (NZ - nzd);
            const double c = kzval(s <= W::H ? s : s - nzd, P.kzL);
            const cplx v = cadd(cadd(spec[0][k], imul(spec[1][k], -c)), cscale(spec[2][k], kz2val(c)));
            lamB[1][s] = cadd(lamB[1][s], cscale(v, P.fac));
            stc(lamBg + nzd + s, lamB[1][s]);
        }
        __syncthreads();
    }
    if (!pre) return;
    const StageConst& S = Y.sc;
    const cplx* lamG_out = Y.s == 2 ? nullptr : B.lamG[Y.par];
    cplx* lamGp = Y.s == 0 ? nullptr : B.lamG[Y.par ^ 1];
    cplx* lamB_in = B.lamB[Y.par ^ 1];
    for (int s = tid; s < nzd; s += nth) {
        const double kz2 = kz2val(kzval(s <= W::H ? s : s - nzd, P.kzL));
        const double Lm = P.ql ? __dmul_rn(P.eta, kz2) : 0.0;
        // exp(linC Lm), or D = 1/(1 - linC Lm) and the direct term (1 + linC Lm) D for RK3CN
        const double e = H.integ == INTEG_CN ? __drcp_rn(__dsub_rn(1.0, __dmul_rn(S.linC, Lm)))
                                             : exp(__dmul_rn(S.linC, Lm));
        cplx nb[2];
#pragma unroll
        for (int m = 0; m < 2; ++m) {
            const cplx muB = cscale(lamB[m][s], e);
            cplx lg = cscale(muB, S.n1);
            if (lamG_out) lg = cadd(lg, ldc(lamG_out + m * nzd + s));
            lamG[m][s] = lg;
            if (lamGp) stc(lamGp + m * nzd + s, cscale(muB, S.n2));
            nb[m] = H.integ == INTEG_CN ? cscale(muB, __dadd_rn(1.0, __dmul_rn(S.linC, Lm))) : muB;
        }
        // G_By = -q Bx + EMF_y (MHD_BQlin.cpp:274-276)
        if (P.ql) nb[0] = csub(nb[0], cscale(lamG[1][s], P.q));
        stc(lamB_in + s, nb[0]);
        stc(lamB_in + nzd + s, nb[1]);
    }
    __syncthreads();
    constexpr int QW = (2 + W::GPW - 1) / W::GPW;  // warps of px, py
    if (warp < QW) {
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const int s = rdead<W>(r) ? -1 : sidx<W>(t, r);
            cplx v = mk(0.0, 0.0);
            if (P.ql && arr < 2 && s >= 1 && s <= W::H) {
                const double c = kzval(s, P.kzL);
                v = imul(cadd(lamG[arr][s], conjc(lamG[arr][nzd - s])), -c * P.rs_fac);
            }
            x[r] = v;
        }
        xform<W>(x, xch[warp], tw, g, t);
        if (arr < 2) {
#pragma unroll
            for (int r = 0; r < 8; ++r) B.prof[(3 + arr) * NZ + t + T * r] = x[r].x;
        }
    }
}

// The window's last step: J's gradient at the window's end state and the adjoint of the
// last step's remap (the other steps' are part of adj_modes_kernel).
__global__ void adj_jgrad_kernel(const __grid_constant__ AdjShared H, const __grid_constant__ DevParams P,
                                 const __grid_constant__ AdjPos X) {
    const AdjSeedBufs& B = H.seeds[blockIdx.y];
    const int nz = P.nz, HH = (nz - 1) / 2;
    const double t = B.t_pre[X.steps];
    const double* kx_before = B.kx_pre + (size_t)(X.steps - 1) * P.nxy;
    cplx* lamU = B.lamU[X.par];
    const size_t n = (size_t)P.nxy * nz;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const int mode = (int)(i / nz), s = (int)(i % nz);
        const double kyv = H.ky[mode];
        const double a = kx_at(B.kx_post[mode], P.q, t, kyv);
        const double ab = __dmul_rn(a, kyv);
        const double c = kzval(s <= HH ? s : s - nz, P.kzL);
        const double il2 = H.ilap2[(size_t)H.kyi[mode] * nz + s];
        const double w = H.weight * P.divfac * (kyv == 0.0 ? 1.0 : 2.0);
        const cplx* u = B.postU + (size_t)mode * 4 * nz;
        cplx* l = lamU + (size_t)mode * 4 * nz;
        if (kx_before[mode] != B.kx_post[mode]) {
            for (int f = 0; f < 4; ++f) l[f * nz + s] = mk(0.0, 0.0);
            continue;
        }
        const cplx bb = u[2 * nz + s], ee = u[3 * nz + s];
        const cplx gb = cadd(cscale(bb, 2.0 * ab * il2), imul(ee, c * il2));
        const cplx ge = imul(bb, -c * il2);
        l[2 * nz + s] = cadd(l[2 * nz + s], cscale(gb, w));
        l[3 * nz + s] = cadd(l[3 * nz + s], cscale(ge, w));
    }
}

}  // namespace qlgpu
