// qlgpu_wide.cuh -- one RK3 stage of the quasi-linear models with a mode's
// transforms side by side (sm_100a): MHD_BQlin and MHD_FullQlin, RK3CN_Elin and
// RK3CN, NZ = 16 ... 256.
//
// What bounds it.  A case of a few thousand modes gives an SM a handful of modes
// per stage, so a stage is latency: the chain of transforms one mode walks.  A
// pair of groups that took the mode's transforms one after another walked 5
// inverse and 4 forward transforms with the pointwise work between them, about
// 31 us whatever NZ is.  Here a mode's inverse transforms are independent tasks
// of the warps of a TEAM, and so are its forward transforms: two transforms
// deep, two team barriers, and code that is one loop over tasks around one
// transform instead of 9 unrolled steps (the instruction cache is cold at every
// launch).
//
// Team.  `tw` warps (any count) share one block of GPW = 32/T modes: a warp-task
// transforms one field of all GPW modes, group g of the warp (T = NZ/8 lanes,
// 8 points each) the field of mode g.  Every task uses the same (lane, register)
// map, index t + T r of mode g, in spectral and in real space, so a task's result
// lies in shared memory at [r][lane] and its readers use their own lane: no bank
// conflicts, no index math.
//
//   MHD_BQlin   (MHD_BQlin.cpp:135-257; 14 transforms, the reference does 22)
//     inverse   R_uz R_bz R_u R_b R_zeta R_eta R_{i kz uz} R_uy R_by
//     forward   i ky By R_b (S) and 2 kx ky dBy R_bz        -> u
//               i ky By R_zeta - i kx dBy R_u - 2 dBy R_{i kz uz} - ddBy R_uz -> eta
//               i ky By R_eta - i kx dBy R_b + ddBy R_bz     -> zeta
//               i ky By R_u                                  -> b
//     stress    Ex += Re(R_bz R_u* - R_uz R_b*), Ey += Re(R_bz R_uy* - R_uz R_by*)
//   MHD_FullQlin (MHD_FullQlin.cpp:209-381; 16 transforms, the reference does 32)
//     inverse   Ux Uy Uz Bx By Bz dzUx dzUy dzBx dzBy
//     forward   T1 T2 T3 S1 S2 S3 (formulas at fq_input)
//     stress    EMF x, y and the two velocity drives
//     update    u, zeta, b, eta from the six spectra (a third barrier)
//
// A CTA holds teams = max(1, warps / TS) teams (TS = 5 / 8: the forward tasks of
// a model), each with its own named barrier and its own blocks.  Partial sums of
// the stresses are lane-private in shared memory; per-CTA sums go through the
// fixed-order two-level reduction to the mean-field stage (reducer CTAs in
// run_kernel, else the CTA that arrives last), its loads issued before the sums
// are waited for and its transforms on the same 8-point layout.
//
// Against the pairs of groups, per step inside qlgpu_step: 16x16 x NZ=32 140 us -> 29,
// 64x64 x NZ=128 171 -> 85, 48x48 x NZ=64 of MHD_FullQlin 171 -> 43, 22x18 x NZ=256
// 176 -> 41 (issue 29 % and 15 warps per SM at 64x64, where it was 20 % and 8).
#pragma once
#include "qlgpu_debug.cuh"
#include "qlgpu_kernel.cuh"
#include "qlgpu_noise.cuh"
#include "qlgpu_stage.cuh"
#include "qlgpu_xform.cuh"

namespace qlgpu {
namespace wide {

// widest CTA: 3 teams of MHD_BQlin, 2 of MHD_FullQlin, at 128 registers a thread (4 teams of
// MHD_BQlin at 96 registers spill: 8 % slower at 64x64 x NZ=128)
template <int MODEL>
constexpr int MAX_WARPS = MODEL == MODEL_BQLIN ? 15 : 16;

// Geometry and shared-memory layout of one NZ class and model.
template <int NZ_, int MODEL>
struct WG {
    static constexpr int NZ = NZ_;
    static constexpr int T = NZ_ / 8;                  // lanes per group
    static constexpr int nz = 1 + 2 * (NZ_ / 3);       // Model.h:34
    static constexpr int H = (nz - 1) / 2;
    static constexpr int GPW = 32 / T;                 // modes per block
    static constexpr int SWZ = T == 4 ? 1 : (T == 2 ? 3 : 0);
    static constexpr bool BQ = MODEL == MODEL_BQLIN;
    static constexpr int TS = BQ ? 5 : 8;              // warps of a full team
    static constexpr int NINV = BQ ? 9 : 10;           // inverse tasks
    static constexpr int NX = BQ ? 0 : 6;              // further buffers: the forward tasks' results
    static constexpr int NE = BQ ? 2 : 4;              // stress profiles
    static constexpr int NPROF = BQ ? 3 : 8;           // real-space mean-field profiles
    static constexpr int PL = NE * NZ_ + 8;            // partial vector (doubles)
    static constexpr int NZE = (nz + 1) & ~1;
    static constexpr bool PAD = T >= 8;
    static constexpr int XW = PAD ? 8 * GPW * (T + 1) : 256;  // a result / exchange buffer (cplx)
    static constexpr size_t o_tw = 0;                                  // [8][T] cplx
    static constexpr size_t o_prof = o_tw + 16 * (size_t)NZ_;          // [NPROF][NZ]
    static constexpr size_t o_kz = o_prof + 8 * (size_t)NPROF * NZ_;   // kz per spectral slot
    static constexpr size_t o_ekz = o_kz + 8 * (size_t)NZ_;            // [2][NZE]
    static constexpr size_t o_dred = o_ekz + 16 * (size_t)NZE;         // [4 teams][6] diagnostic sums
    static constexpr size_t o_team = (o_dred + 8 * 6 * 4 + 15) & ~(size_t)15;
    // per team: results / exchange buffers [NINV + NX][XW] cplx, a result at [8][32], staged fields and
    // (MHD_BQlin: MHD_FullQlin reads them in its update, 4 % faster there) previous right-hand sides
    // [GPW][4][nz] cplx, 1/lap2 [GPW][nz], stress sums [NE][8][32]
    static constexpr size_t TM_STG = 16 * XW * (size_t)(NINV + NX);
    static constexpr size_t TM_FP = TM_STG + 16 * (size_t)GPW * 4 * nz;
    static constexpr size_t TM_IL2 = TM_FP + (BQ ? 16 * (size_t)GPW * 4 * nz : 0);
    static constexpr size_t TM_ACC = (TM_IL2 + 8 * (size_t)GPW * nz + 15) & ~(size_t)15;
    static constexpr size_t TEAM_BYTES = TM_ACC + 8 * 256 * (size_t)NE;
    // the mean-field stage's scratch overlays the teams' buffers
    static constexpr int NMF = BQ ? 2 : 4;             // mean fields
    static constexpr size_t TOP_BYTES = 8 * ((size_t)PL + 2) + 16 * (size_t)NE * (H + 1) + 16 * 2 * NMF * (size_t)nz;
    static_assert(TOP_BYTES + 16 * XW * 4 <= TEAM_BYTES, "mean-field scratch and its exchange buffers in a team's bytes");
    static constexpr size_t TOP_XCH = (TOP_BYTES + 15) & ~(size_t)15;  // four exchange buffers of the scratch
    // named barriers of team i: 1 + i the team, 5 + i its first inverse round, 9 + i its S spectrum
    __host__ __device__ static constexpr int teams(int warps) { return warps / TS > 1 ? warps / TS : 1; }
    __host__ __device__ static constexpr size_t bytes(int warps) {
        // MHD_BQlin teams of fewer than five warps run forward tasks one after another, which takes
        // three buffers more
        return o_team + TEAM_BYTES * (size_t)teams(warps) + (BQ && warps < TS ? 3 * 16 * XW : 0);
    }
};

__device__ __forceinline__ void team_sync(int id, int threads) {
    asm volatile("bar.sync %0, %1;\n" ::"r"(id), "r"(threads) : "memory");
}

__device__ __forceinline__ void team_arrive(int id, int threads) {
    asm volatile("bar.arrive %0, %1;\n" ::"r"(id), "r"(threads) : "memory");
}

// ---------------------------------------------------------------------------
// Mean-field side on the 8-point layout.  A warp transforms GPW profiles.
// ---------------------------------------------------------------------------
// Real-space profiles of the mean fields mf[][nz] (MHD_BQlin.cpp:122-127: By, dz
// By, dz^2 By; MHD_FullQlin.cpp:180-198: Bx, By, Ux, Uy and dz of each) into
// out[NPROF][NZ]; xg = the warp's exchange buffer.  mx (MAXIMA; null: off) takes the
// largest |profile|^2 of each mean field, what Calculate_CFL reads (MHD_BQlin.cpp:540-552,
// MHD_FullQlin.cpp:769-780); number NPROF of MHD_BQlin is Bx, for its maximum alone.  lo, hi:
// the profiles taken.  Ends without a barrier.
template <class W, bool BQ, bool MAXIMA = false, class Load>
__device__ __forceinline__ void mean_profiles8(const DevParams& P, Load&& mf, double* out, cplx* xg, const cplx* tw,
                                               int warp, int nwarps, int lane, double* mx = nullptr, int lo = 0,
                                               int hi = W::NPROF) {
    const int g = lane / W::T, t = lane % W::T;
    for (int base = lo + warp * W::GPW; base < hi; base += nwarps * W::GPW) {
        const int arr = base + g;
        const bool bx = MAXIMA && BQ && arr >= W::NPROF;
        const int src = BQ ? (bx ? 0 : 1) : arr / 2, deriv = BQ ? (bx ? 0 : arr) : arr % 2;
        cplx x[8];
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const int s = rdead<W>(r) ? -1 : sidx<W>(t, r);
            cplx v = mk(0.0, 0.0);
            if (s >= 0 && arr < hi) {
                v = cscale(mf(src, s), P.fac);
                const int k = t + W::T * r;
                const double c = kzval(k <= W::H ? k : k - W::NZ, P.kzL);
                if (deriv == 1) v = imul(v, c);
                if (deriv == 2) v = cscale(v, kz2val(c));
            }
            x[r] = v;
        }
        xform<W>(x, xg, tw, g, t);
        if (arr < hi && !bx) {
#pragma unroll
            for (int r = 0; r < 8; ++r) out[arr * W::NZ + t + W::T * r] = x[r].x;
        }
        if (MAXIMA && mx) {
            double v = 0.0;
#pragma unroll
            for (int r = 0; r < 8; ++r) v = fmax(v, x[r].x * x[r].x + x[r].y * x[r].y);
#pragma unroll
            for (int o = W::T / 2; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
            if (t == 0 && arr < hi && deriv == 0) mx[src] = v;
        }
    }
}

// The mean-field stage's scratch: tot[PL], spec, the mean fields and their previous
// right-hand side.  top_prefetch requests the latter two before the sums are read.
template <class W>
__device__ __forceinline__ cplx* top_mfs(double* tot) {
    return reinterpret_cast<cplx*>(tot + W::PL + (W::PL & 1) + 2 * W::NE * (W::H + 1));
}
template <class W>
__device__ __forceinline__ void top_prefetch(const StageArgs& A, double* tot) {
    cplx* mfs = top_mfs<W>(tot);
    constexpr int n = W::NMF * W::nz;
    const bool hp = A.sc.has_prev && !A.rhs_only;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        cp_async16(mfs + i, A.mf + i);
        if (hp) cp_async16(mfs + n + i, A.Fmf_prev + i);
    }
    cp_async_commit();
}

// Mean-field stage of the CTA that arrived last: tot[PL] holds the stress
// profiles summed over the modes and the diagnostic sums; emf (optional): the integrating
// factors exp(linC eta kz2), exp(linC nu kz2) [2][NZE] of the stage.  Ends with a barrier;
// what it wrote is published by the caller's release.  ONE: a reducer of run_kernel, which
// takes the mean field `only` and its stress, and has the new field in mfo.  Stress spectra
// (MHD_BQlin.cpp:228-240 after the sum over modes; the transform is linear), the
// mean-field update and clock (mean_field_update) and the next stage's profiles.
template <class W, int MODEL, int INTEG, bool ONE = false, bool MAXIMA = false>
__device__ __forceinline__ void top_stage(const StageArgs& A, const DevParams& P, double* tot, cplx* xch,
                                          const cplx* tw, const double* emf, double tclock, double t_new, bool last,
                                          bool diag_due, double* mx = nullptr, int only = -1, cplx* mfo = nullptr) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nwarps = blockDim.x >> 5;
    const int g = lane / W::T, t = lane % W::T;
    double* spec = tot + W::PL + (W::PL & 1);
    cplx* mfs = top_mfs<W>(tot);
    // at most four warps transform (their exchange buffers)
    constexpr int NP = !ONE ? W::NPROF : W::BQ ? 3 : 2;
    constexpr int NT = (NP + W::GPW - 1) / W::GPW < 4 ? (NP + W::GPW - 1) / W::GPW : 4;
    const int ntw = nwarps < NT ? nwarps : NT;
    cplx* xg = xch + (size_t)(warp < ntw ? warp : 0) * W::XW;
    if (warp < ntw) {
        for (int base = warp * W::GPW; base < (ONE ? 1 : W::NE); base += ntw * W::GPW) {
            const int e = !ONE ? base + g : g == 0 ? only : W::NE;
            cplx x[8];
#pragma unroll
            for (int r = 0; r < 8; ++r) x[r] = mk(e < W::NE ? tot[e * W::NZ + t + W::T * r] : 0.0, 0.0);
            xform<W>(x, xg, tw, g, t);
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                const int k = t + W::T * r;
                if (e < W::NE && k <= W::H) {
                    cplx v = cscale(conjc(x[r]), P.rs_fac);
                    if (MODEL == MODEL_BQLIN || e < 2) v = imul(v, kzval(k, P.kzL));  // times kz (z derivative)
                    spec[(e * (W::H + 1) + k) * 2 + 0] = v.x;
                    spec[(e * (W::H + 1) + k) * 2 + 1] = v.y;
                }
            }
        }
    }
    cp_async_wait_all();
    __syncthreads();
    mean_field_update<W, MODEL, INTEG, W::NE>(A, P, tot, spec, mfs, mfs + W::NMF * W::nz, emf, tclock, t_new, last,
                                              diag_due, ONE ? only : -1, ONE ? mfo : A.mf);
    // MHD_BQlin needs the profiles of By alone, the reducer of Bx at most its largest value
    const int lo = !ONE ? 0 : !W::BQ ? 2 * only : only == 1 ? 0 : W::NPROF;
    const int hi = !ONE ? W::NPROF : !W::BQ ? lo + 2 : only == 1 || (MAXIMA && mx) ? lo + (only == 1 ? 3 : 1) : lo;
    if (A.mfr_cache && !A.rhs_only && warp < ntw)
        mean_profiles8<W, W::BQ, MAXIMA>(
            P, [&](int m, int s) { return mfs[m * W::nz + s]; }, A.mfr_cache, xg, tw, warp, ntw, lane, mx, lo, hi);
    if (tid == 0 && A.mfr_cache && !A.rhs_only) A.clk->mfr_valid = 1;
    __syncthreads();
}

// ---------------------------------------------------------------------------
// Per-block constants of one lane: its mode's wavenumbers at the stage.
// ---------------------------------------------------------------------------
struct LaneMode {
    int m, kyi, kxi;
    bool valid, zero;
    double kx0, a, b, kxe, kxo, mult;
    // the mode's part of the integrating factor, exp(linC c (-kx^2 - ky^2)), of the fields this warp
    // updates: side 0 (u, zeta), 1 (b, eta); -1: not computed
    double em;
    int em_side;
    __device__ __forceinline__ double em_of(const StageArgs& A, const DevParams& P, int side) const {
        const double hxy = __dsub_rn(-__dmul_rn(kxe, kxe), __dmul_rn(b, b));
        return exp(A.sc.linC * (side ? P.cb : P.nu) * hxy);
    }
};

// The update of one field of a lane's mode: everything the stage arguments say about it, in
// registers (the arguments may lie in shared memory, where every global store would make the
// compiler read them again).
template <class W, int MODEL, int INTEG, bool RHS>
struct Put {
    cplx *out, *fo;        // new values (rhs-only: F), F of this stage (null: not kept)
    const cplx* fp;        // F of the previous stage (null: none), staged (BQ) or in global memory
    double* linop;         // rhs-only: the operator (may be null)
    const double* ekz;
    double n1, n2, em;
    int f;
    bool rhs_only, zero;
    __device__ __forceinline__ Put(const StageArgs& A, const DevParams& P, const LaneMode& M, int f_,
                                   const cplx* fps, const double* ekz_) {
        const size_t at = ((size_t)M.m * 4 + f_) * W::nz;
        f = f_;
        out = A.lin_out + at;
        fo = A.Fout ? A.Fout + at : nullptr;
        fp = fps ? fps + f_ * W::nz : nullptr;
        rhs_only = RHS && A.rhs_only;
        linop = rhs_only && A.linop_out ? A.linop_out + at : nullptr;
        ekz = ekz_ + (f_ < 2 ? 0 : W::NZE);
        n1 = A.sc.n1;
        n2 = A.sc.n2;
        zero = M.zero;
        em = 1.0;
        if (INTEG == INTEG_EXP && !rhs_only && (MODEL == MODEL_BQLIN || P.factored))
            em = M.em_side == f_ / 2 ? M.em : M.em_of(A, P, f_ / 2);
    }
    // (RK3CN_Elin.cpp:102-104 / RK3CN.cpp:105-107)
    __device__ __forceinline__ cplx value(const StageConst& S, const DevParams& P, const LaneMode& M, const CnOld& cn,
                                          int s, double c, cplx F, cplx uin, cplx fpv) const {
        const double kz2 = kz2val(c);
        if (INTEG == INTEG_EXP) {
            double e;
            if (MODEL == MODEL_BQLIN || P.factored) e = em * ekz[s];
            else e = exp(__dmul_rn(S.linC, linop_f<MODEL>(P, lap_end<MODEL>(P, M.kxe, M.b, kz2), f)));
            const cplx acc = fp ? cadd(cadd(cscale(F, n1), cscale(fpv, n2)), uin) : cadd(cscale(F, n1), uin);
            return cscale(acc, e);
        }
        const bool z0 = (M.kyi == 0 && s == 0);
        const double L = linop_f<MODEL>(P, lap_end<MODEL>(P, M.kxe, M.b, kz2), f);
        const double lo = cn.old_init ? lap_init<MODEL>(P, M.kxo, lap2val(M.b, kz2, z0))
                                      : lap_end<MODEL>(P, M.kxo, M.b, kz2);
        return rk_update(S, L, linop_f<MODEL>(P, lo, f), F, fpv, uin, fp != nullptr);
    }
    // store(s): F and the new value
    __device__ __forceinline__ void store(const StageArgs& A, const DevParams& P, const LaneMode& M, int s, double c,
                                          cplx F, cplx nv) const {
        s = QLGPU_CHECK_INDEX(s, W::nz, &A.clk->status);
        if (RHS && rhs_only) {
            stg(out + s, F);
            if (linop) linop[s] = linop_f<MODEL>(P, lap_end<MODEL>(P, M.kxe, M.b, kz2val(c)), f);
            return;
        }
        if (fo) stg(fo + s, F);
        stg(out + s, zero ? mk(0.0, 0.0) : nv);
    }
    static __device__ __forceinline__ void stg(cplx* p, cplx v) {
        __stcg(reinterpret_cast<double2*>(p), make_double2(v.x, v.y));
    }
};

// Spectral input of an inverse task for this lane's mode, scaled by 1/NZ:
// kind 0 the field, 1 z-component, 2 i kz z-component, 3 y-component
// (MHD_BQlin.cpp:143-146), 4 i kz field, 5 i kz y-component.
template <class W>
__device__ __forceinline__ void inv_input(cplx (&x)[8], const cplx* g0, const double* il2, int kind,
                                          double a, double b, double fac, const double* kzc, int t) {
    const cplx* g1 = g0 + W::nz;
    if (kind == 0 || kind == 4) {
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const int s = rdead<W>(r) ? -1 : sidx<W>(t, r);
            cplx v = mk(0.0, 0.0);
            if (s >= 0) {
                v = g0[s];
                v = kind == 0 ? cscale(v, fac) : imul(v, kzc[t + W::T * r] * fac);
            }
            x[r] = v;
        }
        return;
    }
    if (kind == 3 || kind == 5) {  // (a b) u + i c z
        const double ab = __dmul_rn(a, b);
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const int s = rdead<W>(r) ? -1 : sidx<W>(t, r);
            cplx v = mk(0.0, 0.0);
            if (s >= 0) {
                const double c = kzc[t + W::T * r], sc = il2[s] * fac;
                const cplx u = g0[s], z = g1[s];
                v = mk(fma(ab, u.x, -c * z.y), fma(ab, u.y, c * z.x));
                v = kind == 5 ? imul(v, sc * c) : cscale(v, sc);
            }
            x[r] = v;
        }
        return;
    }
#pragma unroll
    for (int r = 0; r < 8; ++r) {  // (a c) u - i b z
        const int s = rdead<W>(r) ? -1 : sidx<W>(t, r);
        cplx v = mk(0.0, 0.0);
        if (s >= 0) {
            const double c = kzc[t + W::T * r], sc = il2[s] * fac, p = __dmul_rn(a, c);
            const cplx u = g0[s], z = g1[s];
            v = mk(fma(p, u.x, b * z.y), fma(p, u.y, -b * z.x));
            v = kind == 2 ? imul(v, sc * c) : cscale(v, sc);
        }
        x[r] = v;
    }
}

// ---------------------------------------------------------------------------
// MHD_BQlin: result buffers and the forward / stress tasks of one block
// ---------------------------------------------------------------------------
enum { R_UZ = 0, R_BZ, R_U, R_B, R_ZE, R_ET, R_DUZ, R_UY, R_BY };

// Forward task 0: S = T(i ky By R_b), kept in its buffer, 1: T(2 kx ky dBy R_bz) -> u, 2: eta,
// 3: zeta, 4: b.  The input of a task, conjugated.
template <class W>
__device__ __forceinline__ void bq_input(cplx (&x)[8], const LaneMode& M, int task, const cplx* R, const double* prof,
                                         int lane, int t) {
    constexpr int T = W::T;
    const double *By = prof, *dBy = prof + W::NZ, *ddBy = prof + 2 * W::NZ;
    auto buf = [&](int i) { return R + i * W::XW; };
    const double a = M.a, b = M.b;
    if (task == 1) {
        const cplx* p = buf(R_BZ) + lane;
        const double ab2 = 2.0 * __dmul_rn(a, b);
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const cplx v = p[32 * r];
            const double w = ab2 * dBy[t + T * r];
            x[r] = mk(w * v.x, -w * v.y);  // conj(2 kx ky dBy R_bz)
        }
    } else if (task == 0 || task == 4) {
        const cplx* p = buf(task == 0 ? R_B : R_U) + lane;
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const cplx v = p[32 * r];
            const double y = -b * By[t + T * r];
            x[r] = mk(y * v.y, y * v.x);  // conj(i ky By R)
        }
    } else {
        // eta: i ky By R_zeta - i kx dBy R_u - 2 dBy R_{i kz uz} - ddBy R_uz (MHD_BQlin.cpp:189-198)
        // zeta: i ky By R_eta - i kx dBy R_b + ddBy R_bz (MHD_BQlin.cpp:170-178)
        const bool eta = task == 2;
        const cplx* p0 = buf(eta ? R_ZE : R_ET) + lane;
        const cplx* p1 = buf(eta ? R_U : R_B) + lane;
        const cplx* p2 = buf(eta ? R_UZ : R_BZ) + lane;
        const cplx* p3 = buf(R_DUZ) + lane;
        const double sg = eta ? -1.0 : 1.0;
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const int z = t + T * r;
            const cplx v0 = p0[32 * r], v1 = p1[32 * r], v2 = p2[32 * r];
            const double y = b * By[z], d = a * dBy[z], e = sg * ddBy[z];
            double re = fma(-y, v0.y, fma(d, v1.y, e * v2.x));
            double im = fma(y, v0.x, fma(-d, v1.x, e * v2.y));
            if (eta) {
                const cplx v3 = p3[32 * r];
                const double d2 = -2.0 * dBy[z];
                re = fma(d2, v3.x, re);
                im = fma(d2, v3.y, im);
            }
            x[r] = mk(re, -im);
        }
    }
}

// Transform of a task's input in exchange buffer xg and, but for S, the update of its field.
// wait_S() comes before task 1 reads S (in Sb), which another warp may have written.
template <class W, int INTEG, bool RHS, class WaitS>
__device__ __forceinline__ void bq_finish(cplx (&x)[8], const StageArgs& A, const DevParams& P, const LaneMode& M,
                                          const CnOld& cn, int task, cplx* xg, const cplx* Sb, const cplx* stg,
                                          const cplx* fps, const double* ekz, const double* kzc, const cplx* tw, int lane, int g, int t,
                                          WaitS&& wait_S) {
    constexpr int T = W::T, nzd = W::nz;
    const double a = M.a, b = M.b;
    xform<W>(x, xg, tw, g, t);
    if (task == 0) {
#pragma unroll
        for (int r = 0; r < 8; ++r) xg[32 * r + lane] = conjc(x[r]);
        return;
    }
    if (task == 1) wait_S();
    if (!M.valid) return;
    const int f = task == 1 ? 0 : task == 2 ? 3 : task == 3 ? 1 : 2;
    const Put<W, MODEL_BQLIN, INTEG, RHS> put(A, P, M, f, fps, ekz);
    const StageConst& S = A.sc;
    const double Om2 = __dmul_rn(2.0, P.Omega);
    const double cl = f == 3 ? -P.q : (f == 1 ? (P.q - Om2) : 0.0);
    const double rl = __dmul_rn(__dmul_rn(2.0, __dmul_rn(a, b)), P.q);
    const cplx* fin = stg + f * nzd;
    const cplx* l0 = stg + (f == 3 ? 2 : 0) * nzd;
    // four registers at a time: the values, then the stores
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        cplx nv[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = 4 * h + i;
            const int s = rdead<W>(r) ? -1 : sidx<W>(t, r);
            nv[i] = mk(0.0, 0.0);
            if (s < 0) continue;
            const double c = kzc[t + T * r];
            cplx F = conjc(x[r]);
            if (f == 0) {
                // S + ilapF ((2 kx ky q) u + 2 Omega i kz zeta + fwd(...)) (MHD_BQlin.cpp:162)
                const bool z0 = (M.kyi == 0 && s == 0);
                const double lapF = __dadd_rn(-__dmul_rn(a, a), lap2val(b, kz2val(c), z0));
                const double ilapF = (z0 && M.kxi == 0) ? 1.0 : __drcp_rn(lapF);
                const cplx lin = cadd(cadd(F, cscale(stg[s], rl)), imul(stg[nzd + s], Om2 * c));
                F = cadd(Sb[32 * r + lane], cscale(lin, ilapF));
            } else if (f != 2) {
                F = cadd(F, imul(l0[s], cl * c));  // MHD_BQlin.cpp:178,201
            }
            x[r] = F;
            nv[i] = put.value(S, P, M, cn, s, c, F, fin[s], put.fp ? put.fp[s] : mk(0.0, 0.0));
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = 4 * h + i;
            if (rdead<W>(r)) continue;
            const int s = sidx<W>(t, r);
            if (s >= 0) put.store(A, P, M, s, kzc[t + T * r], x[r], nv[i]);
        }
    }
}

// Stress sums, half 0: Ex (from R_uz, R_bz, R_u, R_b), half 1: Ey (MHD_BQlin.cpp:212-241)
template <class W>
__device__ __forceinline__ void bq_stress(const LaneMode& M, int half, const cplx* R, double* acc, int lane) {
    const cplx* p = R + W::XW * (half ? R_UY : R_U) + lane;
    const cplx* q = R + W::XW * (half ? R_BY : R_B) + lane;
    const cplx *pu = R + W::XW * R_UZ + lane, *pb = R + W::XW * R_BZ + lane;
    double* ax = acc + 256 * half + lane;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        const cplx uz = pu[32 * r], bz = pb[32 * r], u = p[32 * r], bb = q[32 * r];
        const double e = fma(bz.x, u.x, bz.y * u.y) - fma(uz.x, bb.x, uz.y * bb.y);
        ax[32 * r] = fma(M.mult, e, ax[32 * r]);
    }
}

// ---------------------------------------------------------------------------
// MHD_FullQlin.  With aU = i(kx MUx + ky MUy), aB = i(kx MBx + ky MBy)
// (MHD_FullQlin.cpp:271-299):
//   T1 = aU Ux + Uz dMUx - aB Bx - Bz dMBx    S1 = aU Bx + Uz dMBx - aB Ux - Bz dMUx
//   T2 = aU Uy + Uz dMUy - aB By - Bz dMBy    S2 = aU By + Uz dMBy - aB Uy - Bz dMUy
//   T3 = aU Uz - aB Bz                        S3 = aU Bz - aB Uz
// ---------------------------------------------------------------------------
enum { Q_UX = 0, Q_UY, Q_UZ, Q_BX, Q_BY, Q_BZ, Q_DUX, Q_DUY, Q_DBX, Q_DBY };

// conj of forward input n (0-2: T1..T3, 3-5: S1..S3)
template <class W>
__device__ __forceinline__ void fq_input(cplx (&x)[8], const LaneMode& M, int n, const cplx* R, const double* prof,
                                         int lane, int t) {
    constexpr int NZ = W::NZ;
    auto rd = [&](int i, int r) { return R[i * W::XW + 32 * r + lane]; };
    const int k = n % 3;
    const bool sside = n >= 3;
    const int own = sside ? Q_BX + k : Q_UX + k, oth = sside ? Q_UX + k : Q_BX + k;
    // dz profiles of the mean x (k = 0) or y (k = 1) components: prof = Bx, dBx, By, dBy, Ux, dUx, Uy, dUy
    const double* d1 = prof + (sside ? 1 + 2 * k : 5 + 2 * k) * NZ;
    const double* d2 = prof + (sside ? 5 + 2 * k : 1 + 2 * k) * NZ;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        const int z = t + W::T * r;
        const double aU = M.a * prof[4 * NZ + z] + M.b * prof[6 * NZ + z];  // times i
        const double aB = M.a * prof[z] + M.b * prof[2 * NZ + z];
        const cplx F = rd(own, r), G = rd(oth, r);
        cplx v = csub(imul(F, aU), imul(G, aB));
        if (k < 2) v = csub(cadd(v, cscale(rd(Q_UZ, r), d1[z])), cscale(rd(Q_BZ, r), d2[z]));
        x[r] = conjc(v);
    }
}

// Stress sums: half 0 the EMFs and the x drive of u, half 1 the rest (MHD_FullQlin.cpp:314-362)
template <class W>
__device__ __forceinline__ void fq_stress(const LaneMode& M, int half, const cplx* R, double* acc, int lane) {
    auto rd = [&](int i, int r) { return R[i * W::XW + 32 * r + lane]; };
    auto rc = [](cplx p, cplx q) { return p.x * q.x + p.y * q.y; };  // Re(p conj q)
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        double* ax = acc + 32 * r + lane;
        const cplx Ux = rd(Q_UX, r), Uy = rd(Q_UY, r), Uz = rd(Q_UZ, r);
        const cplx Bx = rd(Q_BX, r), By = rd(Q_BY, r), Bz = rd(Q_BZ, r);
        if (half == 0) {
            // EMF x (:322) and the x drive (:342-343): Re(Fx (i kx Fx)*) + Re(Fy (i ky Fx)*) + Re(Fz (dz Fx)*)
            const double ex = rc(Bz, Ux) - rc(Uz, Bx);
            const double du = rc(Ux, imul(Ux, M.a)) + rc(Uy, imul(Ux, M.b)) + rc(Uz, rd(Q_DUX, r));
            const double db = rc(Bx, imul(Bx, M.a)) + rc(By, imul(Bx, M.b)) + rc(Bz, rd(Q_DBX, r));
            ax[0] = fma(M.mult, ex, ax[0]);
            ax[512] = fma(M.mult, db - du, ax[512]);
        } else {
            // EMF y (:330) and the y drive (:357-358)
            const double ey = rc(Bz, Uy) - rc(Uz, By);
            const double du = rc(Ux, imul(Uy, M.a)) + rc(Uy, imul(Uy, M.b)) + rc(Uz, rd(Q_DUY, r));
            const double db = rc(Bx, imul(By, M.a)) + rc(By, imul(By, M.b)) + rc(Bz, rd(Q_DBY, r));
            ax[256] = fma(M.mult, ey, ax[256]);
            ax[768] = fma(M.mult, db - du, ax[768]);
        }
    }
}

// Update of field f from the six spectra in X[n][r][lane] (MHD_FullQlin.cpp:283-305)
template <class W, int INTEG, bool RHS>
__device__ __forceinline__ void fq_update(const StageArgs& A, const DevParams& P, const LaneMode& M, const CnOld& cn,
                                          int f, const cplx* X, const cplx* stg, const cplx* fps, const double* ekz,
                                          const double* kzc, int lane, int t) {
    constexpr int nzd = W::nz;
    if (!M.valid) return;
    const StageConst& S = A.sc;
    const double a = M.a, b = M.b, ab = __dmul_rn(a, b), Om2 = __dmul_rn(2.0, P.Omega);
    const Put<W, MODEL_FULLQLIN, INTEG, RHS> put(A, P, M, f, fps, ekz);
    auto X_ = [&](int n, int r) { return X[n * W::XW + 32 * r + lane]; };
    cplx fpv[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        const int s = rdead<W>(r) ? -1 : sidx<W>(t, r);
        fpv[r] = (put.fp && s >= 0) ? ldc(put.fp + s) : mk(0.0, 0.0);
    }
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        if (rdead<W>(r)) continue;
        const int s = sidx<W>(t, r);
        if (s < 0) continue;
        const double c = kzc[t + W::T * r];
        cplx F, uin;
        if (f == 0) {
            const cplx u0 = stg[s], ze = stg[nzd + s], t1 = X_(0, r), t2 = X_(1, r), t3 = X_(2, r);
            const bool z0 = (M.kyi == 0 && s == 0);
            const double lapF = __dadd_rn(-__dmul_rn(a, a), lap2val(b, kz2val(c), z0));
            const double ilapF = (z0 && M.kxi == 0) ? 1.0 : __drcp_rn(lapF);
            // (2 kx ky q) u + 2 Om i kz zeta - kx^2 t1 - kx ky t2 - kx kz t3
            cplx inner = cadd(cscale(u0, __dmul_rn(__dmul_rn(2.0, ab), P.q)), imul(ze, Om2 * c));
            inner = csub(inner, cadd(cadd(cscale(t1, a * a), cscale(t2, ab)), cscale(t3, a * c)));
            F = csub(cadd(cscale(inner, ilapF), imul(stg[2 * nzd + s], P.B0z * c)), t1);
            uin = u0;
        } else if (f == 1) {
            // (q - 2 Om) kz u + B0z kz eta - (kz t2 - ky t3)
            F = csub(cadd(imul(stg[s], (P.q - Om2) * c), imul(stg[3 * nzd + s], P.B0z * c)),
                     csub(imul(X_(1, r), c), imul(X_(2, r), b)));
            uin = stg[nzd + s];
        } else if (f == 2) {
            F = csub(imul(stg[s], P.B0z * c), X_(3, r));  // B0z kz u - s1
            uin = stg[2 * nzd + s];
        } else {
            // -q kz b + B0z kz zeta - (kz s2 - ky s3)
            uin = stg[3 * nzd + s];
            F = csub(cadd(imul(stg[2 * nzd + s], -P.q * c), imul(stg[nzd + s], P.B0z * c)),
                     csub(imul(X_(4, r), c), imul(X_(5, r), b)));
        }
        put.store(A, P, M, s, c, F, put.value(S, P, M, cn, s, c, F, uin, fpv[r]));
    }
}

// Per-mode diagnostic sums of one side (0 velocity, 1 magnetic) from the new
// state just stored (MHD_BQlin.cpp:365-407): energy, stress, dissipation.
template <class W>
__device__ __forceinline__ void side_diag(const DevParams& P, const LaneMode& M, int side, const cplx* uo,
                                          double t_new, const double* kzc, int t, double (&v)[3]) {
    const double an = kx_at(M.kx0, P.q, t_new, M.b);
    const double ab = __dmul_rn(an, M.b);
    const double md = M.b == 0.0 ? 1.0 : 2.0;
    const double vis = side ? P.eta : P.nu;
    const cplx* f0 = uo + (size_t)(2 * side) * W::nz;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        if (rdead<W>(r)) continue;
        const int s = sidx<W>(t, r);
        if (s < 0) continue;
        const double c = kzc[t + W::T * r];
        const bool z0 = (M.kyi == 0 && s == 0);
        const double lap2 = lap2val(M.b, kz2val(c), z0);
        const double il2 = ilap2val(lap2, z0);
        const double lapF = __dadd_rn(-__dmul_rn(an, an), lap2);
        const double l2 = __dmul_rn(lapF, il2);
        const cplx p = ldc(f0 + s), q = ldc(f0 + W::nz + s);
        const double e = l2 * (p.x * p.x + p.y * p.y) - il2 * (q.x * q.x + q.y * q.y);
        const cplx y = cscale(cadd(cscale(p, ab), imul(q, c)), il2);  // (MHD_BQlin.cpp:388-392)
        v[0] += md * e;
        v[1] += md * (p.x * y.x + p.y * y.y);
        v[2] += md * vis * (-lapF * e);
    }
}

}  // namespace wide

// Static shared words of a stage: the last-arriver flag, the gate's answer and, in a reducer of
// run_kernel, that of its wait for the workers (a word of its own: slower warps may still read the other).
struct StageShared {
    int last, ok;
    int arrived, pad;
};

// A case's clock as this CTA follows it through a launch: every CTA advances its own
// copy by the same operations the mean-field stage applies to DevClock, so only the
// mean-field profiles have to come from the CTA that ran the mean-field stage.
struct LocalClock {
    double t, timevar, t_old, dtlin_old;
    unsigned long long nstep;
    int old_init, mfr_valid;
    // forced steps: records after every `every` steps (0: none), step counter, limit of records
    int every, step, max_rec;
};
__device__ __forceinline__ void load_clock(LocalClock& lc, const DevClock* c) {
    lc.t = __ldcg(&c->t);
    lc.timevar = __ldcg(&c->timevar);
    lc.t_old = __ldcg(&c->t_old);
    lc.dtlin_old = __ldcg(&c->dtlin_old);
    lc.nstep = __ldcg(&c->nstep);
    lc.old_init = __ldcg(&c->old_init);
    lc.mfr_valid = __ldcg(&c->mfr_valid);
}

// The clock after stage S of a step that started at tclock (what mean_field_update does to DevClock).
template <bool FORCED>
__device__ __forceinline__ void advance_clock(LocalClock& lc, const StageConst& S, const DevParams& P, bool last,
                                              bool diag_due) {
    lc.t_old = S.abs_time ? S.t_off : __dadd_rn(lc.t, S.t_off);
    lc.dtlin_old = S.dt_lin;
    lc.old_init = 0;
    lc.mfr_valid = 1;
    if (!last) return;
    const double dt = FORCED ? S.dt : P.dt;
    lc.t = __dadd_rn(lc.t, dt);
    lc.timevar = __dadd_rn(lc.timevar, dt);
    if (diag_due) lc.timevar = __dsub_rn(lc.timevar, P.tv_interval);
    lc.nstep += 1;
    if (FORCED) lc.step += 1;
}
// A record is due at the end of this stage (main.cpp:117,127-130).
template <bool FORCED>
__device__ __forceinline__ bool record_due(const LocalClock& lc, const DevParams& P, double dt, bool last) {
    if (FORCED) {
        if (lc.every <= 0) return false;
        const int n = (lc.step + 1) / lc.every;
        return last && n * lc.every == lc.step + 1 && n <= lc.max_rec;
    }
    return last && P.tv_interval > 0.0 && __dsub_rn(__dadd_rn(lc.timevar, dt), P.tv_interval) > -1e-8;
}

enum StageResult { STAGE_DONE = 0, STAGE_TOP = 1, STAGE_ABORT = 2 };

// One stage over the modes of one case, executed by one CTA that is number
// `cta` of the `ncta` CTAs working on that case.  STAGE_TOP in the one CTA that
// arrived last and ran the mean-field stage; every other CTA returns STAGE_DONE
// as soon as its partial sums are published.
//
// A team steps the same blocks in every stage, so a stage's fields, previous
// right-hand sides and kx0 come from the CTA's own last stage: only the mean-field
// profiles wait for the other CTAs.  The first block's inverse transforms therefore
// run before gate(lane) (called by the first warp; false ends the launch), which in a
// persistent launch waits for the case's previous stage.  fresh: the shared-memory
// tables do not hold this case's yet.  REDUCER: the launch has CTAs of their own for the
// mean-field side (reduce_stage); this one only counts itself in at their `arrive`.  RHS: the
// launch may ask for the right-hand side instead of the update (A.rhs_only).  FORCED: driving
// noise and records by step count (run_kernel; work items have the noise alone).
template <int NZ, int MODEL, int INTEG, bool REDUCER, bool RHS, bool FORCED, class Gate>
__device__ __forceinline__ StageResult stage_body(const StageArgs& A, const DevParams& P, const int cta,
                                                  const int ncta, unsigned char* smem_raw, StageShared& ss,
                                                  LocalClock& lc, const bool fresh, unsigned* arrive,
                                                  Gate&& gate) {
    using namespace wide;
    using W = WG<NZ, MODEL>;
    constexpr int T = W::T, nzd = W::nz, GPW = W::GPW;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, warps = blockDim.x >> 5;
    const int g = lane / T, t = lane % T;
    const StageConst& S = A.sc;
    cplx* tw = reinterpret_cast<cplx*>(smem_raw + W::o_tw);
    double* prof = reinterpret_cast<double*>(smem_raw + W::o_prof);
    double* kzc = reinterpret_cast<double*>(smem_raw + W::o_kz);
    double* ekz = reinterpret_cast<double*>(smem_raw + W::o_ekz);
    double* dred = reinterpret_cast<double*>(smem_raw + W::o_dred);
    const int nteams = W::teams(warps), tws = warps / nteams;  // teams, warps per team
    const int team = warp / tws, wt = warp - team * tws;
    const bool in_team = team < nteams;
    unsigned char* tbase = smem_raw + W::o_team + W::TEAM_BYTES * (size_t)(in_team ? team : 0);
    cplx* R = reinterpret_cast<cplx*>(tbase);
    cplx* stg_all = reinterpret_cast<cplx*>(tbase + W::TM_STG);
    cplx* fp_all = reinterpret_cast<cplx*>(tbase + W::TM_FP);
    double* il2_all = reinterpret_cast<double*>(tbase + W::TM_IL2);
    double* acc = reinterpret_cast<double*>(tbase + W::TM_ACC);
    const int bar = 1 + team, bthreads = 32 * tws;
    const bool tr = A.trace && cta == 0 && tid == 0;
    if (tr) A.trace[0] = gtimer();

    // ---- first block's fields requested, then the tables and the cleared sums
    const int step = ncta * nteams * GPW;
    // block b: CTA b mod ncta, so that a last, partial round leaves one team per SM, not full and idle CTAs
    const int first = (team * ncta + cta) * GPW;
    const bool has_prev = A.Fprev && S.has_prev;
    // a block's fields and 1/lap2
    auto stage_block = [&](int base) {
        const int nm = min(GPW, P.nxy - base), n = nm * 4 * nzd;
        const size_t at = (size_t)base * 4 * nzd;
        for (int i = wt * 32 + lane; i < n; i += bthreads) cp_async16(stg_all + i, A.lin_in + at + i);
        // a team of one block keeps its 1/lap2 from stage to stage
        for (int i = wt * 32 + lane; (fresh || first + step < P.nxy) && i < nm * nzd; i += bthreads)
            cp_async8(il2_all + i, A.ilap2 + (size_t)__ldg(A.kyi + base + i / nzd) * nzd + i % nzd);
        cp_async_commit();
    };
    if (in_team && first < P.nxy) stage_block(first);
    const double tclock = lc.t;
    const CnOld cn{lc.t_old, lc.dtlin_old, lc.old_init};
    const bool cached = A.mfr_cache && !A.rhs_only && lc.mfr_valid;
    if (fresh)
        for (int i = tid; i < NZ; i += blockDim.x) {
            tw[i] = ldc_cg(A.tw + i);
            kzc[i] = kzval(i <= W::H ? i : i - NZ, P.kzL);
        }
    if (INTEG == INTEG_EXP) {
        // factored integrating factor: exp(linC c kz2) per stored kz
        for (int s = tid; s < nzd; s += blockDim.x) {
            if (A.ekz_tab) {
                ekz[s] = __ldg(A.ekz_tab + s);
                ekz[W::NZE + s] = __ldg(A.ekz_tab + nzd + s);
            } else {
                const double kz2 = kz2val(kzval(s <= W::H ? s : s - nzd, P.kzL));
                ekz[s] = exp(S.linC * P.nu * kz2);
                ekz[W::NZE + s] = exp(S.linC * P.cb * kz2);
            }
        }
    }
    if (in_team)
        for (int i = wt * 32 + lane; i < 256 * W::NE; i += bthreads) acc[i] = 0.0;
    for (int i = tid; i < 6 * 4; i += blockDim.x) dred[i] = 0.0;
    if (fresh) __syncthreads();
    if (!cached) {
        // a launch's first stage (the gate does not wait then); scratch: the first team's buffers
        const int nw = warps < 8 ? warps : 8;
        if (warp < nw)
            mean_profiles8<W, W::BQ>(
                P, [&](int m, int s) { return ldc_cg(A.mf + m * nzd + s); }, prof,
                reinterpret_cast<cplx*>(smem_raw + W::o_team) + W::XW * warp, tw, warp, nw, lane);
        __syncthreads();
    }
    if (tr) A.trace[1] = gtimer();

    // Last-stage bookkeeping identical in every CTA (main.cpp:111-130)
    const double t_new = __dadd_rn(tclock, FORCED ? S.dt : P.dt);
    const bool last = S.last && !A.rhs_only;
    const bool diag_due = record_due<FORCED>(lc, P, FORCED ? S.dt : P.dt, last);
    const double qt = __dmul_rn(P.q, t_new);
    const double ts = S.abs_time ? S.t_off : __dadd_rn(tclock, S.t_off);

    // ---- the team's blocks of GPW modes
    for (int base = first;; base += step) {
        const bool active = in_team && base < P.nxy;
        if (!active && base != first) break;
        const int nv = active ? min(GPW, P.nxy - base) : 1;
        LaneMode M;
        M.valid = active && g < nv;
        M.m = QLGPU_CHECK_INDEX(active ? base + min(g, nv - 1) : 0, P.nxy, &A.clk->status);
        const cplx* stg = stg_all + (size_t)min(g, nv - 1) * 4 * nzd;
        const cplx* fps = !has_prev ? nullptr
                        : W::BQ ? fp_all + (size_t)min(g, nv - 1) * 4 * nzd : A.Fprev + (size_t)M.m * 4 * nzd;
        const double* il2 = il2_all + min(g, nv - 1) * nzd;
        M.b = __ldg(A.ky + M.m);
        M.kx0 = __ldcg(A.kx0 + M.m);
        M.kyi = __ldg(A.kyi + M.m);
        M.kxi = __ldg(A.kxi + M.m);
        M.a = kx_at(M.kx0, P.q, ts, M.b);  // kx(t_s), MHD_BQlin.cpp:498
        M.mult = M.valid ? (M.b == 0.0 ? 1.0 : 2.0) : 0.0;
        M.kxe = __dadd_rn(M.a, __dmul_rn(__dmul_rn(P.q, S.dt_lin), M.b));  // MHD_BQlin.cpp:248
        M.kxo = M.em = 0.0;
        M.em_side = -1;
        if (INTEG == INTEG_CN) {
            if (cn.old_init) M.kxo = kx_at(M.kx0, P.q, tclock, M.b);
            else M.kxo = __dadd_rn(kx_at(M.kx0, P.q, cn.t_old, M.b), __dmul_rn(__dmul_rn(P.q, cn.dtlin_old), M.b));
        }
        // ShearingBox_Remap(q t) after t += dt (main.cpp:122-123, MHD_BQlin.cpp:319-329)
        M.zero = last && P.remap && __dadd_rn(M.kx0, __dmul_rn(qt, M.b)) > P.remap_thresh;
        if (active) {
            if (base != first) stage_block(base);
            if (wt == 0 && lane == 0) {
                // the next block's fields and previous rhs into L2
                const size_t nb = (size_t)base + step;
                if (nb < (size_t)P.nxy) {
                    const unsigned bytes = 64u * nzd * (unsigned)min(GPW, P.nxy - (int)nb);
                    l2_prefetch(A.lin_in + nb * 4 * nzd, bytes);
                    if (has_prev) l2_prefetch(A.Fprev + nb * 4 * nzd, bytes);
                }
            }
            // computed while the block's fields are on their way
            M.em_side = W::BQ ? (wt == 1 || wt == 3 ? 0 : 1) : (wt < 2 ? 0 : 1);
            if (INTEG == INTEG_EXP && !A.rhs_only && (W::BQ || P.factored) && wt < (W::BQ ? 5 : 4)) M.em = M.em_of(A, P, M.em_side);
            else M.em_side = -1;
            cp_async_wait_all();
            team_sync(bar, bthreads);
            // its previous right-hand sides, on their way under the inverse transforms
            if (W::BQ && has_prev) {
                for (int i = wt * 32 + lane; i < nv * 4 * nzd; i += bthreads)
                    cp_async16(fp_all + i, A.Fprev + (size_t)base * 4 * nzd + i);
                cp_async_commit();
            }
            if (A.rec_lin) {  // record the block's input fields
                cplx* dst = A.rec_lin + (size_t)base * 4 * nzd;
                for (int i = wt * 32 + lane; i < nv * 4 * nzd; i += bthreads) dst[i] = stg_all[i];
            }
            // ---- inverse transforms
#pragma unroll 1
            for (int task = wt; task < W::NINV; task += tws) {
                int kind, side;
                if (W::BQ) {
                    side = (task == R_BZ || task == R_B || task == R_ET || task == R_BY);
                    kind = (task == R_UZ || task == R_BZ) ? 1 : task == R_DUZ ? 2
                         : (task == R_UY || task == R_BY) ? 3 : 0;
                } else {
                    side = (task >= Q_BX && task <= Q_BZ) || task >= Q_DBX;
                    kind = (task == Q_UX || task == Q_BX) ? 0 : (task == Q_UY || task == Q_BY) ? 3
                         : (task == Q_UZ || task == Q_BZ) ? 1 : (task == Q_DUX || task == Q_DBX) ? 4 : 5;
                }
                const int f0 = 2 * side + (W::BQ && (task == R_ZE || task == R_ET) ? 1 : 0);
                cplx x[8];
                inv_input<W>(x, stg + f0 * nzd, il2, kind, M.a, M.b, P.fac, kzc, t);
                cplx* xb = R + task * W::XW;
                xform<W>(x, xb, tw, g, t);
#pragma unroll
                for (int r = 0; r < 8; ++r) xb[32 * r + lane] = x[r];
                // a team of five: its last warp has one task less and takes the Ex sums meanwhile,
                // once R_uz, R_bz, R_u, R_b of the others' first round are there
                if (W::BQ && tws == 5) {
                    if (wt == 4) {
                        team_sync(bar + 4, 160);
                        bq_stress<W>(M, 0, R, acc, lane);
                    } else if (task < 4) {
                        team_arrive(bar + 4, 160);
                    }
                }
            }
        }
        cp_async_wait_all();
        if (base == first) {
            // ---- the mean field of this stage
            if (warp == 0) {
                const int ok = __all_sync(0xffffffffu, gate(lane));
                if (lane == 0) ss.ok = ok;
            }
            __syncthreads();
            if (!ss.ok) return STAGE_ABORT;
            if (tr) A.trace[6] = gtimer();
            if (cached)
                for (int i = tid; i < W::NPROF * NZ; i += blockDim.x) prof[i] = __ldcg(A.mfr_cache + i);
            // optional record of the stage input (the adjoint's window recompute): CTA 0 of the case
            // copies the mean fields and, in a step's first stage, kx0 and the clock
            if (A.rec_mf && cta == 0) {
                for (int i = tid; i < P.nmf * nzd; i += blockDim.x) A.rec_mf[i] = ldc(A.mf + i);
                if (A.rec_kx)
                    for (int i = tid; i < P.nxy; i += blockDim.x) A.rec_kx[i] = __ldcg(A.kx0 + i);
                if (A.rec_t && tid == 0) A.rec_t[0] = tclock;
                if (A.rec_cn && tid == 0) {
                    A.rec_cn->t_old = cn.t_old;
                    A.rec_cn->dtlin_old = cn.dtlin_old;
                    A.rec_cn->old_init = cn.old_init;
                }
            }
            __syncthreads();
            if (tr) A.trace[7] = gtimer();
            if (!active) break;
        } else {
            team_sync(bar, bthreads);
        }
        // ---- products, forward transforms, stresses
        if constexpr (W::BQ) {
            auto buf = [&](int i) { return R + i * W::XW; };
            cplx x[8];
            if (tws >= 5) {
                // one forward task per warp.  Once all inputs (and the Ex sums) are read, the buffers of
                // R_b, R_{i kz uz}, R_zeta, R_eta, R_u are the tasks' exchange buffers; S -> u is a
                // hand-over between two warps, so that no warp has two transforms
                if (wt < 5) bq_input<W>(x, M, wt, R, prof, lane, t);
                else if (wt == 5) bq_stress<W>(M, 0, R, acc, lane);
                team_sync(bar, bthreads);
                if (wt < 5) {
                    cplx* xg = buf(wt == 0 ? R_B : wt == 1 ? R_DUZ : wt == 2 ? R_ZE : wt == 3 ? R_ET : R_U);
                    bq_finish<W, INTEG, RHS>(x, A, P, M, cn, wt, xg, buf(R_B), stg, fps, ekz, kzc, tw, lane, g, t,
                                        [&] { team_sync(bar + 8, 64); });
                }
                if (wt == 0) team_arrive(bar + 8, 64);
                if (wt == (tws == 5 ? 0 : 5)) bq_stress<W>(M, 1, R, acc, lane);
            } else {
                // S and u by warp 0, the others' fields and the stresses by the warps in turn; exchange
                // buffers that no other task still reads (R_zeta and R_eta have one reader each)
                cplx* more = reinterpret_cast<cplx*>(tbase + W::TEAM_BYTES);
#pragma unroll 1
                for (int task = 0; task < 7; ++task) {
                    if ((task < 2 ? 0 : (task - 1) % tws) != wt) continue;
                    if (task >= 5) {
                        bq_stress<W>(M, task - 5, R, acc, lane);
                        continue;
                    }
                    bq_input<W>(x, M, task, R, prof, lane, t);
                    __syncwarp();
                    cplx* xg = task == 2 ? buf(R_ZE) : task == 3 ? buf(R_ET) : more + W::XW * (task == 4 ? 2 : task);
                    bq_finish<W, INTEG, RHS>(x, A, P, M, cn, task, xg, more, stg, fps, ekz, kzc, tw, lane, g, t, [] {});
                }
            }
        } else {
#pragma unroll 1
            for (int task = wt; task < 8; task += tws) {
                if (task >= 6) {
                    fq_stress<W>(M, task - 6, R, acc, lane);
                    continue;
                }
                cplx x[8];
                fq_input<W>(x, M, task, R, prof, lane, t);
                cplx* xb = R + (W::NINV + task) * W::XW;
                xform<W>(x, xb, tw, g, t);
#pragma unroll
                for (int r = 0; r < 8; ++r) xb[32 * r + lane] = conjc(x[r]);
            }
            team_sync(bar, bthreads);
#pragma unroll 1
            for (int f = wt; f < 4; f += tws)
                fq_update<W, INTEG, RHS>(A, P, M, cn, f, R + W::NINV * W::XW, stg, fps, ekz, kzc, lane, t);
        }
        team_sync(bar, bthreads);  // the block's stores are done; its buffers are free
        if (last) {
            if (M.zero && M.valid && wt == 0 && t == 0) A.kx0[M.m] = __dsub_rn(M.kx0, P.remap_shift);
            cplx* uo = A.lin_out + (size_t)M.m * 4 * nzd;
            if ((FORCED || (!REDUCER && !RHS)) && A.noise) {
                // Model::DrivingNoise after the step (main.cpp:111-113), before the diagnostics see it
                if (M.valid && !M.zero)
                    noise_mode(A.noise, lc.nstep, uo, nzd, wt * T + t, tws * T, M.m, M.kx0, M.b, M.kxi, M.kyi, P.q,
                               tclock, P.kzL);
                team_sync(bar, bthreads);
            }
            if (diag_due) {
                for (int side = wt; side < 2; side += tws) {
                    double v[3] = {0.0, 0.0, 0.0};
                    if (M.valid && !M.zero) side_diag<W>(P, M, side, uo, t_new, kzc, t, v);
#pragma unroll
                    for (int q = 0; q < 3; ++q) {
#pragma unroll
                        for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
                        if (lane == 0) dred[team * 6 + 2 * q + side] += v[q];
                    }
                }
            }
        }
    }

    // ---- CTA sums of the stress profiles and diagnostics (fixed order)
    __syncthreads();
    if (tr) A.trace[2] = gtimer();
    double* part = A.partials + (size_t)cta * W::PL;
    for (int idx = tid; idx < W::NE * NZ; idx += blockDim.x) {
        const int e = idx / NZ, z = idx % NZ, r = z / T, tt = z % T;
        double s = 0.0;
        for (int tm = 0; tm < nteams; ++tm) {
            const double* ac = reinterpret_cast<const double*>(smem_raw + W::o_team + W::TEAM_BYTES * (size_t)tm +
                                                               W::TM_ACC) + 256 * e + 32 * r + tt;
#pragma unroll
            for (int gg = 0; gg < GPW; ++gg) s += ac[gg * T];
        }
        part[idx] = s;
    }
    if (tid < 6) {
        double s = 0.0;
        for (int tm = 0; tm < nteams; ++tm) s += dred[tm * 6 + tid];
        part[W::NE * NZ + tid] = s;
    }

    __syncthreads();
    if (tr) A.trace[3] = gtimer();
    if (tid == 0 && !A.rhs_only) advance_clock<FORCED>(lc, S, P, last, diag_due);
    if (REDUCER) {
        if (tid < W::NMF) {
            __threadfence();  // covers the CTA's stores, ordered before it by the barrier
            atomicAdd(arrive + 32 * tid, 1u);
        }
        return STAGE_DONE;
    }
    // ---- two-level last-arriver reduction
    __threadfence();
    __syncthreads();
    const int ngroups = (ncta + RED_GROUP - 1) / RED_GROUP;
    const int grp = QLGPU_CHECK_INDEX(cta / RED_GROUP, 64, &A.clk->status);  // DevClock::cnt_group
    const int c0 = grp * RED_GROUP;
    const int cn_in = min(RED_GROUP, ncta - c0);
    if (tid == 0) {
        unsigned tk = atomicAdd(&A.clk->cnt_group[grp], 1u);
        ss.last = (tk == (unsigned)(cn_in - 1));
    }
    __syncthreads();
    if (!ss.last) return STAGE_DONE;
    __threadfence();
    double* tot = reinterpret_cast<double*>(smem_raw + W::o_team);
    top_prefetch<W>(A, tot);
    if (ngroups > 1) {
        double* gpart = A.gpartials + (size_t)grp * W::PL;
        for (int idx = tid; idx < W::PL; idx += blockDim.x) {
            // CTAs in order, all their loads in flight
            double v[RED_GROUP], s = 0.0;
#pragma unroll
            for (int u = 0; u < RED_GROUP; ++u)
                v[u] = u < cn_in ? __ldcg(A.partials + (size_t)(c0 + u) * W::PL + idx) : 0.0;
#pragma unroll
            for (int u = 0; u < RED_GROUP; ++u)
                if (u < cn_in) s += v[u];
            gpart[idx] = s;
        }
        if (tid == 0) atomicExch(&A.clk->cnt_group[grp], 0u);
        __threadfence();
        __syncthreads();
        if (tid == 0) {
            unsigned tk = atomicAdd(&A.clk->cnt_top, 1u);
            ss.last = (tk == (unsigned)(ngroups - 1));
        }
        __syncthreads();
        if (!ss.last) {
            cp_async_wait_all();  // the scratch is reused by the next stage
            __syncthreads();
            return STAGE_DONE;
        }
        __threadfence();
        for (int idx = tid; idx < W::PL; idx += blockDim.x) {
            double s = 0.0;
            for (int q = 0; q < ngroups; q += 16) {
                double v[16];
#pragma unroll
                for (int u = 0; u < 16; ++u)
                    v[u] = q + u < ngroups ? __ldcg(A.gpartials + (size_t)(q + u) * W::PL + idx) : 0.0;
#pragma unroll
                for (int u = 0; u < 16; ++u)
                    if (q + u < ngroups) s += v[u];
            }
            tot[idx] = s;
        }
        if (tid == 0) atomicExch(&A.clk->cnt_top, 0u);
    } else {
        // one group: its last CTA is the last of all
        for (int idx = tid; idx < W::PL; idx += blockDim.x) {
            double v[RED_GROUP], s = 0.0;
#pragma unroll
            for (int u = 0; u < RED_GROUP; ++u)
                v[u] = u < cn_in ? __ldcg(A.partials + (size_t)u * W::PL + idx) : 0.0;
#pragma unroll
            for (int u = 0; u < RED_GROUP; ++u)
                if (u < cn_in) s += v[u];
            tot[idx] = s;
        }
        if (tid == 0) atomicExch(&A.clk->cnt_group[0], 0u);
    }
    if (A.trace && tid == 0) A.trace[4] = gtimer();
    __syncthreads();
    // exchange buffers of the mean-field transforms: the last four result buffers of the first team
    cplx* xch = reinterpret_cast<cplx*>(smem_raw + W::o_team + W::TOP_XCH);
    wide::top_stage<W, MODEL, INTEG>(A, P, tot, xch, tw, nullptr, tclock, t_new, last, diag_due);
    if (A.trace && tid == 0) A.trace[5] = gtimer();
    return STAGE_TOP;
}

// One stage launch of a single case (Model::rhs, timed stages, host-controlled steps).
template <int NZ, int MODEL, int INTEG>
__global__ void __launch_bounds__(32 * wide::MAX_WARPS<MODEL>, 1) stage_kernel(const __grid_constant__ StageArgs A,
                                                                       const __grid_constant__ DevParams P) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ StageShared ss;
    __shared__ LocalClock lc;
    if (threadIdx.x == 0) load_clock(lc, A.clk);
    __syncthreads();
    stage_body<NZ, MODEL, INTEG, false, true, false>(A, P, (int)blockIdx.x, (int)gridDim.x, smem_raw, ss, lc, true, nullptr,
                                        [](int) { return true; });
}

// ---------------------------------------------------------------------------
// Stage counters shared by the CTAs of one launch (a case's mean field)
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned* p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];\n" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release_u32(unsigned* p, unsigned v) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;\n" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ int ld_volatile_i32(const int* p) { return *reinterpret_cast<const volatile int*>(p); }

// Wait (one thread) until *p has reached target.  False when the launch was aborted or the wait
// exceeded wait_ns; the caller's CTA then leaves, and the abort word makes the others leave.
__device__ __forceinline__ bool run_wait(const unsigned* p, unsigned target, DevClock* C, long long wait_ns) {
    const unsigned long long t0 = gtimer();
    // at least ~16 ns per iteration: the cap ends the wait even if the timer misbehaves
    const long long max_iter = wait_ns / 16 + 1024;
    for (long long it = 0; it < max_iter; ++it) {
        if ((int)(ld_acquire_u32(p) - target) >= 0) return true;
        if ((it & 63) == 63) {
            if (ld_volatile_i32(&C->abort)) return false;
            if ((long long)(gtimer() - t0) > wait_ns) break;
        }
    }
    atomicOr(&C->status, QLGPU_STATUS_TIMEOUT);
    atomicExch(&C->abort, 1);
    return false;
}

// The mean-field side of one stage in the reducer CTA of mean field `e`: the partial sums of
// stress profile e over all `ncta` CTAs, in the order of the two-level reduction (CTAs within
// a group of RED_GROUP, then the groups), then the field's part of the mean-field stage, the
// result in mfo.  What bounds it is one SM's reading of the sums, so 16-byte loads, 16 a thread
// in flight (the guard is in the value: a guarded load makes the compiler wait for each before the
// next, 30 % slower overall).  147 CTAs x NZ = 128 took 5.8 us for both profiles of MHD_BQlin and
// 3.8 for one with 8-byte loads; 40 steps of 64x64 x NZ=128 3.47 -> 3.39 ms with these, 22x18 x
// NZ=256 1.69 -> 1.63.
template <int NZ, int MODEL, int INTEG, bool FORCED>
__device__ __forceinline__ void reduce_stage(const StageArgs& A, const DevParams& P, int e, int ncta,
                                             unsigned char* smem_raw, const cplx* tw, const double* emf, LocalClock& lc,
                                             double* mx, cplx* mfo) {
    using namespace wide;
    using W = WG<NZ, MODEL>;
    const int tid = threadIdx.x, nth = blockDim.x;
    const bool last = A.sc.last != 0, diag_due = record_due<FORCED>(lc, P, FORCED ? A.sc.dt : P.dt, last);
    const double tclock = lc.t, t_new = __dadd_rn(tclock, FORCED ? A.sc.dt : P.dt);
    double* tot = reinterpret_cast<double*>(smem_raw + W::o_team);
    // group sums beside the scratch
    static_assert((size_t)RUN_MAX_GROUPS * 8 * (NZ + 8) + W::TOP_BYTES + 16 <= W::TEAM_BYTES, "group sums fit");
    double* gs = reinterpret_cast<double*>(smem_raw + W::o_team + ((W::TOP_BYTES + 15) & ~(size_t)15));
    const int ngroups = (ncta + RED_GROUP - 1) / RED_GROUP;
    // columns [col, col + NC) of all rows
    auto sum = [&](auto nc_, int col) {
        constexpr int NC = decltype(nc_)::value, C2 = NC / 2;
        for (int i = tid; i < ngroups * C2; i += nth) {
            // a (group, two values) item at a time, all its loads in flight
            const int q = i / C2, n = min(RED_GROUP, ncta - q * RED_GROUP);
            const double2* src = reinterpret_cast<const double2*>(A.partials + (size_t)q * RED_GROUP * W::PL + col) +
                                 (i - q * C2);
            double2 v[RED_GROUP], t = make_double2(0.0, 0.0);
#pragma unroll
            for (int u = 0; u < RED_GROUP; ++u)
                v[u] = u < n ? __ldcg(src + (size_t)u * (W::PL / 2)) : make_double2(0.0, 0.0);
#pragma unroll
            for (int u = 0; u < RED_GROUP; ++u)
                if (u < n) {
                    t.x += v[u].x;
                    t.y += v[u].y;
                }
            reinterpret_cast<double2*>(gs)[i] = t;
        }
        __syncthreads();
        for (int idx = tid; idx < NC; idx += nth) {
            double s = ngroups > 1 ? 0.0 : gs[idx];
            for (int q = 0; q < ngroups && ngroups > 1; ++q) s += gs[(size_t)q * NC + idx];
            tot[col + idx] = s;
        }
        __syncthreads();
    };
    sum(std::integral_constant<int, NZ>{}, e * NZ);
    if (e == 0 && diag_due) sum(std::integral_constant<int, 8>{}, W::NE * NZ);
    if (A.trace && tid == 0 && e == 0) A.trace[4] = gtimer();
    cplx* xch = reinterpret_cast<cplx*>(smem_raw + W::o_team + W::TOP_XCH);
    top_stage<W, MODEL, INTEG, true, FORCED>(A, P, tot, xch, tw, emf, tclock, t_new, last, diag_due, mx, e, mfo);
    if (tid == 0) advance_clock<FORCED>(lc, A.sc, P, last, diag_due);
    if (A.trace && tid == 0 && e == 0) A.trace[5] = gtimer();
}

// The CFL time step (RK3CN_Elin.cpp:76-80 with Calculate_CFL, MHD_BQlin.cpp:531-556,
// MHD_FullQlin.cpp:760-784) from the largest |mean field|^2 before the previous step's last
// stage, mx0 that of the first mean field now.
template <int MODEL>
__device__ __forceinline__ double cfl_step(const RunArgs& L, double mx0) {
    double c, m[4];
#pragma unroll
    for (int f = 0; f < 4; ++f) m[f] = __ldcg(L.forcing + f);
    if (MODEL == MODEL_BQLIN)
        c = __dadd_rn(__dadd_rn(__dmul_rn(L.kmax, sqrt(m[1])), __dmul_rn(L.kmax, sqrt(mx0))), L.P.q);
    else
        c = __dadd_rn(__dmul_rn(L.kmax, __dadd_rn(__dadd_rn(__dadd_rn(sqrt(m[1]), sqrt(m[0])), sqrt(m[2])), sqrt(m[3]))),
                      L.P.q);
    const double dt = __ddiv_rn(L.cfl, c);
    return dt > L.dt_max ? L.dt_max : dt;
}

// Many steps of a single case in one cooperative launch.  Worker CTAs step their blocks
// stage after stage; the last NMF CTAs have no modes and run the mean-field side, one mean
// field each, so that its chain (sums, two transforms, update, profiles) runs under the
// workers' first inverse transforms of the next stage instead of in a worker that would then
// be the last one to arrive again.  A reducer reads all fields of the stage's start, so the
// fields alternate between two buffers.  Against three launches per step this saves the launch
// gap, the tables and the round trips of profiles and clock.  One reducer for all fields:
// 29.5 us a stage at 64x64 x NZ=128, 15.2 at 22x18 x NZ=256, 14.7 at 48x48 x NZ=64 of
// MHD_FullQlin; one per field: 27.0, 13.2, 12.0.  Every wait is bounded in time and iterations; one
// that gives up sets QLGPU_STATUS_TIMEOUT and the abort word, and every CTA leaves.
//
// FORCED, a kernel of its own (with its code in the plain one every launch is 2-3 %
// slower): with the CFL condition (L.cfl > 0) the first reducer sets each step's dt from the
// maxima of the profiles that the reducers form, in the launch's first wait and at the end of
// each step, and the others wait for it before a step's first stage.  Driving noise is added
// by the teams after the last stage.  32x32 x NZ=64 with both: 95 us a step with the host setting
// dt and the noise in a launch of its own, 41 us so.
template <int NZ, int MODEL, int INTEG, bool FORCED>
__global__ void __launch_bounds__(32 * wide::MAX_WARPS<MODEL>, 1) run_kernel(const __grid_constant__ RunArgs L) {
    using W = wide::WG<NZ, MODEL>;
    constexpr int NR = W::NMF;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ StageShared ss;
    __shared__ LocalClock lc;
    __shared__ NoiseSpec s_noise;
    __shared__ double s_mx[4];
    __shared__ __align__(16) StageArgs sA[3];
    const int tid = threadIdx.x, lane = tid & 31, ncta = (int)gridDim.x - NR;
    const int e = (int)blockIdx.x - ncta;  // >= 0: reducer of field e
    const bool cfl = FORCED && L.cfl > 0.0;
    const unsigned e0 = cfl ? 1 : 0;  // epoch 1: the first time step is set
    DevClock* C = L.A[0].clk;
    for (int i = tid; i < (int)(sizeof(sA) / 8); i += blockDim.x)
        reinterpret_cast<unsigned long long*>(sA)[i] = reinterpret_cast<const unsigned long long*>(L.A)[i];
    if (tid == 0) {
        load_clock(lc, C);
        ss.ok = __ldcg(&C->abort) == 0;
        if (FORCED) {
            lc.every = L.diag_every;
            lc.step = L.diag_step0;
            lc.max_rec = L.diag_max;
            s_noise = L.noise;
        }
    }
    __syncthreads();
    if (!ss.ok) return;  // the launch before gave up: its state and counters are no start
    const size_t nlin = (size_t)L.P.nxy * 4 * L.P.nz, nmfe = (size_t)L.P.nmf * L.P.nz;
    const unsigned nstages = 3u * (unsigned)L.nsteps;
    // the mean fields at the start of stage k of the launch
    auto mf_in = [&](unsigned k) {
        return k == 0 || k == nstages ? L.A[0].mf : L.mf_alt + (size_t)((k - 1) & 1u) * nmfe;
    };
    unsigned k = 0;  // stages before this one in the launch
    if (e >= 0) {
        cplx* tw = reinterpret_cast<cplx*>(smem_raw + W::o_tw);
        double* emf = reinterpret_cast<double*>(smem_raw + W::o_ekz);
        double* tot = reinterpret_cast<double*>(smem_raw + W::o_team);
        for (int i = tid; i < NZ; i += blockDim.x) tw[i] = ldc_cg(L.A[0].tw + i);
        // wait by the first warp's lanes for the other reducers' `target` (lane: its reducer)
        auto wait_others = [&](unsigned target, int r) -> bool {
            return r >= NR || r == e || run_wait(C->epoch + 32 * r, target, C, L.wait_ns);
        };
        double dt_sum = 0.0;  // thread 0 of the first reducer
        if (cfl) {
            __syncthreads();
            if (e == 0 && tid < 32 && W::BQ)
                wide::mean_profiles8<W, W::BQ, true>(
                    L.P, [&](int f, int s) { return ldc_cg(L.A[0].mf + f * W::nz + s); }, nullptr,
                    reinterpret_cast<cplx*>(smem_raw + W::o_team + W::TOP_XCH), tw, 0, 1, tid, s_mx, W::NPROF,
                    W::NPROF + 1);
            __syncthreads();
            if (tid == 0) {
                if (e == 0) {
                    dt_sum = __ldcg(L.forcing + 4);
                    L.forcing[5] = cfl_step<MODEL>(L, s_mx[0]);
                }
                st_release_u32(C->epoch + 32 * e, e0);
            }
        }
        for (int n = 0; n < L.nsteps; ++n)
            for (int s = 0; s < 3; ++s, ++k) {
                __syncthreads();
                // the fields at the stage's start, complete once all reducers are (at the launch's start they are)
                if (tid < 32) {
                    const int ok = __all_sync(0xffffffffu, k + e0 == 0 || wait_others(k + e0, lane));
                    if (lane == 0) {
                        ss.ok = ok;
                        sA[s].mf = mf_in(k);
                        if (cfl && s == 0)
                            for (int i = 0; i < 3; ++i)
                                sA[i].sc = stage_const(__ldcg(L.forcing + 5), INTEG == INTEG_CN, i);
                    }
                }
                __syncthreads();
                if (!ss.ok) return;
                wide::top_prefetch<W>(sA[s], tot);
                if (tid == 0)
                    ss.arrived = run_wait(C->arrive + 32 * e, (k + 1) * (unsigned)ncta, C, L.wait_ns) ? 1 : 0;
                if (INTEG == INTEG_EXP)  // under the wait (the last threads: the first one polls)
                    for (int i = blockDim.x - 1 - tid; i < W::nz; i += blockDim.x) {
                        const double kz2 = kz2val(kzval(i <= W::H ? i : i - W::nz, L.P.kzL));
                        const double lc_ = sA[s].sc.linC;
                        emf[i] = L.P.ql ? exp(__dmul_rn(lc_, __dmul_rn(L.P.eta, kz2))) : 1.0;
                        emf[W::NZE + i] = L.P.ql ? exp(__dmul_rn(lc_, __dmul_rn(L.P.nu, kz2))) : 1.0;
                    }
                __syncthreads();
                if (!ss.arrived) {
                    cp_async_wait_all();
                    return;
                }
                const bool rec = e == 0 && record_due<FORCED>(lc, L.P, FORCED ? sA[s].sc.dt : L.P.dt, s == 2);
                reduce_stage<NZ, MODEL, INTEG, FORCED>(sA[s], L.P, e, ncta, smem_raw, tw,
                                                       INTEG == INTEG_EXP ? emf : nullptr, lc, cfl ? s_mx : nullptr,
                                                       mf_in(k + 1));
                const bool end = k + 1 == nstages;
                if (tid == 0) {
                    if (cfl && s == 1) L.forcing[e] = s_mx[e];
                    if (cfl && s == 2 && e == 0) {
                        L.forcing[4] = dt_sum = __dadd_rn(dt_sum, sA[0].sc.dt);
                        L.forcing[5] = cfl_step<MODEL>(L, s_mx[0]);
                    }
                    st_release_u32(C->epoch + 32 * e, k + 1 + e0);
                }
                if (rec || (end && e == 0)) {
                    // the others' new fields, for the record (they are not overwritten before this reducer
                    // has finished another stage); at the end the last use of the others' counters
                    if (tid < 32) {
                        const int ok = __all_sync(0xffffffffu, wait_others(k + 1 + e0, lane));
                        if (lane == 0) ss.ok = ok;
                    }
                    __syncthreads();
                    if (!ss.ok) return;
                    if (rec) {
                        cplx* mfs = wide::top_mfs<W>(tot);
                        for (int i = tid; i < (int)nmfe; i += blockDim.x) mfs[i] = ldc_cg(mf_in(k + 1) + i);
                        __syncthreads();
                        if (tid < 32) step_record<W>(sA[s], L.P, tot + W::NE * NZ, mfs, lc.t, tid);
                    }
                    // nobody waits any more: ready for the next launch
                    if (end && tid < NR) C->arrive[32 * tid] = C->epoch[32 * tid] = 0;
                }
            }
        return;
    }
    if (FORCED && tid == 0 && L.noise_on) {
        lc.nstep = L.step0;
        sA[2].noise = &s_noise;
    }
    for (int n = 0; n < L.nsteps; ++n)
        for (int s = 0; s < 3; ++s, ++k) {
            __syncthreads();
            if (cfl && s == 0) {
                if (tid == 0) {
                    ss.ok = run_wait(C->epoch, k + 1, C, L.wait_ns) ? 1 : 0;
                    const double dt = __ldcg(L.forcing + 5);
                    for (int i = 0; i < 3; ++i) sA[i].sc = stage_const(dt, INTEG == INTEG_CN, i);
                    s_noise.multfac = noise_factor(dt, s_noise.tot2);
                }
                __syncthreads();
                if (!ss.ok) return;
            }
            if (tid == 0) {
                StageArgs& A = sA[s];
                const int in = (int)((k + (unsigned)L.cur) & 1u);
                A.lin_in = L.lin[in];
                A.lin_out = L.lin[in ^ 1];
                if (L.rec_lin) {
                    A.mf = mf_in(k);
                    A.rec_lin = L.rec_lin + (size_t)k * nlin;
                    A.rec_mf = L.rec_mf + (size_t)k * nmfe;
                    A.rec_kx = s == 0 ? L.rec_kx + (size_t)n * L.P.nxy : nullptr;
                    A.rec_t = s == 0 ? L.rec_t + n : nullptr;
                    A.rec_cn = L.rec_cn ? L.rec_cn + k : nullptr;
                }
            }
            __syncthreads();
            const StageResult r = stage_body<NZ, MODEL, INTEG, true, false, FORCED>(
                sA[s], L.P, (int)blockIdx.x, ncta, smem_raw, ss, lc, k == 0, C->arrive, [&](int r_) -> bool {
                    return r_ >= NR || run_wait(C->epoch + 32 * r_, k + e0, C, L.wait_ns);
                });
            if (r == STAGE_ABORT) return;
        }
}

}  // namespace qlgpu
