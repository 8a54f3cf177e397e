// qlgpu_kernel.cuh -- the mean-field side of a stage: update, clock and record,
// run by the CTA that arrives last (sm_100a).
#pragma once
#include "qlgpu_debug.cuh"
#include "qlgpu_stage.cuh"

namespace qlgpu {

constexpr int RED_GROUP = 16;  // CTAs per first-level reduction group
constexpr int RUN_MAX_GROUPS = 16;  // of a many-steps launch

// Energy, stress and dissipation sums of one pair of mean fields at stored index s
// (MHD_BQlin.cpp:408-447): v += {energy, stress, -k^2 energy}.
__device__ __forceinline__ void mf_sums(const cplx* x, const cplx* y, int s, double kz2, double* v) {
    const cplx a = x[s], b = y[s];
    const double na = a.x * a.x + a.y * a.y, nb = b.x * b.x + b.y * b.y;
    v[0] += na + nb;
    v[1] += a.x * b.x + a.y * b.y;
    v[2] += -kz2 * na - kz2 * nb;
}

// The 15-column record (MHD_BQlin.cpp:449-477) from the fluctuation sums ds[6] and
// the mean-field sums v = {eMB, aMB, dMB, eMU, aMU, dMU}.
__device__ __forceinline__ void put_record(const DevParams& P, const double* ds, const double* v, double t,
                                           double* o) {
    const double eMB = v[0] * P.divMF, aMB = v[1] * P.divMF, dMB = v[2] * (P.divMF * P.eta);
    const double eMU = v[3] * P.divMF, aMU = v[4] * P.divMF, dMU = v[5] * (P.divMF * P.nu);
    const double du = ds[4] * P.divfac, db = ds[5] * P.divfac;
    o[0] = t;
    o[1] = eMU / 2; o[2] = eMB / 2; o[3] = ds[0] * P.divfac / 2; o[4] = ds[1] * P.divfac / 2;
    o[5] = aMU; o[6] = aMB; o[7] = ds[2] * P.divfac; o[8] = ds[3] * P.divfac;
    o[9] = dMU; o[10] = dMB; o[11] = du; o[12] = db;
    o[13] = pow(P.nu * P.nu * P.nu / (dMU + du), 0.25) * P.kzmax;
    o[14] = pow(P.eta * P.eta * P.eta / (dMB + db), 0.25) * P.kzmax;
}

// ---------------------------------------------------------------------------
// The diagnostic record of a step (Calc_Energy_AM_Diss, MHD_BQlin.cpp:408-477) by one warp
// from the fluctuation sums ds[6] and the mean fields mfs[nmf][nz]: lanes over kz, then a
// fixed shuffle tree.
// ---------------------------------------------------------------------------
template <class W>
__device__ __forceinline__ void step_record(const StageArgs& A, const DevParams& P, const double* ds, const cplx* mfs,
                                            double t_new, int lane) {
    const int nzd = P.nz;
    DevClock* C = A.clk;
    double v[6] = {0, 0, 0, 0, 0, 0};  // eMB, aMB, dMB, eMU, aMU, dMU
    for (int s = lane; s < nzd; s += 32) {
        const double kz2 = kz2val(kzval(s <= W::H ? s : s - nzd, P.kzL));
        mf_sums(mfs, mfs + nzd, s, kz2, v);
        if (P.nmf == 4) mf_sums(mfs + 2 * nzd, mfs + 3 * nzd, s, kz2, v + 3);
    }
#pragma unroll
    for (int q = 0; q < 6; ++q)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
    if (lane != 0) return;
    const int r = C->ndiag;
    if (r < A.diag_cap)
        put_record(P, ds, v, t_new, A.diag_ring + (size_t)QLGPU_CHECK_INDEX(r, A.diag_cap, &C->status) * 15);
    else
        atomicOr(&C->status, QLGPU_STATUS_DIAG_FULL);  // other CTAs of the launch set bits of the same word
    C->ndiag = r + 1;
    C->timevar = __dsub_rn(C->timevar, P.tv_interval);
    C->since = 0;
}

// ---------------------------------------------------------------------------
// Mean-field update, run by the whole CTA that arrives last: the mean-field
// right-hand side from the stress spectra spec[NEMF][H + 1] and its RK update
// (mfs[nmf][nz] in shared memory, updated in place, and mfo; fps: the previous
// right-hand side; emf: the integrating factors, null to compute them), then the time and
// diagnostic bookkeeping in the last warp.  only >= 0 (a reducer of run_kernel): that field
// alone, and no record.  tot[] holds the stress profiles
// summed over all modes (real z) followed by the six fluctuation diagnostic sums.
// ---------------------------------------------------------------------------
template <class W, int MODEL, int INTEG, int NEMF>
__device__ __forceinline__ void mean_field_update(const StageArgs& A, const DevParams& P, const double* tot,
                                                  const double* spec, cplx* mfs, const cplx* fps, const double* emf,
                                                  double tclock, double t_new, bool last, bool diag_due, int only, cplx* mfo) {
    const StageConst& S = A.sc;
    const int tid = threadIdx.x, lane = tid & 31;
    const int nzd = P.nz;
    for (int s = tid; s < nzd; s += blockDim.x) {
        // unpack: full[s] = half[s] (s <= H) or conj(half[nz - s]) (MHD_BQlin.cpp:264-267)
        cplx drive[NEMF];
#pragma unroll
        for (int e = 0; e < NEMF; ++e) {
            const int hs = s <= W::H ? s : nzd - s;
            cplx v = mk(spec[(e * (W::H + 1) + hs) * 2], spec[(e * (W::H + 1) + hs) * 2 + 1]);
            drive[e] = s <= W::H ? v : conjc(v);
        }
        const int kzi = s <= W::H ? s : s - nzd;
        const double c = kzval(kzi, P.kzL);
        const double kz2 = kz2val(c);
        cplx m[4], F[4];
#pragma unroll
        for (int mm = 0; mm < 4; ++mm) {
            m[mm] = (mm < P.nmf) ? mfs[mm * nzd + s] : mk(0.0, 0.0);
            F[mm] = mk(0.0, 0.0);
        }
        if (MODEL == MODEL_BQLIN) {
            // dBy = -q Bx + EMF_y, dBx = EMF_x (MHD_BQlin.cpp:274-280)
            if (P.ql) {
                F[0] = drive[0];
                F[1] = cadd(cscale(m[0], -P.q), drive[1]);
            }
        } else {
            // MHD_FullQlin.cpp:411-423 (B0z kz terms with kz = i c)
            if (P.ql) {
                F[1] = cadd(cadd(cscale(m[0], -P.q), imul(m[3], P.B0z * c)), drive[1]);
                F[0] = cadd(imul(m[2], P.B0z * c), drive[0]);
                F[2] = cadd(cadd(cscale(m[3], 2.0 * P.Omega), imul(m[0], P.B0z * c)), drive[2]);
                F[3] = cadd(cadd(cscale(m[2], P.q - 2.0 * P.Omega), imul(m[1], P.B0z * c)), drive[3]);
            }
        }
        for (int mm = 0; mm < P.nmf; ++mm) {
            if (only >= 0 && mm != only) continue;
            if (A.rhs_only) {
                stc(A.Fmf_out + mm * nzd + s, F[mm]);
                continue;
            }
            const double Lm = P.ql ? __dmul_rn((MODEL == MODEL_FULLQLIN && mm >= 2) ? P.nu : P.eta, kz2) : 0.0;
            cplx fp = S.has_prev ? fps[mm * nzd + s] : mk(0.0, 0.0);
            cplx nv;
            if (INTEG == INTEG_EXP) {
                const double e = emf ? emf[(MODEL == MODEL_FULLQLIN && mm >= 2 ? W::NZE : 0) + s]
                                     : exp(__dmul_rn(S.linC, Lm));
                const cplx acc = S.has_prev ? cadd(cadd(cscale(F[mm], S.n1), cscale(fp, S.n2)), m[mm])
                                            : cadd(cscale(F[mm], S.n1), m[mm]);
                nv = cscale(acc, e);
            } else {
                nv = rk_update(S, Lm, Lm, F[mm], fp, m[mm], S.has_prev);
            }
            if (A.Fmf_out) stc(A.Fmf_out + mm * nzd + s, F[mm]);
            stc(mfo + mm * nzd + s, nv);
            mfs[mm * nzd + s] = nv;
            const double mag = nv.x * nv.x + nv.y * nv.y;
            if (!(mag == mag) || isinf(mag)) atomicOr(&A.clk->status, QLGPU_STATUS_NONFINITE);
            else if (mag > 1e40) atomicOr(&A.clk->status, QLGPU_STATUS_UNSTABLE);
        }
    }
    __syncthreads();
    // the rest in the last warp: the first ones go on to the next stage's profiles
    if (A.rhs_only || (tid >> 5) != (int)(blockDim.x >> 5) - 1) return;
    DevClock* C = A.clk;
    if (lane == 0 && only <= 0) {
        // CN bookkeeping: this stage's operator time becomes "old" (RK3CN.cpp:119-122)
        C->t_old = S.abs_time ? S.t_off : __dadd_rn(tclock, S.t_off);
        C->dtlin_old = S.dt_lin;
        C->old_init = 0;
        if (last) {
            C->t = t_new;
            C->timevar = __dadd_rn(C->timevar, S.dt);
            C->since += 1;
            C->nstep += 1;
        }
    }
    if (last && diag_due && only < 0) step_record<W>(A, P, tot + NEMF * W::NZ, mfs, t_new, lane);
}

}  // namespace qlgpu
