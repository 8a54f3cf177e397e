// qlgpu_batch.cuh -- the persistent kernel of a batched ensemble: many
// independent quasi-linear cases (different mode grids, NZ, viscosities, mean
// fields) stepped for many RK3 steps by ONE cooperative launch.
//
// Every CTA owns a short list of work items (case c, CTA number i of the n
// CTAs given to c) chosen on the host.  Per stage it runs stage_body() for each
// item, i.e. the same fused stage as the single-case kernel, with the CTA
// index and count of the item in place of blockIdx / gridDim.  The last CTA of
// a case to publish its partial sums runs the case's mean-field stage and then
// releases the case's stage counter; the other CTAs of the case wait for that
// counter in their next stage of the case, after its first inverse transforms.
// There is no grid-wide barrier: cases advance independently, each at the pace of
// its own CTAs.  No cycle: a CTA publishes stage k - 1 of all its items before it
// starts stage k of any.
//
// Every wait is bounded (wait_ns, and an iteration cap): a CTA that gives up
// sets QLGPU_STATUS_TIMEOUT and the abort word, and every CTA then leaves its
// step loop and returns.  The host launches the kernel with the
// cooperative attribute, so all CTAs are co-resident or the launch fails.
#pragma once
#include "qlgpu_wide.cuh"

namespace qlgpu {

// Wait (one thread) until *epoch >= target.  False when the launch was aborted
// or the wait exceeded wait_ns (then the abort word is set here).
static __device__ __noinline__ bool batch_wait(const unsigned* epoch, unsigned target, BatchCtl* ctl, long long wait_ns,
                                               int c, unsigned k) {
    const unsigned long long t0 = gtimer();
    // at least ~32 ns per iteration: the cap ends the wait even if the timer misbehaves
    const long long max_iter = wait_ns / 32 + 1024;
    unsigned ns = 32;
    for (long long it = 0; it < max_iter; ++it) {
        if ((int)(ld_acquire_u32(epoch) - target) >= 0) return true;
        if (ld_volatile_i32(&ctl->abort)) return false;
        if ((long long)(gtimer() - t0) > wait_ns) break;
        __nanosleep(ns);
        if (ns < 512) ns <<= 1;
    }
    if (atomicOr(&ctl->status, QLGPU_STATUS_TIMEOUT) == 0) {
        ctl->fail_case = c;
        ctl->fail_stage = (int)k;
    }
    atomicExch(&ctl->abort, 1);
    return false;
}

// Copy n bytes (a multiple of 8) from global to shared memory with the whole CTA.
__device__ __forceinline__ void cta_copy8(void* dst, const void* src, int n) {
    const unsigned long long* s = reinterpret_cast<const unsigned long long*>(src);
    unsigned long long* d = reinterpret_cast<unsigned long long*>(dst);
    for (int i = threadIdx.x; i < n / 8; i += blockDim.x) d[i] = __ldcg(s + i);
}

// One stage of one work item of a given NZ; returns true in the CTA that
// completed the case's stage.  Kept out of line: one function per NZ class
// keeps the compile time of the kernel linear in the number of classes.  The
// shared-memory objects are declared here so that every access stays a
// shared-space access.
template <int NZ, int MODEL, int INTEG>
__device__ __noinline__ StageResult batch_item_stage(const BatchLaunch& L, const BatchCase* cs, const BatchSlot it,
                                                     int s, int n, LocalClock& lc, bool fresh) {
    static_assert(sizeof(StageArgs) % 8 == 0 && sizeof(DevParams) % 8 == 0, "8-byte copies");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ StageShared ss;
    __shared__ __align__(16) StageArgs sA;
    __shared__ __align__(16) DevParams sP;
    __syncthreads();  // the previous item is done with sA / sP
    if (fresh) cta_copy8(&sP, &cs->P, (int)sizeof(DevParams));
    cta_copy8(&sA, &cs->A[s], (int)sizeof(StageArgs));
    __syncthreads();
    const unsigned k = 3u * (unsigned)n + (unsigned)s;  // stages before this one in the launch
    if (threadIdx.x == 0) {
        if ((n + L.parity) & 1) {
            const cplx* in = sA.lin_in;
            sA.lin_in = sA.lin_out;
            sA.lin_out = const_cast<cplx*>(in);
        }
        cplx* rl = cs->rec_lin;
        if (rl) {
            const size_t nlin = (size_t)sP.nxy * 4 * sP.nz, nmfe = (size_t)sP.nmf * sP.nz;
            sA.rec_lin = rl + (size_t)k * nlin;
            sA.rec_mf = cs->rec_mf + (size_t)k * nmfe;
            sA.rec_kx = s == 0 ? cs->rec_kx + (size_t)n * sP.nxy : nullptr;
            sA.rec_t = s == 0 ? cs->rec_t + n : nullptr;
            sA.rec_cn = cs->rec_cn ? cs->rec_cn + k : nullptr;
        }
    }
    __syncthreads();
    return stage_body<NZ, MODEL, INTEG, false, false, false>(sA, sP, it.cta, it.ncta, smem_raw, ss, lc, fresh, nullptr,
                                               [&](int lane) -> bool {
        return lane > 0 || batch_wait(L.epoch + (size_t)it.c * BATCH_EPOCH_STRIDE, k, L.ctl, L.wait_ns, it.c, k);
    });
}

template <int MODEL, int INTEG>
__global__ void __launch_bounds__(32 * BATCH_MAX_WARPS, 1) batch_kernel(const __grid_constant__ BatchLaunch L) {
    __shared__ BatchSlot s_items[BATCH_MAX_SLOTS];
    __shared__ LocalClock s_clk[BATCH_MAX_SLOTS];
    const int tid = threadIdx.x;
    const BatchCta* me = L.ctas + blockIdx.x;
    const int nitems = min(me->nslots, BATCH_MAX_SLOTS);
    if (tid < nitems) {
        BatchSlot it = me->slot[tid];
        it.c = QLGPU_CHECK_INDEX(it.c, L.ncases, &L.ctl->status);
        s_items[tid] = it;
        load_clock(s_clk[tid], L.cases[it.c].A[0].clk);
    }
    if (blockIdx.x == 0 && tid == 0) L.ctl->t_start = gtimer();
    __syncthreads();
    for (int n = 0; n < L.nsteps; ++n)
        for (int s = 0; s < 3; ++s)
            for (int i = 0; i < nitems; ++i) {
                const BatchSlot it = s_items[i];
                const BatchCase* cs = L.cases + it.c;
                // the tables of a CTA's only item stay in shared memory
                const bool fresh = nitems > 1 || (n == 0 && s == 0);
                StageResult r;
                switch (it.NZ) {
                    case 16: r = batch_item_stage<16, MODEL, INTEG>(L, cs, it, s, n, s_clk[i], fresh); break;
                    case 32: r = batch_item_stage<32, MODEL, INTEG>(L, cs, it, s, n, s_clk[i], fresh); break;
                    case 64: r = batch_item_stage<64, MODEL, INTEG>(L, cs, it, s, n, s_clk[i], fresh); break;
                    case 128: r = batch_item_stage<128, MODEL, INTEG>(L, cs, it, s, n, s_clk[i], fresh); break;
                    default: r = batch_item_stage<256, MODEL, INTEG>(L, cs, it, s, n, s_clk[i], fresh); break;
                }
                if (r == STAGE_ABORT) return;
                if (r == STAGE_TOP) {
                    __syncthreads();
                    if (tid == 0) {
                        if (n == L.nsteps - 1 && s == 2) L.case_end[it.c] = gtimer();
                        st_release_u32(L.epoch + (size_t)it.c * BATCH_EPOCH_STRIDE, 3u * (unsigned)n + s + 1);
                    }
                }
            }
}

}  // namespace qlgpu
