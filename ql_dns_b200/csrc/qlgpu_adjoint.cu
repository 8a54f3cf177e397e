// qlgpu_adjoint.cu -- gradient of the time-averaged Maxwell stress with
// respect to the initial fluctuation field: the forward MHD_BQlin run
// (RK3CN_Elin or RK3CN) with checkpoints, then the discrete adjoint of every step in
// reverse, with the stages of each checkpoint window recomputed
// (qlgpu_adjoint_maxwell in include/qlgpu.h; kernels in qlgpu_adjoint.cuh).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstddef>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/qlgpu.h"
#include "qlgpu_adjoint.cuh"
#include "qlgpu_batch_internal.h"
#include "qlgpu_handle.h"

using namespace qlgpu;

namespace {

struct AdjOps {
    cudaError_t (*modes)(const AdjShared&, const DevParams&, const AdjPos&, int ns, int threads, cudaStream_t);
    cudaError_t (*mf)(const AdjShared&, const DevParams&, const AdjPos&, const AdjPos&, int post, int pre, int ns,
                      cudaStream_t);
    const void* modes_kernel[2];
    size_t modes_smem;
};

// A launch that may start while the kernel before it runs (the kernels wait where they
// need its results).
template <class... KA, class... Args>
cudaError_t launch_pdl(void (*kern)(KA...), dim3 grid, int block, size_t smem, cudaStream_t st, const Args&... args) {
    cudaLaunchConfig_t cfg;
    std::memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, args...);
}
template <int NZ>
cudaError_t ops_modes(const AdjShared& H, const DevParams& P, const AdjPos& X, int ns, int threads, cudaStream_t st) {
    const dim3 grid((unsigned)H.nchunk, (unsigned)ns);
    return threads == ADJ_FEW ? launch_pdl(adj_modes_kernel<NZ, ADJ_FEW>, grid, threads, AG<NZ>::BYTES, st, H, P, X)
                              : launch_pdl(adj_modes_kernel<NZ, ADJ_MANY>, grid, threads, AG<NZ>::BYTES, st, H, P, X);
}
template <int NZ>
cudaError_t ops_mf(const AdjShared& H, const DevParams& P, const AdjPos& X, const AdjPos& Y, int post, int pre, int ns,
                   cudaStream_t st) {
    return launch_pdl(adj_mf_kernel<NZ>, dim3(1, (unsigned)ns), ADJ_MF_THREADS, 0, st, H, P, X, Y, post, pre);
}
template <int NZ>
AdjOps make_ops() {
    return AdjOps{&ops_modes<NZ>, &ops_mf<NZ>,
                  {reinterpret_cast<const void*>(&adj_modes_kernel<NZ, ADJ_FEW>),
                   reinterpret_cast<const void*>(&adj_modes_kernel<NZ, ADJ_MANY>)}, AG<NZ>::BYTES};
}
bool pick_ops(int NZ, AdjOps* o) {
    switch (NZ) {
        case 16: *o = make_ops<16>(); return true;
        case 32: *o = make_ops<32>(); return true;
        case 64: *o = make_ops<64>(); return true;
        case 128: *o = make_ops<128>(); return true;
        case 256: *o = make_ops<256>(); return true;
        default: return false;
    }
}

int afail(qlgpu_t* h, int code, const std::string& msg) {
    h->err = msg;
    return code;
}

int adj_integ(const qlgpu_t* h) { return h->p.integrator == QLGPU_INTEG_RK3CN ? INTEG_CN : INTEG_EXP; }

// the stage-start record of RK3CN copies the clock's bytes from t_old (CnRec's layout)
static_assert(offsetof(DevClock, dtlin_old) == offsetof(DevClock, t_old) + 8 &&
                  offsetof(DevClock, old_init) == offsetof(DevClock, t_old) + 16 && sizeof(CnRec) == 24,
              "CnRec mirrors DevClock from t_old");

#define QA_CK(call)                                                                                \
    do {                                                                                           \
        cudaError_t e_ = (call);                                                                   \
        if (e_ != cudaSuccess) return afail(h, QLGPU_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
    } while (0)

// The workspace of a handle's adjoint calls: one device block as large as the checkpoints and
// one window's records ask for, cut into the call's buffers in two passes, sizes first.  A
// block of at most ADJ_KEEP_BYTES stays with its handle (every seed's has one) for the next call,
// until qlgpu_adjoint_release or the handle's end (25 allocations, clears and frees per seed and
// call took more than half of a 100-step call of 16 seeds); a larger one is given back at the end
// of the call.
constexpr size_t ADJ_KEEP_BYTES = (size_t)512 << 20;

void adj_trim(qlgpu_t* h) {
    if (!h || h->adj_bytes <= ADJ_KEEP_BYTES) return;
    cudaStreamSynchronize(h->stream);
    cudaFree(h->adj_ws);
    h->adj_ws = nullptr;
    h->adj_bytes = 0;
}

struct Arena {
    size_t used = 0;
    unsigned char* base = nullptr;
    template <class T>
    void get(T** out, size_t count) {
        used = (used + 255) & ~(size_t)255;
        if (base) *out = reinterpret_cast<T*>(base + used);
        used += sizeof(T) * count;
    }
};

// One seed's adjoint: the buffers and the position of its sweeps.  The phases
// below only enqueue work on the handle's stream (except where a host copy is
// needed), so several jobs, one per handle, advance together on their own
// streams: qlgpu_adjoint_maxwell_batch interleaves them phase by phase.
struct AdjJob {
    qlgpu_t* h = nullptr;
    AdjOps ops{};
    int N = 0, C = 0, NC = 0;
    size_t nlin = 0, nmfe = 0, nxy = 0;
    cplx *ck_lin = nullptr, *ck_mf = nullptr;
    double* ck_kx0 = nullptr;
    DevClock* ck_clk = nullptr;
    cplx *fin_lin = nullptr, *fin_mf = nullptr;
    double* fin_kx0 = nullptr;
    DevClock* fin_clk = nullptr;
    int fin_cur = 0;
    std::vector<double> rec;
    DevClock cend{};
    cplx *stU = nullptr, *stB = nullptr, *postU = nullptr;
    double *kx_pre = nullptr, *kx_post = nullptr, *t_pre = nullptr;
    CnRec* cn_pre = nullptr;  // RK3CN: the old-operator clock fields at every stage start of the window
    cplx *lamU[2] = {nullptr, nullptr}, *lamB[2] = {nullptr, nullptr};
    cplx *lamF[2] = {nullptr, nullptr}, *lamG[2] = {nullptr, nullptr};
    double *prof = nullptr, *bpart = nullptr;
    AdjSeedBufs* tab = nullptr;  // this seed's entry of the device table
    AdjShared sh{};
    int* rec_status = nullptr;  // status bits of the window recomputes
    int rec_status_host = 0;
    int par = 0;  // stages reversed so far, mod 2
    double J = 0.0;
    // full-window graphs (replayed for every window of C steps when C is even)
    cudaGraphExec_t g_fwd = nullptr, g_rec = nullptr, g_bwd = nullptr;
    ~AdjJob() {
        for (cudaGraphExec_t g : {g_fwd, g_rec, g_bwd})
            if (g) cudaGraphExecDestroy(g);
    }
};

// This call's buffers in the handle's workspace.
void adj_layout(AdjJob& j, Arena& w) {
    const qlgpu_t* h = j.h;
    w.get(&j.ck_lin, (size_t)j.NC * j.nlin);
    w.get(&j.ck_mf, (size_t)j.NC * j.nmfe);
    w.get(&j.ck_kx0, (size_t)j.NC * j.nxy);
    w.get(&j.ck_clk, (size_t)j.NC);
    w.get(&j.fin_lin, j.nlin);
    w.get(&j.fin_mf, j.nmfe);
    w.get(&j.fin_kx0, j.nxy);
    w.get(&j.fin_clk, 1);
    w.get(&j.stU, (size_t)j.C * 3 * j.nlin);
    w.get(&j.stB, (size_t)j.C * 3 * j.nmfe);
    w.get(&j.postU, j.nlin);
    w.get(&j.kx_pre, (size_t)j.C * j.nxy);
    w.get(&j.kx_post, j.nxy);
    w.get(&j.t_pre, (size_t)j.C + 1);
    w.get(&j.cn_pre, (size_t)j.C * 3);
    for (int i = 0; i < 2; ++i) {
        w.get(&j.lamU[i], j.nlin);
        w.get(&j.lamB[i], j.nmfe);
        w.get(&j.lamF[i], j.nlin);
        w.get(&j.lamG[i], j.nmfe);
    }
    w.get(&j.prof, (size_t)5 * h->NZ);
    w.get(&j.bpart, (size_t)3 * h->NZ * j.sh.nchunk);
    w.get(&j.tab, 1);
    w.get(&j.rec_status, 1);
}

AdjSeedBufs adj_seed_bufs(const AdjJob& j) {
    AdjSeedBufs e;
    e.cn_pre = j.cn_pre;
    e.stU = j.stU;
    e.stB = j.stB;
    e.postU = j.postU;
    e.kx_pre = j.kx_pre;
    e.kx_post = j.kx_post;
    e.t_pre = j.t_pre;
    for (int i = 0; i < 2; ++i) {
        e.lamU[i] = j.lamU[i];
        e.lamB[i] = j.lamB[i];
        e.lamF[i] = j.lamF[i];
        e.lamG[i] = j.lamG[i];
    }
    e.prof = j.prof;
    e.bpart = j.bpart;
    return e;
}

int adj_begin(AdjJob& j, qlgpu_t* h, double t0, const double* lin0, const double* mf0, const double* kx0, int nsteps,
              int checkpoint_every, bool load_state) {
    j.h = h;
    if (!lin0 || !mf0 || nsteps < 1 || checkpoint_every < 1)
        return afail(h, QLGPU_ERR_ARG, "null argument, nsteps < 1 or checkpoint_every < 1");
    if (h->p.model != QLGPU_MODEL_MHD_BQLIN)
        return afail(h, QLGPU_ERR_UNSUPPORTED, "the adjoint covers MHD_BQlin (RK3CN_Elin or RK3CN)");
    if (h->noise_f != 0.0 || h->cfl > 0) return afail(h, QLGPU_ERR_UNSUPPORTED, "the adjoint runs at fixed dt, no noise");
    if (!pick_ops(h->NZ, &j.ops)) return afail(h, QLGPU_ERR_UNSUPPORTED, "unsupported NZ");
    QA_CK(cudaSetDevice(h->device));
    for (const void* k : j.ops.modes_kernel) QA_CK(ensure_smem_attr(k, j.ops.modes_smem));
    if (load_state) {
        const int rc = qlgpu_set_state(h, t0, lin0, mf0, kx0);
        if (rc) return rc;
    } else {
        // the forward sweep runs elsewhere; the handle gets its end state at the end of the call
        h->cur = 0;
        h->dt_sum = 0.0;
        h->steps_taken = 0;
    }
    j.N = nsteps;
    j.C = std::min(checkpoint_every, nsteps);
    j.NC = (j.N + j.C - 1) / j.C;
    j.nlin = (size_t)h->nxy * 4 * h->nz;
    j.nmfe = (size_t)h->nmf * h->nz;
    j.nxy = (size_t)h->nxy;
    AdjShared& H = j.sh;
    H.ky = h->d_ky;
    H.kxi = h->d_kxi;
    H.kyi = h->d_kyi;
    H.ilap2 = h->d_ilap2;
    H.tw8 = h->d_tw;
    H.status = h->d_dbg;
    H.nlin = (long long)j.nlin;
    H.nmfe = (long long)j.nmfe;
    // at most 256 chunk sums per seed whatever the number of seeds, so that a seed's result does
    // not depend on the seeds reversed with it
    const int nblocks = (h->nxy + adj_block_modes(h->NZ) - 1) / adj_block_modes(h->NZ);
    H.cblocks = (nblocks + 255) / 256;
    H.nchunk = (nblocks + H.cblocks - 1) / H.cblocks;
    H.integ = adj_integ(h);
    H.weight = 1.0 / j.N;
    Arena w;
    adj_layout(j, w);
    if (w.used > h->adj_bytes) {
        QA_CK(cudaStreamSynchronize(h->stream));
        if (h->adj_ws) cudaFree(h->adj_ws);
        h->adj_ws = nullptr;
        h->adj_bytes = 0;
        QA_CK(cudaMalloc(&h->adj_ws, w.used));
        h->adj_bytes = w.used;
    }
    w.used = 0;
    w.base = static_cast<unsigned char*>(h->adj_ws);
    adj_layout(j, w);
    H.seeds = j.tab;
    const AdjSeedBufs e = adj_seed_bufs(j);
    QA_CK(cudaMemcpyAsync(j.tab, &e, sizeof(e), cudaMemcpyHostToDevice, h->stream));
    // the adjoint of the final state is zero
    QA_CK(cudaMemsetAsync(j.lamU[0], 0, j.nlin * sizeof(cplx), h->stream));
    QA_CK(cudaMemsetAsync(j.lamB[0], 0, j.nmfe * sizeof(cplx), h->stream));
    QA_CK(cudaMemsetAsync(j.rec_status, 0, sizeof(int), h->stream));
    if (h->diag_cap < j.N) {
        if (h->d_diag) cudaFree(h->d_diag);
        h->d_diag = nullptr;
        h->diag_cap = 0;
        QA_CK(cudaMalloc(&h->d_diag, sizeof(double) * 15 * (size_t)j.N));
        h->diag_cap = j.N;
    }
    const int zero = 0;
    QA_CK(cudaMemcpyAsync(&h->d_clk->ndiag, &zero, sizeof(int), cudaMemcpyHostToDevice, h->stream));
    h->dp.tv_interval = h->p.dt;  // the AM_b record of every step
    return QLGPU_OK;
}

// checkpoint c of the forward sweep (the state at the start of window c)
int adj_checkpoint(AdjJob& j, int c) {
    qlgpu_t* h = j.h;
    cudaStream_t st = h->stream;
    QA_CK(cudaMemcpyAsync(j.ck_lin + c * j.nlin, h->d_lin[h->cur], j.nlin * sizeof(cplx), cudaMemcpyDeviceToDevice, st));
    QA_CK(cudaMemcpyAsync(j.ck_mf + c * j.nmfe, h->d_mf, j.nmfe * sizeof(cplx), cudaMemcpyDeviceToDevice, st));
    QA_CK(cudaMemcpyAsync(j.ck_kx0 + c * j.nxy, h->d_kx0, j.nxy * sizeof(double), cudaMemcpyDeviceToDevice, st));
    QA_CK(cudaMemcpyAsync(j.ck_clk + c, h->d_clk, sizeof(DevClock), cudaMemcpyDeviceToDevice, st));
    return QLGPU_OK;
}

// record: every stage's input too (the last window, which is reversed first)
int adj_forward_window(AdjJob& j, int steps, bool record) {
    qlgpu_t* h = j.h;
    const RunRecord r{j.stU, j.stB, j.kx_pre, j.t_pre, j.cn_pre};
    QA_CK(qlgpu_enqueue_run(h, steps, record ? &r : nullptr, nullptr));
    return QLGPU_OK;
}

int adj_forward_end(AdjJob& j) {
    qlgpu_t* h = j.h;
    cudaStream_t st = h->stream;
    QA_CK(cudaGetLastError());
    j.rec.assign((size_t)15 * j.N, 0.0);
    QA_CK(cudaMemcpyAsync(j.rec.data(), h->d_diag, j.rec.size() * sizeof(double), cudaMemcpyDeviceToHost, st));
    QA_CK(cudaMemcpyAsync(&j.cend, h->d_clk, sizeof(DevClock), cudaMemcpyDeviceToHost, st));
    QA_CK(cudaMemcpyAsync(j.fin_lin, h->d_lin[h->cur], j.nlin * sizeof(cplx), cudaMemcpyDeviceToDevice, st));
    QA_CK(cudaMemcpyAsync(j.fin_mf, h->d_mf, j.nmfe * sizeof(cplx), cudaMemcpyDeviceToDevice, st));
    QA_CK(cudaMemcpyAsync(j.fin_kx0, h->d_kx0, j.nxy * sizeof(double), cudaMemcpyDeviceToDevice, st));
    QA_CK(cudaMemcpyAsync(j.fin_clk, h->d_clk, sizeof(DevClock), cudaMemcpyDeviceToDevice, st));
    j.fin_cur = h->cur;
    return QLGPU_OK;
}

// after the stream is synchronised: J
int adj_forward_finish(AdjJob& j) {
    qlgpu_t* h = j.h;
    h->dp.tv_interval = 0.0;
    if (j.cend.status & QLGPU_STATUS_TIMEOUT) {
        QA_CK(qlgpu_clear_abort(h));
        return afail(h, QLGPU_ERR_STATUS, "forward run: a CTA gave up waiting for the other CTAs of the case");
    }
    if (j.cend.status & (QLGPU_STATUS_NONFINITE | QLGPU_STATUS_UNSTABLE))
        return afail(h, QLGPU_ERR_STATUS, "forward run: non-finite or unstable solution");
    if (j.cend.ndiag != j.N) return afail(h, QLGPU_ERR_STATUS, "forward run: missing diagnostic records");
    double s = 0.0;
    for (int n = 0; n < j.N; ++n) s += j.rec[(size_t)15 * n + 8];  // AM_b (MHD_BQlin.cpp:459)
    j.J = s / j.N;
    return QLGPU_OK;
}

int window_steps(const AdjJob& j, int w) { return std::min(j.N, w * j.C + j.C) - w * j.C; }

// restore checkpoint w before recomputing its window
int adj_window_begin(AdjJob& j, int w) {
    qlgpu_t* h = j.h;
    cudaStream_t st = h->stream;
    h->cur = 0;
    QA_CK(cudaMemcpyAsync(h->d_lin[0], j.ck_lin + w * j.nlin, j.nlin * sizeof(cplx), cudaMemcpyDeviceToDevice, st));
    QA_CK(cudaMemcpyAsync(h->d_mf, j.ck_mf + w * j.nmfe, j.nmfe * sizeof(cplx), cudaMemcpyDeviceToDevice, st));
    QA_CK(cudaMemcpyAsync(h->d_kx0, j.ck_kx0 + w * j.nxy, j.nxy * sizeof(double), cudaMemcpyDeviceToDevice, st));
    QA_CK(cudaMemcpyAsync(h->d_clk, j.ck_clk + w, sizeof(DevClock), cudaMemcpyDeviceToDevice, st));
    // the mean-field profile cache holds a later mean field: recompute it in the first stage
    const int zero = 0;
    QA_CK(cudaMemcpyAsync(&h->d_clk->mfr_valid, &zero, sizeof(int), cudaMemcpyHostToDevice, st));
    return QLGPU_OK;
}

// recompute a window, recording every stage's input
int adj_recompute_window(AdjJob& j, int steps) {
    qlgpu_t* h = j.h;
    const RunRecord r{j.stU, j.stB, j.kx_pre, j.t_pre, j.cn_pre};
    QA_CK(qlgpu_enqueue_run(h, steps, &r, nullptr));
    return QLGPU_OK;
}

__global__ void adj_or_status_kernel(const DevClock* c, int* out) { *out |= c->status; }

int adj_window_end(AdjJob& j, int w) {
    qlgpu_t* h = j.h;
    cudaStream_t st = h->stream;
    adj_or_status_kernel<<<1, 1, 0, st>>>(h->d_clk, j.rec_status);
    const int steps = window_steps(j, w);
    QA_CK(cudaMemcpyAsync(j.postU, h->d_lin[h->cur], j.nlin * sizeof(cplx), cudaMemcpyDeviceToDevice, st));
    QA_CK(cudaMemcpyAsync(j.kx_post, h->d_kx0, j.nxy * sizeof(double), cudaMemcpyDeviceToDevice, st));
    QA_CK(cudaMemcpyAsync(j.t_pre + steps, &h->d_clk->t, sizeof(double), cudaMemcpyDeviceToDevice, st));
    return QLGPU_OK;
}

// The adjoint of a window of `steps` steps for the ns seeds of H.seeds, on one stream (the
// step times are read on the device).  Every seed's arithmetic is the same for any ns.
int adj_reverse_window(qlgpu_t* h, const AdjOps& ops, const AdjShared& H, int ns, int steps, int* par,
                       cudaStream_t st) {
    AdjPos X;
    std::memset(&X, 0, sizeof(X));
    X.steps = steps;
    X.n = steps - 1;
    X.s = 2;
    X.par = *par;
    X.sc = h->sc[2];
    // J = (1/N) sum AM_b(post-step state), recorded after the remap (main.cpp:122-130)
    adj_jgrad_kernel<<<dim3(148, ns), 256, 0, st>>>(H, h->dp, X);
    QA_CK(cudaGetLastError());
    QA_CK(ops.mf(H, h->dp, X, X, 0, 1, ns, st));
    int sms = 0;
    QA_CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, h->device));
    const int threads = (long long)H.nchunk * ns <= sms ? ADJ_FEW : ADJ_MANY;
    for (int left = 3 * steps; left > 0; --left) {
        QA_CK(ops.modes(H, h->dp, X, ns, threads, st));
        AdjPos Y = X;
        Y.par ^= 1;
        if (--Y.s < 0) {
            Y.s = 2;
            --Y.n;
        }
        Y.sc = h->sc[Y.s];
        QA_CK(ops.mf(H, h->dp, X, Y, 1, left > 1, ns, st));
        X = Y;
    }
    *par = X.par;
    return QLGPU_OK;
}

int adj_backward_window(AdjJob& j, int steps) {
    return adj_reverse_window(j.h, j.ops, j.sh, 1, steps, &j.par, j.h->stream);
}

// gradients out, and the handle left at the end of the forward run
int adj_finish(AdjJob& j, double* grad_lin, double* grad_mf) {
    qlgpu_t* h = j.h;
    cudaStream_t st = h->stream;
    QA_CK(cudaMemcpyAsync(grad_lin, j.lamU[j.par], j.nlin * sizeof(cplx), cudaMemcpyDeviceToHost, st));
    if (grad_mf) QA_CK(cudaMemcpyAsync(grad_mf, j.lamB[j.par], j.nmfe * sizeof(cplx), cudaMemcpyDeviceToHost, st));
    QA_CK(cudaMemcpyAsync(&j.rec_status_host, j.rec_status, sizeof(int), cudaMemcpyDeviceToHost, st));
    h->cur = j.fin_cur;
    QA_CK(cudaMemcpyAsync(h->d_lin[h->cur], j.fin_lin, j.nlin * sizeof(cplx), cudaMemcpyDeviceToDevice, st));
    QA_CK(cudaMemcpyAsync(h->d_mf, j.fin_mf, j.nmfe * sizeof(cplx), cudaMemcpyDeviceToDevice, st));
    QA_CK(cudaMemcpyAsync(h->d_kx0, j.fin_kx0, j.nxy * sizeof(double), cudaMemcpyDeviceToDevice, st));
    QA_CK(cudaMemcpyAsync(h->d_clk, j.fin_clk, sizeof(DevClock), cudaMemcpyDeviceToDevice, st));
    // the handle's mean-field profile cache is of the last recompute (or, where the forward sweep ran in
    // the batch, of an earlier run): the next step forms the profiles from the restored mean field
    QA_CK(cudaMemsetAsync(&h->d_clk->mfr_valid, 0, sizeof(int), st));
    return QLGPU_OK;
}

int sync_job(AdjJob& j) {
    qlgpu_t* h = j.h;
    QA_CK(cudaStreamSynchronize(h->stream));
    if (j.rec_status_host & QLGPU_STATUS_TIMEOUT) {
        QA_CK(qlgpu_clear_abort(h));
        return afail(h, QLGPU_ERR_STATUS, "window recompute: a CTA gave up waiting for the other CTAs of the case");
    }
    return QLGPU_OK;
}

// The seeds' forward sweep and window recompute in the persistent batch kernel
// (one launch per window for all seeds, the recompute recording every stage's
// input through the kernel's record pointers); the reverse sweep on the batch's
// stream, every kernel launched once for all seeds (per seed on its handle's
// stream when the seeds differ in a parameter).  The batch's reduction order differs from
// the single-case kernel's, so each seed's results agree with
// qlgpu_adjoint_maxwell to round-off rather than bit for bit.
template <class F>
int capture(AdjJob& j, cudaGraphExec_t* out, F body);
int launch_graph(AdjJob& j, cudaGraphExec_t g);

// The reverse sweep runs once for all seeds (one adj_reverse_window) when the
// seeds share every parameter and the device; otherwise per seed.
bool same_params(const qlgpu_params& p, const qlgpu_params& r) {
    return p.model == r.model && p.integrator == r.integrator && p.nx == r.nx &&
           p.ny == r.ny && p.NZ == r.NZ && p.L[0] == r.L[0] && p.L[1] == r.L[1] && p.L[2] == r.L[2] && p.q == r.q &&
           p.omega == r.omega && p.nu == r.nu && p.eta == r.eta && p.B0z == r.B0z &&
           p.viscosity_order == r.viscosity_order && p.dt == r.dt && p.remap == r.remap &&
           p.quasilinear == r.quasilinear;
}
bool same_setup(const qlgpu_t* a, const qlgpu_t* b) { return a->device == b->device && same_params(a->p, b->p); }

// The batch that runs the seeds' forward sweep and recompute: the first handle's from its last
// call when it was made for the same cases (creating and destroying one takes 9 ms at 16
// seeds), else a new one.  It goes back to the handle when the call succeeds and its fields
// take at most ADJ_KEEP_BYTES; the handle frees it.
struct BatchGuard {
    qlgpu_batch_t* b = nullptr;
    ~BatchGuard() {
        if (b) qlgpu_batch_destroy(b);
    }
    int take(qlgpu_t* h, const std::vector<qlgpu_params>& ps) {
        std::swap(b, h->adj_batch);
        bool same = b && ps.size() == h->adj_batch_ps.size();
        for (size_t i = 0; same && i < ps.size(); ++i) same = same_params(ps[i], h->adj_batch_ps[i]);
        if (same) return QLGPU_OK;
        if (b) qlgpu_batch_destroy(b);
        b = nullptr;
        return qlgpu_batch_create(ps.data(), (int)ps.size(), h->device, &b);
    }
    void give(qlgpu_t* h, const std::vector<qlgpu_params>& ps, size_t bytes) {
        if (bytes > ADJ_KEEP_BYTES) return;
        std::swap(b, h->adj_batch);
        h->adj_batch_ps = ps;
    }
};

int run_jobs_persistent(std::vector<AdjJob>& jobs, double t0, const double* lin0, const double* mf0, const double* kx0,
                        double* J, double* const* grad_lin, double* const* grad_mf) {
    const int nj = (int)jobs.size();
    const int N = jobs[0].N, C = jobs[0].C, NC = jobs[0].NC;
    qlgpu_t* h0 = jobs[0].h;
    qlgpu_t* h = h0;  // for QA_CK
    std::vector<qlgpu_params> ps(nj);
    for (int q = 0; q < nj; ++q) ps[q] = jobs[q].h->p;
    BatchGuard g;
    int rc = g.take(h0, ps);
    if (rc) {
        char buf[256];
        qlgpu_batch_last_error(nullptr, buf, sizeof(buf));
        return afail(h0, rc, std::string("adjoint batch: ") + buf);
    }
    qlgpu_batch_t* b = g.b;
    cudaStream_t bs = qlgpu_batch_cuda_stream(b);
    const size_t nlin = jobs[0].nlin, nmfe = jobs[0].nmfe, nxy = jobs[0].nxy;
    // reverse windows as graphs (C even keeps the ping-pong buffers in place across
    // windows) only with QLGPU_ADJ_GRAPH=1: at 16 seeds x 496 modes they measured
    // slower (3.9 s) than direct launches (3.4 s) for 2000 steps
    const char* genv = getenv("QLGPU_ADJ_GRAPH");
    const bool graphs = (C % 2 == 0) && genv && genv[0] == '1';
    for (int q = 0; q < nj; ++q) {
        rc = qlgpu_batch_set_state(b, q, t0, lin0 + q * 2 * nlin, mf0 + q * 2 * nmfe, kx0 ? kx0 + q * nxy : nullptr);
        if (rc) return afail(h0, rc, "adjoint batch: set_state");
    }
    // ---- forward sweep: checkpoints, then one launch per window with a record every step
    std::vector<double> recs((size_t)nj * C * 15);
    std::vector<int> nd(nj);
    std::vector<double> Js(nj, 0.0);
    for (int w = 0; w < NC; ++w) {
        const int steps = std::min(N, w * C + C) - w * C;
        for (int q = 0; q < nj; ++q) {
            AdjJob& j = jobs[q];
            BatchCaseDev d;
            qlgpu_batch_case_dev(b, q, &d);
            QA_CK(cudaMemcpyAsync(j.ck_lin + w * nlin, d.lin, nlin * sizeof(cplx), cudaMemcpyDeviceToDevice, bs));
            QA_CK(cudaMemcpyAsync(j.ck_mf + w * nmfe, d.mf, nmfe * sizeof(cplx), cudaMemcpyDeviceToDevice, bs));
            QA_CK(cudaMemcpyAsync(j.ck_kx0 + w * nxy, d.kx0, nxy * sizeof(double), cudaMemcpyDeviceToDevice, bs));
            QA_CK(cudaMemcpyAsync(j.ck_clk + w, d.clk, sizeof(DevClock), cudaMemcpyDeviceToDevice, bs));
        }
        // the last window is reversed first: its stage inputs are recorded right away
        if (w == NC - 1)
            for (int q = 0; q < nj; ++q) {
                const AdjJob& j = jobs[q];
                qlgpu_batch_set_record(b, q, j.stU, j.stB, j.kx_pre, j.t_pre, j.cn_pre);
            }
        rc = qlgpu_batch_step(b, steps, 1, recs.data(), C, nd.data());
        if (rc) {
            char buf[256];
            qlgpu_batch_last_error(b, buf, sizeof(buf));
            return afail(h0, rc, std::string("adjoint forward sweep: ") + buf);
        }
        for (int q = 0; q < nj; ++q) {
            if (nd[q] != steps) return afail(h0, QLGPU_ERR_STATUS, "forward run: missing diagnostic records");
            for (int n = 0; n < steps; ++n) Js[q] += recs[((size_t)q * C + n) * 15 + 8];  // AM_b
        }
    }
    for (int q = 0; q < nj; ++q) {
        AdjJob& j = jobs[q];
        j.J = Js[q] / N;
        BatchCaseDev d;
        qlgpu_batch_case_dev(b, q, &d);
        QA_CK(cudaMemcpyAsync(j.fin_lin, d.lin, nlin * sizeof(cplx), cudaMemcpyDeviceToDevice, bs));
        QA_CK(cudaMemcpyAsync(j.fin_mf, d.mf, nmfe * sizeof(cplx), cudaMemcpyDeviceToDevice, bs));
        QA_CK(cudaMemcpyAsync(j.fin_kx0, d.kx0, nxy * sizeof(double), cudaMemcpyDeviceToDevice, bs));
        QA_CK(cudaMemcpyAsync(j.fin_clk, d.clk, sizeof(DevClock), cudaMemcpyDeviceToDevice, bs));
        j.fin_cur = 0;
        j.h->dp.tv_interval = 0.0;
    }
    // the reverse sweep: one launch per kernel for all seeds (default), or every seed on its
    // own stream (QLGPU_ADJ_REVERSE=streams, or seeds that differ in a parameter)
    const char* renv = getenv("QLGPU_ADJ_REVERSE");
    bool seeds_rev = !(renv && std::string(renv) == "streams");
    for (int q = 1; q < nj; ++q)
        if (!same_setup(jobs[q].h, h0)) seeds_rev = false;
    AdjShared SH = jobs[0].sh;  // all seeds' entries, in the first handle's table
    int spar = 0;
    if (seeds_rev) {
        std::vector<AdjSeedBufs> hb(nj);
        for (int q = 0; q < nj; ++q) hb[q] = adj_seed_bufs(jobs[q]);
        if (h0->adj_tab_cap < nj) {
            if (h0->adj_tab) cudaFree(h0->adj_tab);
            h0->adj_tab = nullptr;
            h0->adj_tab_cap = 0;
            QA_CK(cudaMalloc(&h0->adj_tab, sizeof(AdjSeedBufs) * nj));
            h0->adj_tab_cap = nj;
        }
        QA_CK(cudaMemcpy(h0->adj_tab, hb.data(), sizeof(AdjSeedBufs) * nj, cudaMemcpyHostToDevice));
        SH.seeds = static_cast<const AdjSeedBufs*>(h0->adj_tab);
        // the seeds' zeroed adjoints were enqueued on their own streams
        for (int q = 0; q < nj; ++q) QA_CK(cudaStreamSynchronize(jobs[q].h->stream));
    }
    // ---- reverse sweep, window by window
    cudaEvent_t ev_b = nullptr;
    std::vector<cudaEvent_t> ev_h(nj, nullptr);
    struct EvGuard {
        cudaEvent_t* e;
        std::vector<cudaEvent_t>* v;
        ~EvGuard() {
            if (*e) cudaEventDestroy(*e);
            for (cudaEvent_t x : *v)
                if (x) cudaEventDestroy(x);
        }
    } evg{&ev_b, &ev_h};
    QA_CK(cudaEventCreateWithFlags(&ev_b, cudaEventDisableTiming));
    for (int q = 0; q < nj; ++q) QA_CK(cudaEventCreateWithFlags(&ev_h[q], cudaEventDisableTiming));
    const int zero = 0;
    for (int w = NC - 1; w >= 0; --w) {
        const int steps = std::min(N, w * C + C) - w * C;
        // the previous window's reverse steps must be done with stU before the recompute rewrites it
        if (w != NC - 1 && !seeds_rev)
            for (int q = 0; q < nj; ++q) {
                QA_CK(cudaEventRecord(ev_h[q], jobs[q].h->stream));
                QA_CK(cudaStreamWaitEvent(bs, ev_h[q], 0));
            }
        for (int q = 0; q < nj && w != NC - 1; ++q) {
            AdjJob& j = jobs[q];
            BatchCaseDev d;
            qlgpu_batch_case_dev(b, q, &d);
            QA_CK(cudaMemcpyAsync(d.lin, j.ck_lin + w * nlin, nlin * sizeof(cplx), cudaMemcpyDeviceToDevice, bs));
            QA_CK(cudaMemcpyAsync(d.mf, j.ck_mf + w * nmfe, nmfe * sizeof(cplx), cudaMemcpyDeviceToDevice, bs));
            QA_CK(cudaMemcpyAsync(d.kx0, j.ck_kx0 + w * nxy, nxy * sizeof(double), cudaMemcpyDeviceToDevice, bs));
            QA_CK(cudaMemcpyAsync(d.clk, j.ck_clk + w, sizeof(DevClock), cudaMemcpyDeviceToDevice, bs));
            // the mean-field profile cache holds a later mean field: recompute it in the first stage
            QA_CK(cudaMemcpyAsync(&d.clk->mfr_valid, &zero, sizeof(int), cudaMemcpyHostToDevice, bs));
            qlgpu_batch_set_record(b, q, j.stU, j.stB, j.kx_pre, j.t_pre, j.cn_pre);
        }
        if (w != NC - 1) rc = qlgpu_batch_step(b, steps, 0, nullptr, 0, nullptr);
        if (rc) {
            char buf[256];
            qlgpu_batch_last_error(b, buf, sizeof(buf));
            return afail(h0, rc, std::string("adjoint recompute: ") + buf);
        }
        for (int q = 0; q < nj; ++q) {
            AdjJob& j = jobs[q];
            BatchCaseDev d;
            qlgpu_batch_case_dev(b, q, &d);  // the buffer parity after the launch
            QA_CK(cudaMemcpyAsync(j.postU, d.lin, nlin * sizeof(cplx), cudaMemcpyDeviceToDevice, bs));
            QA_CK(cudaMemcpyAsync(j.kx_post, d.kx0, nxy * sizeof(double), cudaMemcpyDeviceToDevice, bs));
            QA_CK(cudaMemcpyAsync(j.t_pre + steps, &d.clk->t, sizeof(double), cudaMemcpyDeviceToDevice, bs));
        }
        if (seeds_rev) {
            rc = adj_reverse_window(h0, jobs[0].ops, SH, nj, steps, &spar, bs);
            if (rc) return rc;
            continue;
        }
        QA_CK(cudaEventRecord(ev_b, bs));
        for (int q = 0; q < nj; ++q) {
            AdjJob& j = jobs[q];
            QA_CK(cudaStreamWaitEvent(j.h->stream, ev_b, 0));
            if (graphs && steps == C) {
                // a full window's reverse steps, one graph launch
                if (!j.g_bwd) {
                    rc = capture(j, &j.g_bwd, [&] { return adj_backward_window(j, C); });
                    if (rc) return rc;
                }
                rc = launch_graph(j, j.g_bwd);
                if (rc) return rc;
                continue;
            }
            rc = adj_backward_window(j, steps);
            if (rc) return rc;
        }
    }
    if (seeds_rev) {
        // every seed's buffers in the state adj_backward_window would have left them
        QA_CK(cudaEventRecord(ev_b, bs));
        for (int q = 0; q < nj; ++q) {
            AdjJob& j = jobs[q];
            j.par = spar;
            QA_CK(cudaStreamWaitEvent(j.h->stream, ev_b, 0));
        }
    }
    for (int q = 0; q < nj; ++q) qlgpu_batch_set_record(b, q, nullptr, nullptr, nullptr, nullptr);
    for (int q = 0; q < nj; ++q) {
        rc = adj_finish(jobs[q], grad_lin[q], grad_mf ? grad_mf[q] : nullptr);
        if (rc) return rc;
    }
    for (int q = 0; q < nj; ++q) {
        rc = sync_job(jobs[q]);
        if (rc) return rc;
    }
    QA_CK(cudaStreamSynchronize(bs));
    for (int q = 0; q < nj; ++q) J[q] = jobs[q].J;
    g.give(h0, ps, 4 * sizeof(cplx) * nlin * nj);
    return QLGPU_OK;
}

// Capture `body` on the job's stream into an executable graph.
template <class F>
int capture(AdjJob& j, cudaGraphExec_t* out, F body) {
    qlgpu_t* h = j.h;
    QA_CK(cudaStreamBeginCapture(h->stream, cudaStreamCaptureModeThreadLocal));
    const int rc = body();
    cudaGraph_t g = nullptr;
    const cudaError_t e = cudaStreamEndCapture(h->stream, &g);
    if (rc) {
        if (g) cudaGraphDestroy(g);
        return rc;
    }
    QA_CK(e);
    const cudaError_t e2 = cudaGraphInstantiate(out, g, 0);
    cudaGraphDestroy(g);
    QA_CK(e2);
    return QLGPU_OK;
}

int launch_graph(AdjJob& j, cudaGraphExec_t g) {
    qlgpu_t* h = j.h;
    QA_CK(cudaGraphLaunch(g, h->stream));
    return QLGPU_OK;
}

// All jobs phase by phase; every job's work goes to its own handle's stream.
// Optionally a window of C steps (forward, recompute, reverse) is one graph
// launch per job after its first capture: the buffers a window uses do not
// depend on the window, and with C even the adjoint's ping-pong buffers are
// back in the same order after every window, so the graphs replay unchanged.
int run_jobs(std::vector<AdjJob>& jobs, double* J, double* const* grad_lin, double* const* grad_mf) {
    const int nj = (int)jobs.size();
    const int N = jobs[0].N, C = jobs[0].C, NC = jobs[0].NC;
    // opt-in (QLGPU_ADJ_GRAPH=1): at 16 seeds x 496 modes the graphs measured slower
    // (5.4 s) than direct launches (3.5 s) for 2000 steps
    const char* env = getenv("QLGPU_ADJ_GRAPH");
    const bool graphs = (C % 2 == 0) && env && env[0] == '1';
#define QA_ALL(expr)                                    \
    for (int q_ = 0; q_ < nj; ++q_) {                   \
        AdjJob& jj = jobs[q_];                          \
        (void)jj;                                       \
        int rc_ = (expr);                               \
        if (rc_) return rc_;                            \
    }
    auto rec_window = [&](AdjJob& j, int w, int steps) -> int {
        int rc = adj_recompute_window(j, steps);
        return rc ? rc : adj_window_end(j, w);
    };
    for (int w = 0; w < NC; ++w) {
        const int steps = std::min(N, w * C + C) - w * C;
        QA_ALL(adj_checkpoint(jj, w));
        if (graphs && steps == C && w != NC - 1) {
            QA_ALL(jj.g_fwd ? QLGPU_OK : capture(jj, &jj.g_fwd, [&] { return adj_forward_window(jj, C, false); }));
            QA_ALL(launch_graph(jj, jj.g_fwd));
        } else {
            QA_ALL(adj_forward_window(jj, steps, w == NC - 1));
        }
    }
    QA_ALL(adj_window_end(jj, NC - 1));
    QA_ALL(adj_forward_end(jj));
    QA_ALL(sync_job(jj));
    QA_ALL(adj_forward_finish(jj));
    for (int w = NC - 1; w >= 0; --w) {
        const int steps = std::min(N, w * C + C) - w * C;
        if (w != NC - 1) {
            QA_ALL(adj_window_begin(jj, w));
            if (graphs && steps == C) {
                QA_ALL(jj.g_rec ? QLGPU_OK : capture(jj, &jj.g_rec, [&] { return rec_window(jj, w, C); }));
                QA_ALL(launch_graph(jj, jj.g_rec));
            } else {
                QA_ALL(rec_window(jj, w, steps));
            }
        }
        if (graphs && steps == C) {
            QA_ALL(jj.g_bwd ? QLGPU_OK : capture(jj, &jj.g_bwd, [&] { return adj_backward_window(jj, C); }));
            QA_ALL(launch_graph(jj, jj.g_bwd));
        } else {
            QA_ALL(adj_backward_window(jj, steps));
        }
    }
    for (int q = 0; q < nj; ++q) {
        int rc = adj_finish(jobs[q], grad_lin[q], grad_mf ? grad_mf[q] : nullptr);
        if (rc) return rc;
    }
    QA_ALL(sync_job(jj));
#undef QA_ALL
    for (int q = 0; q < nj; ++q) J[q] = jobs[q].J;
    return QLGPU_OK;
}

}  // namespace

extern "C" int qlgpu_adjoint_maxwell(qlgpu_t* h, double t0, const double* lin0, const double* mf0,
                                     const double* kx0, int nsteps, int checkpoint_every, double* J,
                                     double* grad_lin, double* grad_mf) {
    if (!h) return QLGPU_ERR_ARG;
    if (!J || !grad_lin) return afail(h, QLGPU_ERR_ARG, "null argument");
    std::vector<AdjJob> jobs(1);
    int rc = adj_begin(jobs[0], h, t0, lin0, mf0, kx0, nsteps, checkpoint_every, true);
    double* gl[1] = {grad_lin};
    double* gm[1] = {grad_mf};
    if (!rc) rc = run_jobs(jobs, J, gl, grad_mf ? gm : nullptr);
    adj_trim(h);
    return rc ? rc : qlgpu_debug_verify(h);
}

extern "C" int qlgpu_adjoint_release(qlgpu_t* h) {
    if (!h) return QLGPU_ERR_ARG;
    QA_CK(cudaSetDevice(h->device));
    QA_CK(cudaStreamSynchronize(h->stream));
    if (h->adj_ws) cudaFree(h->adj_ws);
    if (h->adj_tab) cudaFree(h->adj_tab);
    if (h->adj_batch) qlgpu_batch_destroy(h->adj_batch);
    h->adj_ws = h->adj_tab = nullptr;
    h->adj_batch = nullptr;
    h->adj_bytes = 0;
    h->adj_tab_cap = 0;
    h->adj_batch_ps.clear();
    return QLGPU_OK;
}

extern "C" int qlgpu_adjoint_maxwell_batch(qlgpu_t* const* handles, int nseeds, double t0, const double* lin0,
                                           const double* mf0, const double* kx0, int nsteps, int checkpoint_every,
                                           double* J, double* grad_lin, double* grad_mf) {
    if (!handles || nseeds < 1 || !handles[0]) return QLGPU_ERR_ARG;
    qlgpu_t* h0 = handles[0];
    if (!lin0 || !mf0 || !J || !grad_lin) return afail(h0, QLGPU_ERR_ARG, "null argument");
    for (int q = 0; q < nseeds; ++q) {
        if (!handles[q]) return afail(h0, QLGPU_ERR_ARG, "null handle");
        for (int r = 0; r < q; ++r)
            if (handles[r] == handles[q]) return afail(h0, QLGPU_ERR_ARG, "each seed needs its own handle");
        if (handles[q]->nxy != h0->nxy || handles[q]->nz != h0->nz || handles[q]->nmf != h0->nmf)
            return afail(h0, QLGPU_ERR_ARG, "handles of a batch must have the same dimensions");
    }
    const size_t nlin = (size_t)h0->nxy * 4 * h0->nz, nmfe = (size_t)h0->nmf * h0->nz;
    const char* mode = getenv("QLGPU_ADJ_BATCH");
    const bool streams = mode && std::string(mode) == "streams";
    std::vector<AdjJob> jobs(nseeds);
    std::vector<double*> gl(nseeds), gm(nseeds);
    for (int q = 0; q < nseeds; ++q) {
        int rc = adj_begin(jobs[q], handles[q], t0, lin0 + q * 2 * nlin, mf0 + q * 2 * nmfe,
                           kx0 ? kx0 + q * (size_t)h0->nxy : nullptr, nsteps, checkpoint_every, streams);
        if (rc) {
            if (handles[q] != h0) h0->err = handles[q]->err;
            for (int r = 0; r <= q; ++r) adj_trim(handles[r]);
            return rc;
        }
        gl[q] = grad_lin + q * 2 * nlin;
        gm[q] = grad_mf ? grad_mf + q * 2 * nmfe : nullptr;
    }
    // default: forward sweep and recompute of all seeds in the persistent batch kernel;
    // QLGPU_ADJ_BATCH=streams interleaves the single-case path of every seed on its stream
    // (results bit-identical to qlgpu_adjoint_maxwell) from one host thread (threads per
    // seed were slower: their launches contend in the driver)
    int rc = streams ? run_jobs(jobs, J, gl.data(), grad_mf ? gm.data() : nullptr)
                     : run_jobs_persistent(jobs, t0, lin0, mf0, kx0, J, gl.data(), grad_mf ? gm.data() : nullptr);
    for (int q = 0; q < nseeds; ++q) adj_trim(handles[q]);
    for (int q = 0; q < nseeds && !rc; ++q) rc = qlgpu_debug_verify(handles[q]);
    if (rc) {
        for (int q = 0; q < nseeds; ++q)
            if (!handles[q]->err.empty() && handles[q] != h0) h0->err = handles[q]->err;
    }
    return rc;
}
