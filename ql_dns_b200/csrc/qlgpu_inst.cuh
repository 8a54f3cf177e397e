// qlgpu_inst.cuh -- the stage-variant table for one NZ: launch wrappers and
// sizes of stage_kernel<NZ, model, integrator>.  Included by one translation
// unit per NZ (qlgpu_nz<NZ>.cu) so the variants compile in parallel.
#pragma once
#include "qlgpu_host.h"
#include "qlgpu_wide.cuh"

namespace qlgpu {

template <int NZ, int MODEL, int INTEG>
void launch_stage(const StageArgs& A, const DevParams& P, int grid, int block, size_t smem, cudaStream_t st) {
    stage_kernel<NZ, MODEL, INTEG><<<grid, block, smem, st>>>(A, P);
}
template <int NZ, int MODEL, int INTEG>
const void* stage_ptr() {
    return reinterpret_cast<const void*>(&stage_kernel<NZ, MODEL, INTEG>);
}
template <int NZ, int MODEL, int INTEG, bool FORCED>
cudaError_t launch_run(const RunArgs& R, int grid, int block, size_t smem, cudaStream_t st) {
    cudaLaunchConfig_t cfg;
    std::memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;  // all CTAs co-resident, or the launch fails
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, run_kernel<NZ, MODEL, INTEG, FORCED>, R);
}
template <int NZ, int MODEL, int INTEG, bool FORCED>
const void* run_ptr() {
    return reinterpret_cast<const void*>(&run_kernel<NZ, MODEL, INTEG, FORCED>);
}
template <int NZ, int MODEL>
size_t stage_smem(int warps) {
    return wide::WG<NZ, MODEL>::bytes(warps);
}

template <int NZ, int MODEL, int INTEG>
Variant make_variant() {
    Variant v;
    v.launch = &launch_stage<NZ, MODEL, INTEG>;
    v.kernel = &stage_ptr<NZ, MODEL, INTEG>;
    v.run[0] = &launch_run<NZ, MODEL, INTEG, false>;
    v.run[1] = &launch_run<NZ, MODEL, INTEG, true>;
    v.run_kernel[0] = &run_ptr<NZ, MODEL, INTEG, false>;
    v.run_kernel[1] = &run_ptr<NZ, MODEL, INTEG, true>;
    v.smem = &stage_smem<NZ, MODEL>;
    v.PL = wide::WG<NZ, MODEL>::PL;
    v.max_warps = wide::MAX_WARPS<MODEL>;
    return v;
}

template <int NZ>
bool make_variant_for(int model, int integ, Variant* out) {
    if (model == MODEL_BQLIN && integ == INTEG_EXP)
        *out = make_variant<NZ, MODEL_BQLIN, INTEG_EXP>();
    else if (model == MODEL_BQLIN && integ == INTEG_CN)
        *out = make_variant<NZ, MODEL_BQLIN, INTEG_CN>();
    else if (model == MODEL_FULLQLIN && integ == INTEG_EXP)
        *out = make_variant<NZ, MODEL_FULLQLIN, INTEG_EXP>();
    else if (model == MODEL_FULLQLIN && integ == INTEG_CN)
        *out = make_variant<NZ, MODEL_FULLQLIN, INTEG_CN>();
    else
        return false;
    return true;
}

}  // namespace qlgpu

#define QLGPU_DEFINE_NZ(NZV)                                        \
    namespace qlgpu {                                               \
    bool make_variant_nz##NZV(int model, int integ, Variant* out) { \
        return make_variant_for<NZV>(model, integ, out);            \
    }                                                               \
    }
