// Stage kernels for NZ = 32 (all models and integrators).
#include "qlgpu_inst.cuh"

QLGPU_DEFINE_NZ(32)
