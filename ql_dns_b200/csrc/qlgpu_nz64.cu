// Stage kernels for NZ = 64 (all models and integrators).
#include "qlgpu_inst.cuh"

QLGPU_DEFINE_NZ(64)
