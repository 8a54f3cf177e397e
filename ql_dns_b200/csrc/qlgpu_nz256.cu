// Stage kernels for NZ = 256 (all models and integrators).
#include "qlgpu_inst.cuh"

QLGPU_DEFINE_NZ(256)
