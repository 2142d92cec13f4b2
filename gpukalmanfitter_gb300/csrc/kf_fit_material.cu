// kf_fit_material.cu — fit kernels with surface material effects (process
// noise; fixed-point smoother of the first state).
#include <cuda_runtime.h>

#include "kf_kernels.cuh"

KF_FIT_LAUNCHER(launchFitMaterial_fp64_uniform, kfd::kUniform64, true, 256, 1)
KF_FIT_LAUNCHER(launchFitMaterial_fp64_grid, kfd::kGrid64, true, 256, 1)
KF_FIT_LAUNCHER(launchFitMaterial_mixed, kfd::kMixed, true, 256, 1)
KF_FIT_LAUNCHER(launchFitMaterial_fp64_any, kfd::kUniformAny, true, 256, 1)
KF_FIT_LAUNCHER(launchFitMaterial_mixed_uniform, kfd::kMixedUniform, true, 256, 1)
