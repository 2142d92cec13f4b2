// kf_fit_coop.cu — fit kernels for small batches: eight lanes a track.
#include <cuda_runtime.h>

#include "kf_kernels.cuh"

KF_COOP_LAUNCHER(launchFitCoop_fp64_uniform, kfd::kUniform64)
KF_COOP_LAUNCHER(launchFitCoop_fp64_grid, kfd::kGrid64)
KF_COOP_LAUNCHER(launchFitCoop_mixed, kfd::kMixed)
KF_COOP_LAUNCHER(launchFitCoop_mixed_uniform, kfd::kMixedUniform)
