// kf_fit_fp64_168.cu — FP64 fit kernels with up to 168 registers a thread
// (threads per block x blocks per SM: 128 x 3).
#include <cuda_runtime.h>

#include "kf_kernels.cuh"

KF_FIT_LAUNCHER(launchFit_fp64_uniform_168, kfd::kUniform64, false, 128, 3)
KF_FIT_LAUNCHER(launchFit_fp64_grid_168, kfd::kGrid64, false, 128, 3)
