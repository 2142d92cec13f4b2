// kf_fit_fp64_128.cu — FP64 fit kernels with up to 128 registers a thread
// (threads per block x blocks per SM: 128 x 4, 64 x 8, 256 x 2).
#include <cuda_runtime.h>

#include "kf_kernels.cuh"

KF_FIT_LAUNCHER(launchFit_fp64_uniform_128, kfd::kUniform64, false, 256, 2)
KF_FIT_LAUNCHER(launchFit_fp64_grid_128, kfd::kGrid64, false, 256, 2)
