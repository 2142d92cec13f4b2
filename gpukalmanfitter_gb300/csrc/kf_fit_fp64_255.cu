// kf_fit_fp64_255.cu — FP64 fit kernels with up to 255 registers a thread
// (threads per block x blocks per SM: 128 x 2, 64 x 4, 256 x 1, and the plain form).
#include <cuda_runtime.h>

#include "kf_kernels.cuh"

KF_FIT_LAUNCHER(launchFit_fp64_uniform_255, kfd::kUniform64, false, 256, 1)
KF_FIT_LAUNCHER(launchFit_fp64_grid_255, kfd::kGrid64, false, 256, 1)
