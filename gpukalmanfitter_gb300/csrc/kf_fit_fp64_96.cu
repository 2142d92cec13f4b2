// kf_fit_fp64_96.cu — FP64 fit kernels with up to 96 registers a thread
// (threads per block x blocks per SM: 128 x 5, of which shared memory holds four).
#include <cuda_runtime.h>

#include "kf_kernels.cuh"

KF_FIT_LAUNCHER(launchFit_fp64_uniform_96, kfd::kUniform64, false, 128, 5)
KF_FIT_LAUNCHER(launchFit_fp64_grid_96, kfd::kGrid64, false, 128, 5)
