// kf_fit_mixed_128.cu — mixed fit kernels with up to 128 registers a thread
// (threads per block x blocks per SM: 128 x 4, 64 x 8, 256 x 2).
#include <cuda_runtime.h>

#include "kf_kernels.cuh"

KF_FIT_LAUNCHER(launchFit_mixed_128, kfd::kMixed, false, 256, 2)
KF_FIT_LAUNCHER(launchFit_mixed_uniform_128, kfd::kMixedUniform, false, 256, 2)
