// kf_fit_mixed_168.cu — mixed fit kernels with up to 168 registers a thread
// (threads per block x blocks per SM: 128 x 3).
#include <cuda_runtime.h>

#include "kf_kernels.cuh"

KF_FIT_LAUNCHER(launchFit_mixed_168, kfd::kMixed, false, 128, 3)
KF_FIT_LAUNCHER(launchFit_mixed_uniform_168, kfd::kMixedUniform, false, 128, 3)
