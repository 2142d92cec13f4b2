// kf_fit_mixed_255.cu — mixed fit kernels with up to 255 registers a thread
// (threads per block x blocks per SM: 128 x 2, 64 x 4, 256 x 1, and the plain form).
#include <cuda_runtime.h>

#include "kf_kernels.cuh"

KF_FIT_LAUNCHER(launchFit_mixed_255, kfd::kMixed, false, 256, 1)
KF_FIT_LAUNCHER(launchFit_mixed_uniform_255, kfd::kMixedUniform, false, 256, 1)
