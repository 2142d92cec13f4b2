// kf_fit_mixed_96.cu — mixed fit kernels with up to 96 registers a thread
// (threads per block x blocks per SM: 128 x 5, of which shared memory holds four).
#include <cuda_runtime.h>

#include "kf_kernels.cuh"

KF_FIT_LAUNCHER(launchFit_mixed_96, kfd::kMixed, false, 128, 5)
KF_FIT_LAUNCHER(launchFit_mixed_uniform_96, kfd::kMixedUniform, false, 128, 5)
