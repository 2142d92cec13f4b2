// kf_fit_fp64_any.cu — FP64 fit kernel for a uniform field off the z axis, up
// to 255 registers a thread (it serves every launch shape).
#include <cuda_runtime.h>

#include "kf_kernels.cuh"

KF_FIT_LAUNCHER(launchFit_fp64_any, kfd::kUniformAny, false, 256, 1)
