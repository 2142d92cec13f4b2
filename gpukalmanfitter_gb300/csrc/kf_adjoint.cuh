// kf_adjoint.cuh — what the two kernels of the chi2 adjoint share: their
// parameters and the tape's records.
#pragma once

#include <cuda_runtime.h>

#include "kf_device.cuh"

namespace kfd {
namespace adj {

enum { REC_STEP = 1, REC_ACT = 2, REC_HIT = 3 };

struct AdjParams {
  const int32_t *perm; // [n] queue position -> track
  double *stateBar;  // [S][37][n] adjoints of predicted, filtered, Jacobian (by position)
  double *xs;        // [S][6][n] smoothed parameters (by position)
  int32_t *info;     // [S][n] plane index | outlier << 8 (by position)
  double *snap;      // [nCk][kSnapWords][n] (by position)
  double *tape;      // [tapeCap][n] (by position: a warp's lanes at the same tape
                     // offset touch one contiguous line)
  int tapeCap;       // tape words per track
  int fwdTape;       // the forward records the whole track's tape
  double *alignPart; // [S][6][n] (by track)
  double *trackFs;   // [n] per-track d chi2 / d field scale (by track)
  double *chi2;      // [n]
  int32_t *status;   // [n]
  double *gradStart; // [6][stride] or null
  double B0[3];      // field value before scaling
  int grad;
  int onlyMarked;    // adjointKernel: the tracks with status kLeft only
};
constexpr int32_t kLeft = -1; // status of a track that adjointZ leaves to adjointKernel

// kf_adjoint_z.cu
cudaError_t launchAdjointZ(const Params &P, const AdjParams &A, cudaStream_t s);


__device__ __forceinline__ double hdr(int type, int len) { return (double)(type * 65536 + len); }

// a lane's tape: word k at p[k * n]
struct TapeRef {
  const double *p;
  int64_t n;
  // each word is read once: a streaming load, so that the tape passing
  // through does not evict the spilled registers and state arrays from L2
  __device__ __forceinline__ double operator[](int k) const { return __ldcs(p + (int64_t)k * n); }
  __device__ __forceinline__ TapeRef operator+(int k) const { return {p + (int64_t)k * n, n}; }
};

} // namespace adj
} // namespace kfd
