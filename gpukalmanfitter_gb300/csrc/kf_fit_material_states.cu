// kf_fit_material_states.cu — fit kernels with surface material effects that
// return every smoothed state: the lane of kf_device.cuh, which stores each
// state's predicted and filtered covariance, and the general gain-matrix
// smoother over them.  One launch shape (128 threads, 4 blocks per SM).
#include <cuda_runtime.h>

#include "kf_device.cuh"

namespace kfd {

template <typename R>
__global__ void __launch_bounds__(kLaneSlots, 4) fitMaterialStates(const __grid_constant__ Params P) {
  using H = MaterialHook;
  __shared__ PlaneD sp[KF_MAX_PLANES];
  for (int k = threadIdx.x; k < P.nSurf; k += blockDim.x) sp[k] = P.planes[k];
  __syncthreads();
  const int64_t w = (int64_t)blockIdx.x * kLaneSlots + threadIdx.x;
  const int64_t i = (w < P.n) ? (P.perm ? (int64_t)P.perm[w] : w) : -1;
  Lane<R, H> L;
  initLane(L, P, sp, i, w < P.n ? w : 0);
  for (;;) {
    if (!L.parked && L.pc != PC_DONE) advance(L, P, sp);
    const bool waiting = L.parked || L.pc == PC_DONE;
    if (__all_sync(0xffffffffu, waiting)) {
      if (L.parked) runEvent(L, P, sp);
      if (__all_sync(0xffffffffu, L.pc == PC_DONE)) break;
    }
  }
  if (i < 0) return;
  P.oStatus[i] = L.status;
  P.oChi2[i] = L.chi2;
  P.oNMeas[i] = L.measStates;
  if (P.oNSteps) P.oNSteps[i] = L.rkSteps;
  if (P.oNTrials) P.oNTrials[i] = L.rkTrials;
  if (L.status != KF_TRACK_OK && !L.finished) {
    for (int e = 0; e < 6; ++e) P.oParams[(size_t)e * P.stride + i] = 0.;
    for (int e = 0; e < 21; ++e) P.oCov[(size_t)e * P.stride + i] = 0.;
  }
}

} // namespace kfd

#define KF_STATES_LAUNCHER(NAME, R)                                                            \
  cudaError_t NAME(const kfd::Params &P, int, cudaStream_t s) {                              \
    const unsigned grid = (unsigned)((P.n + kfd::kLaneSlots - 1) / kfd::kLaneSlots);         \
    kfd::fitMaterialStates<R><<<grid, kfd::kLaneSlots, kfd::coldStateBytes<R>(), s>>>(P);    \
    return cudaGetLastError();                                                               \
  }

KF_STATES_LAUNCHER(launchFitMaterialStates_fp64, double)
KF_STATES_LAUNCHER(launchFitMaterialStates_mixed, float)
