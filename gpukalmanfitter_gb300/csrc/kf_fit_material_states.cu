// kf_fit_material_states.cu — fit kernels with surface material effects that
// return every smoothed state: the lane of kf_device.cuh, which stores each
// state's predicted and filtered covariance, and the general gain-matrix
// smoother over them.  One launch shape (128 threads, 4 blocks per SM).
#include <cuda_runtime.h>

#include "kf_device.cuh"

namespace kfd {

// With P.queueCounter a grid of the device's resident capacity whose warps
// claim their next 32 tracks in P.perm's order; without, warp w fits the w-th
// 32, in P.perm's order where the lengths differ (tracks of one length would
// be gathered by curvature only, and the warp of the most curved ones be the
// longest: 300 tracks in a map 15.2 -> 16.5 ms).
template <typename R>
__global__ void __launch_bounds__(kLaneSlots, 4) fitMaterialStates(const __grid_constant__ Params P) {
  using H = MaterialHook;
  __shared__ PlaneD sp[KF_MAX_PLANES];
  for (int k = threadIdx.x; k < P.nSurf; k += blockDim.x) sp[k] = P.planes[k];
  __syncthreads();
  const int lane = threadIdx.x & 31;
  for (;;) {
    int64_t base = (int64_t)blockIdx.x * kLaneSlots + (threadIdx.x & ~31);
    if (P.queueCounter) {
      int b = 0;
      if (lane == 0) b = atomicAdd(P.queueCounter, 32);
      base = (int64_t)__shfl_sync(0xffffffffu, b, 0);
    }
    if (base >= P.n) return;
    const int64_t w = base + lane;
    auto length = [&](int64_t q) { return min(max(P.nplanes[P.perm[q]], 0), P.nSurf); };
    const bool ordered =
        P.perm && (P.queueCounter || (P.nplanes && length(0) != length(P.n - 1)));
    const int64_t i = (w < P.n) ? (ordered ? (int64_t)P.perm[w] : w) : -1;
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
    if (i >= 0) {
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
    if (!P.queueCounter) return;
  }
}

} // namespace kfd

// A sorted batch that fits on the device takes static shares: its blocks start
// longest first, and those of the shortest tracks share an SM with another
// (lengths 5-30, 20011 tracks: 15.3 ms, through a queue 19.3).  A larger one
// takes the queue (100003 tracks of one length 60.6 ms, static shares 66.9; of
// lengths 5-30 35.4 and 31.1).
namespace {
template <typename R> cudaError_t launchStates(kfd::Params P, cudaStream_t s) {
  const int64_t need = (P.n + kfd::kLaneSlots - 1) / kfd::kLaneSlots;
  const size_t smem = kfd::coldStateBytes<R>();
  int64_t grid = need;
  if (P.queueCounter) {
    const cudaError_t e = kfd::residentBlocks(kfd::fitMaterialStates<R>, kfd::kLaneSlots, smem, grid);
    if (e != cudaSuccess) return e;
    if (grid == need) P.queueCounter = nullptr;
  }
  kfd::fitMaterialStates<R><<<(unsigned)grid, kfd::kLaneSlots, smem, s>>>(P);
  return cudaGetLastError();
}
} // namespace

cudaError_t launchFitMaterialStates_fp64(const kfd::Params &P, int, cudaStream_t s) {
  return launchStates<double>(P, s);
}
cudaError_t launchFitMaterialStates_mixed(const kfd::Params &P, int, cudaStream_t s) {
  return launchStates<float>(P, s);
}
