// kf_kernels.cuh — fit kernels over the per-track lane (kf_fit.cuh).
//
// fitTracks: one thread per track, P.lanes tracks per warp.  With a queue
// counter a grid of the device's resident capacity whose warps claim their
// next tracks (sorted longest first) with one atomic until the queue is
// empty; without, warp w fits the w-th share.  launchFit chooses, for some
// sizes the kernel (unevenTracks).
//
// Lanes step independently and park at every plane they reach and at other
// heavy actor work (smoothing, final transport); when every lane of the warp
// is parked or done, the parked lanes run their events together, so the
// FP64-heavy Kalman algebra executes without divergence.  A lane whose plane
// has no hit waits too: passing it would put that lane a plane ahead, and its
// steps there would run with the others idle (tracks with 10 % holes: 1.24
// instead of 1.45 times the warp instructions of a track without divergence).
// Smoothing and the perigee come after the warp's last plane (eventDue).
//
// With P.align (the mixed form's queue) the eight warps of a block run each
// event together: the mixed kernel's code is larger than the instruction
// caches near the schedulers, and a third of its stalls were instruction
// fetches; warps in step share them (1M map tracks 44.8 -> 40.2 ms; stepping
// together too gave no more, and the FP64 forms, whose pipe is full, lose 1 %).
//
// The block size is a run-time value: an instantiation is a register budget,
// so that every shape of one budget, queue or not, gives the same bits.
#pragma once

#include "kf_fit_coop.cuh"

namespace kfd {

// Fit the tracks i (inputs/outputs) with workspace columns w of one warp;
// i < 0 marks an idle lane.  All 32 lanes must call it together.
// align: the block's warps run their events together (all must call).
template <int FORM, bool MAT, class H = NoHook>
__device__ __forceinline__ void fitWarp(const Params &P, const PlaneD *sp, int64_t i, int64_t w,
                                        bool align = false) {
  FitLane<FORM, MAT, H> L;
  initFit(L, P, sp, i, w);
  for (;;) {
    if (!L.parked && L.pc != PC_DONE) advance(L, P, sp);
    const bool waiting = L.parked || L.pc == PC_DONE;
    if (__all_sync(0xffffffffu, waiting)) {
      if (align) __syncthreads();
      if (eventDue(L)) runEvent(L, P, sp);
      if (align ? __syncthreads_and(L.pc == PC_DONE) : __all_sync(0xffffffffu, L.pc == PC_DONE)) break;
    }
  }
  if (i >= 0 && i < P.n && (threadIdx.x & (H::kGroup - 1)) == 0) {
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
}

// P.split (batches of 4 ... 8 warps an SM, sorted, one-warp blocks): are the
// tracks' lengths uneven enough to run one warp on each SM sub-partition,
// P.split in all, and let these claim the shorter rest as they finish, instead
// of giving some sub-partitions two warps from the start?  The queue's time is
// the longest warp's, or that of the shortest first one and what follows it, at
// a lone warp's 85 cycles per FP64 instruction; two warps that share a
// sub-partition take 65-70 each.  Measured (FP64 with smoothed states, lengths
// 5-30: 20011 tracks 1.56 -> 1.49 ms, 30000 1.80 -> 1.51, 38900 (the ratio below
// at 1.17) 1.99 -> 1.76; mixed, 30000 tracks 1.20 -> 0.98 ms); with one length
// (the ratio at 2) the queue would lose: uniform field 0.56 -> 0.59 and 0.73 ->
// 0.78 ms at 20011 and 38900 tracks, material 0.72 -> 0.87 ms at 20011.
__device__ __forceinline__ bool unevenTracks(const Params &P) {
  if (!P.nplanes) return false;
  auto length = [&](int64_t q) { return min(max(P.nplanes[P.perm[q]], 1), P.nSurf); };
  const int64_t last = 32 * (int64_t)P.split; // the first track past the first warps
  return last < P.n && 4 * (length(last - 1) + length(last)) <= 5 * length(0);
}

template <int FORM, bool MAT, int MAXT, int MINB>
__global__ void __launch_bounds__(MAXT, MINB) fitTracks(const __grid_constant__ Params P) {
  // the plane table behind the threads' columns
  PlaneD *sp = reinterpret_cast<PlaneD *>(kfColdSmem + (size_t)blockDim.x * coldSlots<MAT>() * sizeof(double));
  for (int k = threadIdx.x; k < P.nSurf; k += blockDim.x) sp[k] = P.planes[k];
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const bool align = P.align != 0;
  bool queue = P.queueCounter != nullptr;
  int lanes = P.lanes;
  if (P.split) {
    queue = unevenTracks(P);
    if (queue && blockIdx.x >= P.split) return;
    if (queue) lanes = 32;
  }
  __shared__ int claim;
  for (;;) {
    int64_t base;
    if (align) { // the block claims its next tracks together
      __syncthreads();
      if (threadIdx.x == 0) claim = atomicAdd(P.queueCounter, (int)blockDim.x);
      __syncthreads();
      if (claim >= P.n) break;
      base = claim + (threadIdx.x & ~31);
    } else if (queue) {
      int b = 0;
      if (lane == 0) b = atomicAdd(P.queueCounter, lanes);
      base = (int64_t)__shfl_sync(0xffffffffu, b, 0);
    } else {
      base = ((int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * lanes;
    }
    if (!align && base >= P.n) break;
    const int64_t q = base + lane;
    const bool own = lane < lanes && q < P.n;
    const int64_t i = own ? (P.perm ? (int64_t)P.perm[q] : q) : -1;
    fitWarp<FORM, MAT>(P, sp, i, own ? q : 0, align);
    if (!queue) break;
  }
}

// P.lanes (1 ... 4) tracks a warp, eight lanes each (kf_fit_coop.cuh).
template <int FORM> __global__ void __launch_bounds__(32, 8) fitCoop(const __grid_constant__ Params P) {
  PlaneD *sp = reinterpret_cast<PlaneD *>(kfColdSmem + (size_t)blockDim.x * coldSlots<false>() * sizeof(double));
  for (int k = threadIdx.x; k < P.nSurf; k += blockDim.x) sp[k] = P.planes[k];
  __syncthreads();
  const int g = threadIdx.x >> 3;
  const int64_t i = (int64_t)blockIdx.x * P.lanes + g;
  const bool own = g < P.lanes && i < P.n;
  fitWarp<FORM, false, CoopHook>(P, sp, own ? i : -1, own ? i : 0);
}

} // namespace kfd

#define KF_COOP_LAUNCHER(NAME, FORM)                                                           \
  cudaError_t NAME(const kfd::Params &P, int, cudaStream_t s) {                              \
    kfd::fitCoop<FORM><<<(unsigned)((P.n + P.lanes - 1) / P.lanes), 32, kfd::fitSmemBytes<false>(32, P.nSurf), s>>>(P); \
    return cudaGetLastError();                                                               \
  }

// Launcher of one instantiation: bs threads per block; with a queue as many
// blocks as the device holds at once, never more than the batch needs.
#define KF_FIT_LAUNCHER(NAME, FORM, MAT, MAXT, MINB)                                           \
  cudaError_t NAME(const kfd::Params &P, int bs, cudaStream_t s) {                           \
    auto *kernel = kfd::fitTracks<FORM, MAT, MAXT, MINB>;                                    \
    const size_t smem = kfd::fitSmemBytes<MAT>(bs, P.nSurf);                                 \
    cudaError_t e = cudaSuccess;                                                             \
    if (smem > 48 * 1024) /* above the default limit of dynamic shared memory */             \
      e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,          \
                               (int)kfd::fitSmemBytes<MAT>(MAXT, KF_MAX_PLANES));            \
    if (e != cudaSuccess) return e;                                                          \
    const int64_t per_block = (int64_t)(bs / 32) * P.lanes;                                  \
    const int64_t need = (P.n + per_block - 1) / per_block;                                  \
    int64_t blocks = need;                                                                   \
    if (P.queueCounter && !P.split) {                                                        \
      e = kfd::residentBlocks(kernel, bs, smem, blocks);                                     \
      if (e != cudaSuccess) return e;                                                        \
    }                                                                                        \
    if (blocks < 1) blocks = 1;                                                              \
    kernel<<<(unsigned)blocks, bs, smem, s>>>(P);                                            \
    return cudaGetLastError();                                                               \
  }
