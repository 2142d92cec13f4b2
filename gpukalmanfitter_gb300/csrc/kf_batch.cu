// kf_batch.cu — the work queue (tracks sorted by expected work), and the
// batched form: CUDA-graph plan and autotuner.
//
// The reference fits one track per GPU thread or block with one launch per
// stream (Run/GPU/Kernels.cu:6-94, Run/GPU/KalmanFitterGPUTest.cu:461-472); tracks
// of very different length share warps and the grid's tail idles.  Here the
// tracks are first ordered by expected work (sequence length, then |q/p|),
// longest first, by a counting sort over 2048 buckets (batches of more than a
// few thousand tracks, see launchFit); warps of a persistent
// grid then claim 32 consecutive queue positions at a time, so a warp holds
// tracks of similar length and the longest tracks start first.

#include <cuda_runtime.h>

#include <cstdio>
#include <cstring>
#include <new>

#include "kf_host.h"

using namespace kfd;
using namespace kfh;

namespace {

constexpr int kBuckets = kSortBuckets;

size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

struct BatchLayout {
  size_t ws, perm, hist, offs, counter, total;
};
BatchLayout batchLayout(int64_t n, int32_t S, bool material) {
  BatchLayout L{};
  size_t o = 0;
  auto take = [&](size_t bytes) {
    const size_t at = o;
    o = align256(o + bytes);
    return at;
  };
  L.ws = take(wsBytes(n, S, material));
  L.perm = take((size_t)n * sizeof(int32_t));
  L.hist = take(kBuckets * sizeof(int32_t));
  L.offs = take(kBuckets * sizeof(int32_t));
  L.counter = take(sizeof(int32_t));
  L.total = o;
  return L;
}

// Ascending key = descending expected work: sequence length first, then
// |q/p| in quarter octaves (a track's RK steps between planes grow with its
// curvature, and a warp takes as many as its slowest lane).
__device__ __forceinline__ int workKey(const Params &P, int64_t i) {
  int L = P.nplanes ? P.nplanes[i] : P.nSurf;
  L = min(max(L, 1), P.nSurf);
  const float qop = (float)fabs(P.start[4 * P.stride + i]);
  int qb = 0;
  if (qop > 0.f && qop < 3.0e38f) qb = (int)floorf((log2f(qop) + 7.f) * 4.f);
  qb = min(max(qb, 0), 31);
  return (64 - L) * 32 + (31 - qb);
}

// The sort's tracks fall into few buckets (one length: a dozen), so counts
// and ranks are formed per block in shared memory; a global atomic per
// bucket and block instead of per track (1M tracks: 0.4 ms -> 0.03 ms).
constexpr int kSortThreads = 256, kSortItems = 16;

__global__ void __launch_bounds__(kSortThreads) keyHistogram(const __grid_constant__ Params P, int32_t *hist) {
  __shared__ int32_t h[kBuckets];
  for (int b = threadIdx.x; b < kBuckets; b += kSortThreads) h[b] = 0;
  __syncthreads();
  const int64_t first = (int64_t)blockIdx.x * (kSortThreads * kSortItems) + threadIdx.x;
#pragma unroll
  for (int k = 0; k < kSortItems; ++k) {
    const int64_t i = first + (int64_t)k * kSortThreads;
    if (i < P.n) atomicAdd(&h[workKey(P, i)], 1);
  }
  __syncthreads();
  for (int b = threadIdx.x; b < kBuckets; b += kSortThreads)
    if (h[b]) atomicAdd(&hist[b], h[b]);
}

// exclusive scan of kBuckets counts by one CTA of 1024 threads; resets the
// queue's counter if there is one
__global__ void __launch_bounds__(1024) scanOffsets(const int32_t *hist, int32_t *offs, int32_t *counter) {
  __shared__ int32_t part[1024];
  const int t = threadIdx.x;
  if (t == 0 && counter) *counter = 0;
  const int a = hist[2 * t], b = hist[2 * t + 1];
  part[t] = a + b;
  __syncthreads();
  for (int d = 1; d < 1024; d <<= 1) {
    const int v = (t >= d) ? part[t - d] : 0;
    __syncthreads();
    part[t] += v;
    __syncthreads();
  }
  const int before = part[t] - (a + b);
  offs[2 * t] = before;
  offs[2 * t + 1] = before + a;
}

__global__ void __launch_bounds__(kSortThreads) scatterPerm(const __grid_constant__ Params P, int32_t *offs, int32_t *perm) {
  __shared__ int32_t h[kBuckets];
  for (int b = threadIdx.x; b < kBuckets; b += kSortThreads) h[b] = 0;
  __syncthreads();
  const int64_t first = (int64_t)blockIdx.x * (kSortThreads * kSortItems) + threadIdx.x;
  int key[kSortItems], rank[kSortItems];
#pragma unroll
  for (int k = 0; k < kSortItems; ++k) {
    const int64_t i = first + (int64_t)k * kSortThreads;
    key[k] = -1;
    if (i < P.n) {
      key[k] = workKey(P, i);
      rank[k] = atomicAdd(&h[key[k]], 1);
    }
  }
  __syncthreads();
  for (int b = threadIdx.x; b < kBuckets; b += kSortThreads)
    if (h[b]) h[b] = atomicAdd(&offs[b], h[b]);
  __syncthreads();
#pragma unroll
  for (int k = 0; k < kSortItems; ++k)
    if (key[k] >= 0) perm[h[key[k]] + rank[k]] = (int32_t)(first + (int64_t)k * kSortThreads);
}

} // namespace

int32_t kfh::sortQueue(const Params &P, int32_t *hist, int32_t *offs, int32_t *perm,
                       int32_t *counter, cudaStream_t s) {
  if (P.n == 0) return KF_SUCCESS;
  cudaError_t e = cudaMemsetAsync(hist, 0, kBuckets * sizeof(int32_t), s);
  if (e != cudaSuccess) return cudaFail(e, "work-queue reset");
  const unsigned g = (unsigned)((P.n + kSortThreads * kSortItems - 1) / (kSortThreads * kSortItems));
  keyHistogram<<<g, kSortThreads, 0, s>>>(P, hist);
  scanOffsets<<<1, 1024, 0, s>>>(hist, offs, counter);
  scatterPerm<<<g, kSortThreads, 0, s>>>(P, offs, perm);
  e = cudaGetLastError();
  return e == cudaSuccess ? KF_SUCCESS : cudaFail(e, "work-queue sort");
}

namespace {

int32_t enqueueBatched(Params &P, const kf_config_t *cfg, char *base, const BatchLayout &L,
                       cudaStream_t s) {
  if (P.n == 0) return KF_SUCCESS;
  HostRange range("work-queue sort + persistent fit");
  QueueBuffers q;
  q.perm = reinterpret_cast<int32_t *>(base + L.perm);
  q.hist = reinterpret_cast<int32_t *>(base + L.hist);
  q.offs = reinterpret_cast<int32_t *>(base + L.offs);
  q.counter = reinterpret_cast<int32_t *>(base + L.counter);
  q.apart = true;
  // with material effects the shape fields say nothing (prepare), whether the
  // geometry has material or not
  const bool shape = !cfg->material_effects;
  return launchFit(P, cfg->precision, shape ? cfg->block_size : 0, shape ? cfg->min_blocks_per_sm : 0, q, s);
}

int32_t prepare(const kf_inputs_t *in, kf_outputs_t *out, const kf_config_t *cfg,
                const kf_geometry_t *geo, const kf_field_t *field, void *workspace,
                size_t bytes, Params &P, BatchLayout &L) {
  int32_t rc = checkCommon(in, cfg, geo, field);
  if (rc) return rc;
  if (!out || !out->params || !out->cov || !out->chi2 || !out->status || !out->n_meas)
    return fail(KF_ERR_INVALID_ARGUMENT, "missing output array%s");
  if (in->n_tracks > 0 && (!in->meas || !in->start_params || !in->start_cov || !in->perigee))
    return fail(KF_ERR_INVALID_ARGUMENT, "missing input array%s");
  // the int32 queue counter runs up to n + 32 x (resident warps)
  if (in->n_tracks > 0x7f000000LL) return fail(KF_ERR_INVALID_ARGUMENT, "batch above 2^31 - 2^24 tracks%s");
  // with material effects there is one shape, whatever the fields say
  if (!cfg->material_effects && !shapeCompiled(cfg->block_size, cfg->min_blocks_per_sm))
    return fail(KF_ERR_UNSUPPORTED, "no persistent kernel for this block size / CTAs per SM%s");
  L = batchLayout(in->n_tracks, in->n_surfaces, cfg->material_effects != 0);
  if (in->n_tracks > 0 && (!workspace || bytes < L.total))
    return fail(KF_ERR_WORKSPACE_TOO_SMALL, "workspace smaller than kf_batch_workspace_size()%s");
  char *base = static_cast<char *>(workspace);
  fillParams(P, in, out, cfg, geo, field, base + L.ws);
  return KF_SUCCESS;
}

} // namespace

struct kf_batch_plan {
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
};

extern "C" {

size_t kf_batch_workspace_size(const kf_config_t *cfg, int64_t n_tracks, int32_t n_surfaces) {
  (void)cfg;
  if (n_tracks <= 0 || n_surfaces <= 0) return 0;
  return batchLayout(n_tracks, n_surfaces, cfg && cfg->material_effects).total;
}

int32_t kf_fit_batch_sorted(const kf_inputs_t *in, kf_outputs_t *out, const kf_config_t *cfg,
                            const kf_geometry_t *geo, const kf_field_t *field, void *workspace,
                            size_t workspace_bytes, void *stream) {
  Params P;
  BatchLayout L;
  int32_t rc = prepare(in, out, cfg, geo, field, workspace, workspace_bytes, P, L);
  if (rc) return rc;
  return enqueueBatched(P, cfg, static_cast<char *>(workspace), L, static_cast<cudaStream_t>(stream));
}

int32_t kf_batch_plan_create(kf_batch_plan_t **plan, const kf_inputs_t *in, kf_outputs_t *out,
                             const kf_config_t *cfg, const kf_geometry_t *geo,
                             const kf_field_t *field, void *workspace, size_t workspace_bytes,
                             void *stream) {
  if (!plan) return fail(KF_ERR_INVALID_ARGUMENT, "null plan pointer%s");
  *plan = nullptr;
  if (!stream) return fail(KF_ERR_INVALID_ARGUMENT, "a plan needs a created stream (not the legacy default stream)%s");
  Params P;
  BatchLayout L;
  int32_t rc = prepare(in, out, cfg, geo, field, workspace, workspace_bytes, P, L);
  if (rc) return rc;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  cudaError_t e = cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal);
  if (e != cudaSuccess) return cudaFail(e, "stream capture begin");
  rc = enqueueBatched(P, cfg, static_cast<char *>(workspace), L, s);
  cudaGraph_t graph = nullptr;
  e = cudaStreamEndCapture(s, &graph);
  if (rc) {
    if (graph) cudaGraphDestroy(graph);
    return rc;
  }
  if (e != cudaSuccess) return cudaFail(e, "stream capture end");
  cudaGraphExec_t exec = nullptr;
  e = cudaGraphInstantiate(&exec, graph, 0);
  if (e != cudaSuccess) {
    cudaGraphDestroy(graph);
    return cudaFail(e, "graph instantiate");
  }
  kf_batch_plan *p = new (std::nothrow) kf_batch_plan;
  if (!p) {
    cudaGraphExecDestroy(exec);
    cudaGraphDestroy(graph);
    return fail(KF_ERR_INVALID_ARGUMENT, "out of host memory%s");
  }
  p->graph = graph;
  p->exec = exec;
  *plan = p;
  return KF_SUCCESS;
}

int32_t kf_batch_plan_launch(kf_batch_plan_t *plan, void *stream) {
  HostRange range("kf_batch_plan_launch");
  if (!plan || !plan->exec) return fail(KF_ERR_INVALID_ARGUMENT, "null plan%s");
  cudaError_t e = cudaGraphLaunch(plan->exec, static_cast<cudaStream_t>(stream));
  if (e != cudaSuccess) return cudaFail(e, "graph launch");
  return KF_SUCCESS;
}

void kf_batch_plan_destroy(kf_batch_plan_t *plan) {
  if (!plan) return;
  if (plan->exec) cudaGraphExecDestroy(plan->exec);
  if (plan->graph) cudaGraphDestroy(plan->graph);
  delete plan;
}

int32_t kf_autotune(const kf_inputs_t *in, kf_outputs_t *out, const kf_config_t *cfg,
                    const kf_geometry_t *geo, const kf_field_t *field, void *workspace,
                    size_t workspace_bytes, void *stream, kf_config_t *tuned, double *best_ms) {
  if (!in || !cfg || !tuned) return fail(KF_ERR_INVALID_ARGUMENT, "null argument%s");
  HostRange range("kf_autotune");
  // The first tracks (same stride) as the sample: at least several waves of
  // the resident grid, so that the queue's tail does not decide the timing.
  kf_inputs_t sample = *in;
  if (sample.n_tracks > 524288) sample.n_tracks = 524288;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  cudaEvent_t e0, e1;
  if (cudaEventCreate(&e0) != cudaSuccess || cudaEventCreate(&e1) != cudaSuccess)
    return cudaFail(cudaGetLastError(), "event create");
  double best = 1e300;
  kf_config_t bestCfg = *cfg;
  int32_t rc = KF_SUCCESS;
  int bs = 0, minb = 0;
  // the library's own launch first, where it is none of the shapes; with
  // material effects there is one shape
  const bool own = !cfg->material_effects && !launchesAShape(sample.n_tracks);
  for (int v = own ? -1 : 0; v < 0 || (fitShape(v, &bs, &minb) && (v == 0 || !cfg->material_effects)); ++v) {
    kf_config_t c = *cfg;
    c.kernel = KF_KERNEL_PERSISTENT;
    c.block_size = bs;
    c.min_blocks_per_sm = minb;
    rc = kf_fit_batch_sorted(&sample, out, &c, geo, field, workspace, workspace_bytes, stream);
    // best of three timed runs after one warm-up
    for (int r = 0; r < 3 && rc == KF_SUCCESS; ++r) {
      cudaEventRecord(e0, s);
      rc = kf_fit_batch_sorted(&sample, out, &c, geo, field, workspace, workspace_bytes, stream);
      cudaEventRecord(e1, s);
      if (rc) break;
      if (cudaEventSynchronize(e1) != cudaSuccess) {
        rc = cudaFail(cudaGetLastError(), "autotune timing");
        break;
      }
      float ms = 0.f;
      cudaEventElapsedTime(&ms, e0, e1);
      if (ms < best) {
        best = ms;
        bestCfg = c;
      }
    }
    if (rc) break;
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (rc) return rc;
  *tuned = bestCfg;
  if (best_ms) *best_ms = best;
  return KF_SUCCESS;
}

} // extern "C"
