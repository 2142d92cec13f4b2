// kf_launch.cu — which compiled fit kernel serves a call.
#include "kf_host.h"

#include <algorithm>

using kfd::Params;

#define KF_DECLARE(NAME) cudaError_t NAME(const Params &, int, cudaStream_t);
#define KF_DECLARE_BUDGET(R)              \
  KF_DECLARE(launchFit_fp64_uniform_##R)  \
  KF_DECLARE(launchFit_fp64_grid_##R)     \
  KF_DECLARE(launchFit_mixed_##R)         \
  KF_DECLARE(launchFit_mixed_uniform_##R)
KF_DECLARE_BUDGET(255)
KF_DECLARE_BUDGET(168)
KF_DECLARE_BUDGET(128)
KF_DECLARE_BUDGET(96)
KF_DECLARE(launchFit_fp64_any)
KF_DECLARE(launchFitMaterial_fp64_any)
KF_DECLARE(launchFitMaterial_fp64_uniform)
KF_DECLARE(launchFitMaterial_fp64_grid)
KF_DECLARE(launchFitMaterial_mixed)
KF_DECLARE(launchFitMaterial_mixed_uniform)
KF_DECLARE(launchFitCoop_fp64_uniform)
KF_DECLARE(launchFitCoop_fp64_grid)
KF_DECLARE(launchFitCoop_mixed)
KF_DECLARE(launchFitCoop_mixed_uniform)
KF_DECLARE(launchFitMaterialStates_fp64)
KF_DECLARE(launchFitMaterialStates_mixed)

namespace {

using Launch = cudaError_t (*)(const Params &, int, cudaStream_t);
struct Budget {
  Launch uniform, grid, mixedGrid, mixedUniform, anyField; // anyField: uniform, off the z axis
};
#define KF_BUDGET(R) \
  {launchFit_fp64_uniform_##R, launchFit_fp64_grid_##R, launchFit_mixed_##R,  \
   launchFit_mixed_uniform_##R, launchFit_fp64_any}
const Budget kBudget255 = KF_BUDGET(255), kBudget168 = KF_BUDGET(168), kBudget128 = KF_BUDGET(128),
             kBudget96 = KF_BUDGET(96);
const Budget kMaterial = {launchFitMaterial_fp64_uniform, launchFitMaterial_fp64_grid,
                          launchFitMaterial_mixed, launchFitMaterial_mixed_uniform,
                          launchFitMaterial_fp64_any};

struct Shape {
  int bs, minb;
  const Budget *budget;
};
// (threads per block, blocks per SM: the register budget that the kernel is
// compiled for; shared memory may hold fewer, of 128 x 5 four).  The first
// gives the budget of the library's own launches.
const Shape kShapes[] = {
    {128, 2, &kBudget255}, {64, 4, &kBudget255},  {256, 1, &kBudget255}, {128, 3, &kBudget168},
    {128, 4, &kBudget128}, {64, 8, &kBudget128},  {256, 2, &kBudget128}, {128, 5, &kBudget96},
};
// one-warp blocks spread over the SMs most evenly
constexpr int kDefaultBlock = 32, kQueueBlock = 256;

} // namespace

namespace kfh {

bool fitShape(int index, int *bs, int *minb) {
  if (index < 0 || index >= (int)(sizeof(kShapes) / sizeof(kShapes[0]))) return false;
  *bs = kShapes[index].bs;
  *minb = kShapes[index].minb;
  return true;
}

// the shape for a request: the first for (0, 0), else 0 stands for 128
// threads and for 4 blocks per SM
static const Shape *findShape(int bs, int minb) {
  if (!bs && !minb) return &kShapes[0];
  for (const Shape &s : kShapes)
    if (s.bs == (bs ? bs : 128) && s.minb == (minb ? minb : 4)) return &s;
  return nullptr;
}

bool shapeCompiled(int bs, int minb) { return findShape(bs, minb) != nullptr; }

// Rotate the planes into a frame with the field along z (kf_fit.cuh's uniform
// form); a field along +-z keeps the frame.
static void toFieldFrame(Params &P) {
  const double *B = P.field.B;
  for (int i = 0; i < 9; ++i) P.rot[i] = (i % 4 == 0) ? 1. : 0.;
  P.rotated = B[0] != 0. || B[1] != 0.;
  P.Bz = B[2];
  if (!P.rotated) return;
  // (by a power of two to about 1, so that no square leaves the range)
  const double big = std::fmax(std::fabs(B[0]), std::fmax(std::fabs(B[1]), std::fabs(B[2])));
  const int e = std::isfinite(big) ? std::ilogb(big) : 0;
  const double b[3] = {std::scalbn(B[0], -e), std::scalbn(B[1], -e), std::scalbn(B[2], -e)};
  const double n = std::sqrt(b[0] * b[0] + b[1] * b[1] + b[2] * b[2]);
  const double z[3] = {b[0] / n, b[1] / n, b[2] / n};
  // x axis: the coordinate axis least along z, made orthogonal to it
  int a = 0;
  for (int i = 1; i < 3; ++i)
    if (std::fabs(z[i]) < std::fabs(z[a])) a = i;
  double x[3] = {-z[a] * z[0], -z[a] * z[1], -z[a] * z[2]};
  x[a] += 1.;
  const double m = std::sqrt(x[0] * x[0] + x[1] * x[1] + x[2] * x[2]);
  for (double &v : x) v /= m;
  const double y[3] = {z[1] * x[2] - z[2] * x[1], z[2] * x[0] - z[0] * x[2], z[0] * x[1] - z[1] * x[0]};
  for (int i = 0; i < 3; ++i) {
    P.rot[i] = x[i];
    P.rot[3 + i] = y[i];
    P.rot[6 + i] = z[i];
  }
  P.Bz = std::scalbn(n, e);
  auto turn = [&](double v[3]) {
    double o[3];
    for (int i = 0; i < 3; ++i)
      o[i] = P.rot[3 * i] * v[0] + P.rot[3 * i + 1] * v[1] + P.rot[3 * i + 2] * v[2];
    for (int i = 0; i < 3; ++i) v[i] = o[i];
  };
  for (int k = 0; k < P.nSurf; ++k) {
    turn(P.planes[k].c);
    turn(P.planes[k].U);
    turn(P.planes[k].V);
    turn(P.planes[k].T); // (T . c is unchanged)
  }
}

constexpr int64_t kLeastWarps = 3; // warps an SM that a small batch spreads over
constexpr int64_t kFillWarps = 4;  // one on each SM sub-partition

// How a batch is laid over the chip.  One FP64 instruction of a warp costs the
// same whatever its active lanes, each SM sub-partition starts one every 64
// cycles, and four warps (one a sub-partition) fill an SM's FP64 pipe.  So a
// batch first spreads over 3 warps on every SM with as few tracks a warp as
// that takes (fewer lanes to wait for: 1000 map tracks mixed, one lane a track,
// 1530 -> 1393 us; such batches now run eight lanes a track, kCoopMost, and
// this serves the ones that cannot), then over 4 ... 8 of them, the kernel's
// residency (from 5 on the kernel may take a queue of 4 instead,
// unevenTracks); beyond that warps of 32 tracks claim work from the queue.
// Sorting (3 small kernels, 15 us) pays from 8 tracks a warp on.
struct Spread {
  int lanes;  // tracks per warp
  bool sort;  // order the tracks by expected work
  bool queue; // more warps than the chip holds
};
static Spread spread(int64_t n, int sms) {
  if (n > 0x7f000000) return {32, false, false}; // the queue counts in 32 bits
  const bool room = n > kSortBuckets + 16;       // for the sort's counts (kf_fit_batch)
  const int64_t full = 32 * (int64_t)sms;
  const int64_t perSm = std::max<int64_t>(kLeastWarps, (n + full - 1) / full);
  if (perSm > 8) return {32, room, room};
  const int lanes = (int)((n + sms * perSm - 1) / (sms * perSm));
  return {lanes, room && lanes >= 8, false};
}

bool launchesAShape(int64_t n) {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return true;
  return spread(n, sms).queue;
}

// Batches of up to kCoopMost tracks an SM run eight lanes a track, again as few
// tracks a warp as kLeastWarps warps an SM allow (the line is at five such
// warps of four tracks an SM: 3040 tracks of 10 planes 361 us, 3041 one lane a
// track 449 us; in the field map 1.86 and 2.25 ms, mixed 1.08 and 1.23 ms).
constexpr int64_t kCoopMost = 20;

int32_t launchFit(Params &P, int precision, int bs, int minb, const QueueBuffers &q, cudaStream_t s) {
  const bool mixed = precision == KF_PRECISION_MIXED;
  const Shape *shape = findShape(bs, minb);
  if (!shape) return fail(KF_ERR_UNSUPPORTED, "no fit kernel for this block size / blocks per SM%s");
  cudaError_t e;
  P.lanes = 32;
  P.split = 0;
  if (P.materialEffects && P.oSmoothed) {
    if (q.apart) { // (this form's records leave no words for the plain call to sort in)
      const int32_t rc = sortQueue(P, q.hist, q.offs, q.perm, q.counter, s);
      if (rc) return rc;
      P.perm = q.perm;
      P.queueCounter = q.counter;
    }
    e = (mixed ? launchFitMaterialStates_mixed : launchFitMaterialStates_fp64)(P, 0, s);
    return e == cudaSuccess ? KF_SUCCESS : cudaFail(e, "fit kernel launch");
  }
  int dev = 0, sms = 0;
  e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return cudaFail(e, "device query");
  const bool asked = (bs || minb) && !P.materialEffects; // a requested shape: always the queue
  const bool uniform = P.field.kind == KF_FIELD_CONSTANT;
  const bool offAxis = !mixed && uniform && (P.field.B[0] != 0. || P.field.B[1] != 0.);
  if (!asked && !P.materialEffects && !P.oSmoothed && !offAxis && P.n <= kCoopMost * sms) {
    if (!mixed && uniform) toFieldFrame(P);
    P.lanes = (int)std::min<int64_t>(4, (P.n + kLeastWarps * sms - 1) / (kLeastWarps * sms));
    e = (mixed ? (uniform ? launchFitCoop_mixed_uniform : launchFitCoop_mixed)
               : (uniform ? launchFitCoop_fp64_uniform : launchFitCoop_fp64_grid))(P, 0, s);
    return e == cudaSuccess ? KF_SUCCESS : cudaFail(e, "fit kernel launch");
  }
  Spread sp = spread(P.n, sms);
  if (asked) sp = {32, sp.sort || P.n > kSortBuckets + 16, P.n > kSortBuckets + 16};
  P.lanes = sp.lanes;
  if (sp.sort) {
    const int32_t rc = sortQueue(P, q.hist, q.offs, q.perm, q.counter, s);
    if (rc) return rc;
    P.perm = q.perm;
  }
  if (!sp.queue && sp.sort && P.n > kFillWarps * 32 * sms) P.split = (int)(kFillWarps * sms);
  if (sp.queue || P.split) P.queueCounter = q.counter;
  const Budget *b = P.materialEffects ? &kMaterial : shape->budget;
  // with a queue one block of 8 warps an SM (2 % over one-warp blocks: warps
  // that start together share instruction fetches)
  const int block = asked ? shape->bs : sp.queue ? kQueueBlock : kDefaultBlock;
  P.align = sp.queue && mixed && block == kQueueBlock && !P.materialEffects;
  if (mixed) {
    e = (uniform ? b->mixedUniform : b->mixedGrid)(P, block, s);
  } else if (!uniform) {
    e = b->grid(P, block, s);
  } else {
    toFieldFrame(P);
    e = (P.rotated ? b->anyField : b->uniform)(P, block, s);
  }
  return e == cudaSuccess ? KF_SUCCESS : cudaFail(e, "fit kernel launch");
}

} // namespace kfh
