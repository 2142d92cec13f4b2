// kf_launch.cu — which compiled fit kernel serves a call.
#include "kf_host.h"

using kfd::Params;

#define KF_DECLARE(NAME) cudaError_t NAME(const Params &, int, cudaStream_t);
#define KF_DECLARE_BUDGET(R)              \
  KF_DECLARE(launchFit_fp64_uniform_##R)  \
  KF_DECLARE(launchFit_fp64_grid_##R)     \
  KF_DECLARE(launchFit_mixed_##R)
KF_DECLARE_BUDGET(255)
KF_DECLARE_BUDGET(168)
KF_DECLARE_BUDGET(128)
KF_DECLARE_BUDGET(96)
KF_DECLARE(launchFit_fp64_any)
KF_DECLARE(launchFitMaterial_fp64_any)
KF_DECLARE(launchFitMaterial_fp64_uniform)
KF_DECLARE(launchFitMaterial_fp64_grid)
KF_DECLARE(launchFitMaterial_mixed)
KF_DECLARE(launchFitMaterialStates_fp64)
KF_DECLARE(launchFitMaterialStates_mixed)

namespace {

using Launch = cudaError_t (*)(const Params &, int, cudaStream_t);
struct Budget {
  Launch uniform, grid, mixed, anyField; // anyField: a uniform field off the z axis
};
#define KF_BUDGET(R) \
  {launchFit_fp64_uniform_##R, launchFit_fp64_grid_##R, launchFit_mixed_##R, launchFit_fp64_any}
const Budget kBudget255 = KF_BUDGET(255), kBudget168 = KF_BUDGET(168), kBudget128 = KF_BUDGET(128),
             kBudget96 = KF_BUDGET(96);
const Budget kMaterial = {launchFitMaterial_fp64_uniform, launchFitMaterial_fp64_grid,
                          launchFitMaterial_mixed, launchFitMaterial_fp64_any};

struct Shape {
  int bs, minb;
  const Budget *budget;
};
// (threads per block, blocks per SM); the first is the default
const Shape kShapes[] = {
    {128, 2, &kBudget255}, {64, 4, &kBudget255},  {256, 1, &kBudget255}, {128, 3, &kBudget168},
    {128, 4, &kBudget128}, {64, 8, &kBudget128},  {256, 2, &kBudget128}, {128, 5, &kBudget96},
};
constexpr int kPlainBlock = 32;

} // namespace

namespace kfh {

bool fitShape(int index, int *bs, int *minb) {
  if (index < 0 || index >= (int)(sizeof(kShapes) / sizeof(kShapes[0]))) return false;
  *bs = kShapes[index].bs;
  *minb = kShapes[index].minb;
  return true;
}

// the shape for a request: the default for (0, 0), else 0 stands for 128
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
  const double n = std::sqrt(B[0] * B[0] + B[1] * B[1] + B[2] * B[2]);
  const double z[3] = {B[0] / n, B[1] / n, B[2] / n};
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
  P.Bz = n;
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

cudaError_t launchFit(Params &P, int precision, int bs, int minb, cudaStream_t s) {
  const bool plain = P.queueCounter == nullptr;
  const bool mixed = precision == KF_PRECISION_MIXED;
  const Shape *shape = plain ? &kShapes[0] : findShape(bs, minb);
  if (!shape) return cudaErrorInvalidValue;
  if (P.materialEffects && P.oSmoothed)
    return (mixed ? launchFitMaterialStates_mixed : launchFitMaterialStates_fp64)(P, 0, s);
  const Budget *b = P.materialEffects ? &kMaterial : shape->budget;
  const int block = plain ? kPlainBlock : (P.materialEffects ? kShapes[0].bs : shape->bs);
  if (mixed) return b->mixed(P, block, s);
  if (P.field.kind != KF_FIELD_CONSTANT) return b->grid(P, block, s);
  toFieldFrame(P);
  return (P.rotated ? b->anyField : b->uniform)(P, block, s);
}

} // namespace kfh
