// kf_fit.cuh — the fit program of one track: the lane that the fit kernels
// run (kf_kernels.cuh).
//
// The control flow (propagation loop, navigation, step constraints, actor and
// aborters) is kf_device.cuh's; this file holds the lane's RK step, the
// measurement update, the smoothed first state and the transport to the
// perigee line, in a form that needs no smoother pass and no covariance
// transport per plane.
//
// FP64 is what bounds these kernels: one FP64 instruction of a warp holds the
// SM's FP64 pipe for 16 cycles (19 measured) whatever its active lanes, an
// SM sub-partition starts one every 64, and conversions from FP32 cost the
// same, while FP32, integer and memory instructions are nearly free next to
// it.  So the aim throughout is fewer FP64 instructions per track:
//
//  * Covariance in the start frame (no process noise).  With F = J_k ... J_1
//    the accumulated bound-to-bound Jacobian, the reference's predicted
//    covariance J C J^T and filtered covariance (I - KH) C
//    (CovarianceEngine.hpp:269-290, GainMatrixUpdater.hpp:77-84) are
//    F C0 F^T, where C0 starts as the start covariance and every hit takes
//    off the rank-2 term of its measurement h = (first two rows of F).  The
//    gain-matrix smoother's gain is then J^-1 (GainMatrixSmoother.hpp:21-94
//    with C_p' = J C_f J^T), so that a state's smoothed parameters are
//    x_s = x_p + F sum K0 r over this and all later hits and its covariance
//    F C0 F^T with the final C0: the smoother is a running sum (D), and
//    neither states nor Jacobians need storing.  Per hit 84 (F) + 160
//    instead of 145 (J C J^T) + 65 (update) + 200 (smoother) FP64
//    instructions, and none of the 592 bytes per state the smoother pass
//    wrote and read back.
//  * With process noise (material) the smoothed first state is a fixed-point
//    smoother: its covariance with the current state, X, is carried along
//    (X <- X J^T, X <- X - K_x H C) next to the current covariance, which
//    equals the reference's RTS gains multiplied out
//    (C_f J^T C_p'^-1 ... = X C_p^-1).  No inverse of a 6x6 covariance.
//  * The arrival time is no part of any measurement: its row is carried only
//    where a caller reads it (the first state, or smoothed states), and its
//    covariance with the others only if the start covariance has one.
//  * Uniform field: the step's transport matrix is a polynomial in the cross
//    product with the field, and these commute, so in a frame with the field
//    along z a leg's transport Jacobian is 5 scalars and the q/p column 2 + 2
//    (stepUniform): 66 instead of 250 FP64 instructions a step.
//  * Field map: the leg's three direction columns (phi, theta, q/p) go
//    through the RK stages themselves instead of 3x3 blocks formed and then
//    multiplied (stepGrid), and the grid's FP32 values are widened on the
//    integer pipe.
//
// Measured on a GB300 (2070 MHz) against the filter with a covariance
// transport per plane and a smoother pass over stored states: 1M tracks of 10
// planes in a uniform field 39.2 -> 14.8 ms, 50021 tracks of 30 planes in a
// field map 13.0 -> 5.4 ms, 1M of those mixed 91.7 -> 37.6 ms, 100003 tracks
// through material 7.1 -> 2.4 ms.  19.5 cycles per FP64 instruction and SM:
// the pipe is full.
#pragma once

#include "kf_device.cuh"
#include "kf_recip.cuh"

namespace kfd {

// kUniform64: FP64, uniform field along +-z; kUniformAny: in any other
// direction (planes rotated into the field's frame); kGrid64: FP64, field
// map; kMixed: mixed precision, field map; kMixedUniform: mixed precision,
// uniform field (without the lookups' code: the mixed kernels wait for
// instruction fetches)
enum FitForm { kUniform64 = 0, kGrid64 = 1, kMixed = 2, kUniformAny = 3, kMixedUniform = 4 };
__host__ __device__ constexpr bool isMixed(int form) { return form == kMixed || form == kMixedUniform; }
__host__ __device__ constexpr bool isUniform(int form) { return form == kUniform64 || form == kUniformAny; }

// ---- shared-memory layout ---------------------------------------------------
// One column per thread ([element][thread]).  Without process noise: F rows
// 0-3 (20), C0 (15, row-major upper triangle of 5x5), its time column (6),
// D (6), the direction's trigonometry at the last surface (4).  With: C (15),
// X (6x5), the first state's covariance (21), D (6), trigonometry (4).
template <bool MAT> __host__ __device__ constexpr int coldSlots() { return MAT ? 76 : 51; }
template <bool MAT> __host__ __device__ constexpr size_t fitSmemBytes(int threads, int nSurf) {
  return (size_t)threads * coldSlots<MAT>() * sizeof(double) + (size_t)nSurf * sizeof(PlaneD);
}
__host__ __device__ constexpr int u5(int i, int j) { // upper triangle of 5x5
  return i <= j ? i * 5 - (i * (i - 1)) / 2 + (j - i) : j * 5 - (j * (j - 1)) / 2 + (i - j);
}

// a state's record in the workspace: x_p - F D (6), F rows 0-3 (20), F's time
// row (5), and for the first state the direction's trigonometry (4) and, once
// its x is read, in place of phi the time's q/p factor that the leg to the line
// owes to an earlier momentum
enum { kRecX = 0, kRecRest = 2, kRecF = 6, kRecT = 26, kRecTrig = 31 };
static_assert(kRecTrig + 4 <= kStateStride, "state record");

template <int FORM, int GROUP = 1> struct LegState;
// eight lanes on one track (kf_fit_coop.cuh)
struct CoopHook : NoHook {
  static constexpr int kGroup = 8;
};
// uniform field, z along the field: with A v = v x z the leg's transport is
// dir: I + b A + (1 - g) A^2, pos: s I + q1 A + (s - r) A^2; c, a: q/p column
template <> struct LegState<kUniform64> {
  double g, b, r, q1, s, c[2], a[2];
  double y, dx, dy; // last step: h q/p B and the direction it started from (k4)
};
template <> struct LegState<kUniformAny> : LegState<kUniform64> {};
// field map: columns phi, theta, q/p of position and direction
template <> struct LegState<kGrid64> {
  double p[3][3], v[3][3], s, k4[3];
};
// mixed: FP32 transport blocks as offsets from the straight line
// (applyTransportOffsets)
template <> struct LegState<kMixed> {};
template <> struct LegState<kMixedUniform> {};
// each lane its 2-vector of those that the step turns alike, (v, p) = the
// track's (dir, pos) in lanes 0 and 1, ((g, -b), (r, -q1)) in 2 and 3, (c, a)
// in the others
template <> struct LegState<kUniform64, 8> {
  double v[2], p[2], s;
  double y, dx, dy;
};
template <> struct LegState<kMixed, 8> {};
template <> struct LegState<kMixedUniform, 8> {};
// each lane of a group carries its own column (2: phi, 3: theta, 4: q/p, 5: the
// direction that the leg started with, see legRebase)
template <> struct LegState<kGrid64, 8> {
  double p[3], v[3], s, k4[3];
};
struct NoBlocks {};
struct MixedBlocks {
  float JA[3][3], Ja[3], Jb, JB[3][3], Jc[3], k4[3];
  float qopf, d37f; // of the leg
  double sTr;
};

template <int FORM, bool MAT_, class H_ = NoHook>
struct FitLane : std::conditional<isMixed(FORM), MixedBlocks, NoBlocks>::type {
  static constexpr int kForm = FORM;
  static constexpr bool kMat = MAT_;
  static constexpr bool kTape = H_::kTape;
  static constexpr bool kCoop = H_::kGroup > 1;
  double pos[3], dir[3]; // FP64 uniform field: in the field's frame
  double q, qop, t, dtds, d37;
  double idn;            // 1 / (T . dir) of the plane last looked at
  double ss[4];
  int ssDir, navDir;
  LegState<FORM, H_::kGroup> g;
  bool stepped;
  int next, current, nSeq, navCache, navCacheSt;
  long long navCacheLim;
  uint64_t mask;
  int nHits, measStates, firstPlane, lastPlane; // lastPlane: of the jacToGlobal in use
  bool targetReached, navBreak, smoothed, finished, result, tn, timeCorr, badJ;
  int parked; // 0: runs, else its pending event's EventStage
  int pc, steps, status, rkSteps, rkTrials;
  double chi2;
  int64_t idx, wsIdx;
  H_ hook;

  __device__ __forceinline__ double &cold(int e) const {
    return reinterpret_cast<double *>(kfColdSmem)[e * blockDim.x + threadIdx.x];
  }
  // the column of lane l of this thread's group
  __device__ __forceinline__ double &coldOf(int e, int l) const {
    return reinterpret_cast<double *>(kfColdSmem)[e * blockDim.x + (threadIdx.x & ~(H_::kGroup - 1)) + l];
  }
  // no process noise; in a group, lane c holds column c of F, row c of C0's
  // upper triangle and entry c of D
  __device__ __forceinline__ double &F(int r, int c) const {
    return kCoop ? coldOf(r, c) : cold(5 * r + c);
  }
  __device__ __forceinline__ double &C0(int e) const {
    if (!kCoop) return cold(20 + e);
    const int i = e < 5 ? 0 : e < 9 ? 1 : e < 12 ? 2 : e < 14 ? 3 : 4;
    return coldOf(4 + e - u5(i, i), i);
  }
  __device__ __forceinline__ double &Ct(int i) const { return cold(35 + i); }
  // process noise
  __device__ __forceinline__ double &C(int e) const { return cold(e); }
  __device__ __forceinline__ double &X(int r, int c) const { return cold(15 + 5 * r + c); }
  __device__ __forceinline__ double &P1(int e) const { return cold(45 + e); }
  // both: D (sum of K0 r) and the trigonometry (cos phi, sin phi, cos theta, sin theta)
  __device__ __forceinline__ double &D(int i) const {
    return kCoop && i < 5 ? coldOf(9, i) : cold((MAT_ ? 66 : 41) + i);
  }
  __device__ __forceinline__ double &trigS(int i) const { return cold((MAT_ ? 72 : 47) + i); }
};

struct Trig {
  double cP, sP, cT, sT;
};
template <class LT> __device__ __forceinline__ void trigSave(const LT &L, const Trig &t) {
  L.trigS(0) = t.cP;
  L.trigS(1) = t.sP;
  L.trigS(2) = t.cT;
  L.trigS(3) = t.sT;
}
template <class LT> __device__ __forceinline__ Trig trigLoad(const LT &L) {
  return {L.trigS(0), L.trigS(1), L.trigS(2), L.trigS(3)};
}
// of a direction in the global frame; invS = 1 / sin theta
__device__ __forceinline__ Trig trigOf(const double d[3], double &invS) {
  const double s2 = d[0] * d[0] + d[1] * d[1];
  invS = rsqrtFast(s2);
  return {d[0] * invS, d[1] * invS, d[2], s2 * invS};
}

// global <-> field frame (the identity unless the field is off the z axis)
template <class LT>
__device__ __forceinline__ void toGlobal(const Params &P, const double v[3], double o[3]) {
  if (LT::kForm == kUniformAny) {
#pragma unroll
    for (int i = 0; i < 3; ++i) o[i] = P.rot[i] * v[0] + P.rot[3 + i] * v[1] + P.rot[6 + i] * v[2];
  } else {
#pragma unroll
    for (int i = 0; i < 3; ++i) o[i] = v[i];
  }
}
template <class LT>
__device__ __forceinline__ void toFrame(const Params &P, const double v[3], double o[3]) {
  if (LT::kForm == kUniformAny) {
#pragma unroll
    for (int i = 0; i < 3; ++i)
      o[i] = P.rot[3 * i] * v[0] + P.rot[3 * i + 1] * v[1] + P.rot[3 * i + 2] * v[2];
  } else {
#pragma unroll
    for (int i = 0; i < 3; ++i) o[i] = v[i];
  }
}

template <class LT> __device__ __forceinline__ double *recPtr(const Params &P, const LT &L, int s, int e) {
  return P.ws + ((size_t)s * kStateStride + e) * (size_t)P.wsStride + L.wsIdx;
}

// q/p, and where the time is carried dt/ds and the time's q/p factor
// (legConstantsIp), from 1/p
template <class LT>
__device__ __forceinline__ void setMomentum(LT &L, const Params &P, double ip, bool time) {
  L.qop = L.q * ip;
  if constexpr (isMixed(LT::kForm)) L.qopf = narrow(L.qop);
  if (time) {
    const double x = P.mass * ip, a = fma(x, x, 1.);
    const double y = rsqrtFast(a);
    L.dtds = a * y;
    L.d37 = P.mass * P.mass * L.qop * y;
    if constexpr (isMixed(LT::kForm)) L.d37f = (float)L.d37;
  }
}

// the jacToGlobal in use from here on: bound parameters on plane `plane` (or
// the start's line), angles at the direction `t` (re-initialised Jacobians,
// CovarianceEngine.hpp:169-201)
template <int FORM, bool MAT, class H>
__device__ __forceinline__ void legReset(FitLane<FORM, MAT, H> &L, const Trig &t) {
  L.stepped = false;
  if constexpr (FORM == kUniform64 && H::kGroup > 1) {
    L.g.v[0] = (threadIdx.x & 6) == 2 ? 1. : 0.;
    L.g.v[1] = L.g.p[0] = L.g.p[1] = L.g.s = 0.;
    L.g.y = L.g.dx = L.g.dy = 0.;
  } else if constexpr (isUniform(FORM)) {
    L.g.g = 1.;
    L.g.b = L.g.r = L.g.q1 = L.g.s = 0.;
    L.g.c[0] = L.g.c[1] = L.g.a[0] = L.g.a[1] = 0.;
    L.g.y = L.g.dx = L.g.dy = 0.;
  } else if constexpr (FORM == kGrid64 && H::kGroup > 1) {
    const int c = threadIdx.x & 7;
    const bool phi = c == 2, th = c == 3, rad = c == 5;
    L.g.p[0] = L.g.p[1] = L.g.p[2] = 0.;
    L.g.v[0] = phi ? -t.sT * t.sP : (th ? t.cT * t.cP : (rad ? t.sT * t.cP : 0.));
    L.g.v[1] = phi ? t.sT * t.cP : (th ? t.cT * t.sP : (rad ? t.sT * t.sP : 0.));
    L.g.v[2] = th ? -t.sT : (rad ? t.cT : 0.);
    L.g.s = 0.;
    L.g.k4[0] = L.g.k4[1] = L.g.k4[2] = 0.;
  } else if constexpr (FORM == kGrid64) {
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) L.g.p[i][j] = L.g.v[i][j] = 0.;
    L.g.v[0][0] = -t.sT * t.sP;
    L.g.v[0][1] = t.sT * t.cP;
    L.g.v[1][0] = t.cT * t.cP;
    L.g.v[1][1] = t.cT * t.sP;
    L.g.v[1][2] = -t.sT;
    L.g.s = 0.;
    L.g.k4[0] = L.g.k4[1] = L.g.k4[2] = 0.;
  } else {
#pragma unroll
    for (int i = 0; i < 3; ++i) {
#pragma unroll
      for (int j = 0; j < 3; ++j) L.JA[i][j] = L.JB[i][j] = 0.f;
      L.Ja[i] = L.Jc[i] = L.k4[i] = 0.f;
    }
    L.Jb = 0.f;
    L.sTr = 0.;
  }
}

// Field map, faithful_jacobian = 0: where the track runs out of planes, the
// smoothed state's jacToGlobal takes the place of the last hit's under a leg
// that has begun (finalizeSmooth).  The leg's transport of any direction is
// that of the last hit's phi and theta columns and of the leg's first
// direction itself; the last is carried only in such a fit, in the record of
// the state that the leg may still reach (a group's lane 5 has it for nothing).
template <class LT> __device__ __forceinline__ bool keepsDirection(const LT &L, const Params &P) {
  return !P.faithful && P.smoothing && !L.smoothed && L.measStates > 0 && L.measStates < P.nSurf;
}
// the columns phi and theta at `t` in place of those at `t0`
template <bool MAT, class H>
__device__ __forceinline__ void legRebase(FitLane<kGrid64, MAT, H> &L, const Params &P, const Trig &t0,
                                          const Trig &t) {
  const double is2 = 1. / (t0.sT * t0.sT);
  const double d0[3] = {t0.sT * t0.cP, t0.sT * t0.sP, t0.cT};
  const double ph0[3] = {-t0.sT * t0.sP, t0.sT * t0.cP, 0.}, th0[3] = {t0.cT * t0.cP, t0.cT * t0.sP, -t0.sT};
  double np[2][3], nv[2][3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    double p[3], v[3]; // of ph0, th0, d0
    if constexpr (H::kGroup > 1) {
      const unsigned group = 0xffu << (threadIdx.x & 24);
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        p[k] = __shfl_sync(group, L.g.p[i], k < 2 ? 2 + k : 5, 8);
        v[k] = __shfl_sync(group, L.g.v[i], k < 2 ? 2 + k : 5, 8);
      }
    } else {
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        p[k] = L.g.p[k][i];
        v[k] = L.g.v[k][i];
      }
      p[2] = *recPtr(P, L, L.measStates, i);
      v[2] = *recPtr(P, L, L.measStates, 3 + i);
    }
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const double e[3] = {c ? t.cT * t.cP : -t.sT * t.sP, c ? t.cT * t.sP : t.sT * t.cP, c ? -t.sT : 0.};
      double a[3] = {0., 0., 0.};
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        a[0] += e[k] * ph0[k] * is2;
        a[1] += e[k] * th0[k];
        a[2] += e[k] * d0[k];
      }
      np[c][i] = a[0] * p[0] + a[1] * p[1] + a[2] * p[2];
      nv[c][i] = a[0] * v[0] + a[1] * v[1] + a[2] * v[2];
    }
  }
#pragma unroll
  for (int c = 0; c < 2; ++c)
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      if constexpr (H::kGroup > 1) {
        if ((threadIdx.x & 7) == 2 + c) {
          L.g.p[i] = np[c][i];
          L.g.v[i] = nv[c][i];
        }
      } else {
        L.g.p[c][i] = np[c][i];
        L.g.v[c][i] = nv[c][i];
      }
    }
}

// ---------------------------------------------------------------------------
// RK steps
// ---------------------------------------------------------------------------
// step-size scale of a rejected trial (EigenStepper.ipp:281-290)
__device__ __forceinline__ double rejectScale(double tol, double err) {
  const double r = tol / fabs(2. * err);
  return smin(smax(0.25, sqrt(sqrt(r))), 4.);
}
// set the accuracy constraint and the next trial's step; false: give up
template <class LT>
__device__ __forceinline__ bool rejectTrial(LT &L, const Params &P, double err, double &h,
                                            long &nTrials) {
  const double hn = h * rejectScale(P.tol, err);
  L.ss[kAccuracy] = hn;
  L.ssDir = hn > 0. ? 1 : -1;
  h = ssValue(L);
  if (h * h < P.cutoff * P.cutoff || nTrials > P.maxTrials) return false;
  nTrials++;
  return true;
}

// 1/|d| for |d|^2 = 1 + e: one Newton step of 1/sqrt from 1 (error 3/8 e^2)
// where e is below 1e-8, as in all but steps that turn far
__device__ __forceinline__ double unitFactor(const double d[3]) {
  const double n2 = fma(d[0], d[0], fma(d[1], d[1], d[2] * d[2]));
  const double f = fma(n2, -0.5, 1.5);
  // 1 +- 1e-8 by the bits of 3/2 - n2/2
  const long long k = __double_as_longlong(f) - 0x3ff0000000000000LL;
  if (k > 22517998LL || k < -45035996LL) return rsqrt(n2);
  return f;
}

// Uniform field along z.  With A v = v x z (A^3 = -A), y = h q/p B and
// x = y^2 the RK4 step of EigenStepper.ipp:243-269 and its transport matrix
// (:50-124) are
//   dir' = (I + al A + be A^2) dir, pos' = pos + (h I + mu A + nu A^2) dir,
//   al = y (1 - x/6), be = x (1/2 - x/24), mu = h y (1/2 - x/24), nu = h x/6,
// the same two matrices D_B, D_A for the transport Jacobian, and the q/p
// column's sources are their q/p derivatives (kfa::polyAcceptFwd has the
// general field).  The error estimate
// h^2 |k1 - k2 - k3 + k4|_1 = |h y| x/4 |A dir + y A^2 dir|_1
// is at most |h y| x times P.errBound's factor for |y| <= 0.1, which accepts
// with one product; only beyond that bound it is evaluated.
// |dir'|^2 - |dir|^2 = |dir_perp|^2 x^3 (x/576 - 1/72): below half an ulp, so
// that there is nothing to normalise, where |x| < 1e-5.
template <int FORM, bool MAT, class H>
__device__ __forceinline__ void stepUniform(FitLane<FORM, MAT, H> &L, const Params &P) {
  long nTrials = 0;
  double h = ssValue(L);
  const double k = L.qop * P.Bz;
  const double dx = L.dir[0], dy = L.dir[1];
  double y, x, hy;
  L.hook.stepBegin(L);
  for (;;) {
    L.rkTrials++;
    L.hook.trial(L, h);
    y = h * k;
    x = y * y;
    hy = h * y;
    // (a step whose square overflows, towards no plane, is rejected in any field)
    const bool far = akey(h) > 0x5fefffffffffffffLL;
    if (akey(hy * x) <= P.errBound && akey(y) <= 0x3fb999999999999aLL && !far) break;
    const double v0 = fma(-y, dx, dy), v1 = fma(-y, dy, -dx);
    double n1;
    if (FORM == kUniformAny)
      n1 = fabs(P.rot[0] * v0 + P.rot[3] * v1) + fabs(P.rot[1] * v0 + P.rot[4] * v1) +
           fabs(P.rot[2] * v0 + P.rot[5] * v1);
    else
      n1 = fabs(v0) + fabs(v1);
    const double e0 = far ? DBL_MAX : 0.25 * fabs(hy) * x * n1;
    const double err = e0 < 1e-20 ? 1e-20 : e0;
    if (err <= P.tol) break;
    if (!rejectTrial(L, P, err, h, nTrials)) {
      L.hook.stepEnd(L, false);
      return;
    }
  }
  L.hook.stepEnd(L, true);
  auto &g = L.g;
  const double m = fma(x, -1. / 24., 0.5), n = fma(x, -1. / 6., 1.);
  const double al = y * n, be1 = fma(-x, m, 1.);
  const double mu = hy * m, nu = h * x * (1. / 6.), hn = h - nu;
  // q/p derivatives (y's is h B)
  const double hb = h * P.Bz, hhb = h * hb;
  const double al1 = hb * fma(x, -0.5, 1.), be2 = hb * al;
  const double mu1 = hhb * fma(x, -0.125, 0.5), nu1 = hhb * y * (1. / 3.);
  if constexpr (H::kGroup > 1) {
    // this lane's 2-vector (LegState); the q/p column has a source besides (a
    // product plus -0 rounds as the product)
    const unsigned group = 0xffu << (threadIdx.x & 24);
    const int l = threadIdx.x & 7;
    const bool track = l < 2, qp = l >= 4;
    const double v0 = track ? dx : g.v[0], v1 = track ? dy : g.v[1];
    const double p0 = track ? L.pos[0] : g.p[0], p1 = track ? L.pos[1] : g.p[1];
    const double sc0 = fma(al1, dy, -be2 * dx), sc1 = fma(-al1, dx, -be2 * dy);
    const double sa0 = fma(mu1, dy, fma(-nu1, dx, p0)), sa1 = fma(-mu1, dx, fma(-nu1, dy, p1));
    g.p[0] = fma(hn, v0, fma(mu, v1, qp ? sa0 : p0));
    g.p[1] = fma(hn, v1, fma(-mu, v0, qp ? sa1 : p1));
    g.v[0] = fma(be1, v0, fma(al, v1, qp ? sc0 : -0.));
    g.v[1] = fma(be1, v1, fma(-al, v0, qp ? sc1 : -0.));
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      L.dir[i] = __shfl_sync(group, g.v[i], 0, 8);
      L.pos[i] = __shfl_sync(group, g.p[i], 0, 8);
    }
    L.pos[2] = fma(h, L.dir[2], L.pos[2]);
    g.s += h;
    g.y = y;
    g.dx = dx;
    g.dy = dy;
  } else {
    // q/p column
    const double a0 = fma(hn, g.c[0], fma(mu, g.c[1], fma(mu1, dy, fma(-nu1, dx, g.a[0]))));
    const double a1 = fma(hn, g.c[1], fma(-mu, g.c[0], fma(-mu1, dx, fma(-nu1, dy, g.a[1]))));
    const double c0 = fma(be1, g.c[0], fma(al, g.c[1], fma(al1, dy, -be2 * dx)));
    const double c1 = fma(be1, g.c[1], fma(-al, g.c[0], fma(-al1, dx, -be2 * dy)));
    g.a[0] = a0;
    g.a[1] = a1;
    g.c[0] = c0;
    g.c[1] = c1;
    // transport of the direction columns
    g.r = fma(hn, g.g, fma(-mu, g.b, g.r));
    g.q1 = fma(hn, g.b, fma(mu, g.g, g.q1));
    g.s += h;
    const double gg = fma(be1, g.g, -al * g.b);
    g.b = fma(be1, g.b, al * g.g);
    g.g = gg;
    g.y = y;
    g.dx = dx;
    g.dy = dy;
    // the track
    L.pos[0] = fma(hn, dx, fma(mu, dy, L.pos[0]));
    L.pos[1] = fma(hn, dy, fma(-mu, dx, L.pos[1]));
    L.pos[2] = fma(h, L.dir[2], L.pos[2]);
    L.dir[0] = fma(be1, dx, al * dy);
    L.dir[1] = fma(be1, dy, -al * dx);
  }
  if (!(akey(x) < 0x3ee4f8b588e368f1LL)) { // |x| >= 1e-5
    const double f = unitFactor(L.dir);
    L.dir[0] *= f;
    L.dir[1] *= f;
    L.dir[2] *= f;
  }
  L.stepped = true;
  L.rkSteps++;
}
template <bool MAT, class H> __device__ __forceinline__ void rkStep(FitLane<kUniform64, MAT, H> &L, const Params &P) {
  stepUniform(L, P);
}
template <bool MAT, class H> __device__ __forceinline__ void rkStep(FitLane<kUniformAny, MAT, H> &L, const Params &P) {
  stepUniform(L, P);
}

// field at p times s (s = scale q/p), FP64 trilinear: the lookup of getField
// with the cell index from one rounding addition and the grid's values
// widened on the integer pipe (24 conversions a lookup otherwise, each as
// long on the FP64 pipe as an FMA)
static __device__ __noinline__ double3 fieldRZ64(const FieldD &F, double x, double y, double z) {
  const double p[3] = {x, y, z};
  double B[3];
  getFieldRZ(F, p, B);
  return make_double3(B[0], B[1], B[2]);
}
__device__ __forceinline__ void fieldScaled(const FieldD &F, const double p[3], double qop, double B[3]) {
  if (F.kind != KF_FIELD_GRID3D) {
    const double3 b = fieldRZ64(F, p[0], p[1], p[2]);
    B[0] = b.x * qop;
    B[1] = b.y * qop;
    B[2] = b.z * qop;
    return;
  }
  int idx[3];
  double f[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    // floor by adding 2^52 + 2^51, whose unit in the last place is 1, with
    // rounding down
    const double gr = fma(p[a], F.invw[a], F.off[a]);
    const double t = __dadd_rd(gr, 6755399441055744.);
    // clamped to the grid (outside it the edge cell extends): the low word is
    // the index where the high word says so, and beyond 2^31 only the sign counts
    int i = __double2loint(t);
    const int hi = __double2hiint(t);
    if (hi != 0x43380000 || i < 0) i = hi == 0x4337ffff || __double2hiint(gr) < 0 ? 0 : F.n[a] - 2;
    i = min(i, F.n[a] - 2);
    idx[a] = i;
    f[a] = gr - (__hiloint2double(0x43380000, i) - 6755399441055744.);
  }
  const size_t nx = F.n[0], nxy = (size_t)F.n[0] * F.n[1];
  const float4 *g = F.grid + ((size_t)idx[2] * nxy + (size_t)idx[1] * nx + idx[0]);
  const float4 v000 = __ldg(g), v100 = __ldg(g + 1), v010 = __ldg(g + nx), v110 = __ldg(g + nx + 1);
  const float4 v001 = __ldg(g + nxy), v101 = __ldg(g + nxy + 1), v011 = __ldg(g + nxy + nx),
               v111 = __ldg(g + nxy + nx + 1);
  const double s = F.scale * qop;
  // The differences of neighbours along x are taken in FP32, where they are
  // exact for values within a factor of 2 of each other (Sterbenz), as almost
  // all are; TwoSum's error term tells, and any inexact one sends the lookup
  // through FP64 differences: 12 of 42 FP64 instructions a lookup less.  A
  // value or difference that is not finite makes the term NaN.
  unsigned off = 0;
  auto dif = [&](float a, float b) {
    const float e = __fsub_rn(b, a), t = __fsub_rn(e, b);
    off |= __float_as_uint(__fsub_rn(__fsub_rn(b, __fsub_rn(e, t)), __fadd_rn(a, t)));
    return widenFinite(e);
  };
  auto mix = [](double a, double b, double w) { return fma(w, b - a, a); };
  auto tri = [&](float a000, float a100, float a010, float a110, float a001, float a101,
                 float a011, float a111) {
    const double c00 = fma(f[0], dif(a000, a100), widenFinite(a000));
    const double c10 = fma(f[0], dif(a010, a110), widenFinite(a010));
    const double c01 = fma(f[0], dif(a001, a101), widenFinite(a001));
    const double c11 = fma(f[0], dif(a011, a111), widenFinite(a011));
    return mix(mix(c00, c10, f[1]), mix(c01, c11, f[1]), f[2]) * s;
  };
  B[0] = tri(v000.x, v100.x, v010.x, v110.x, v001.x, v101.x, v011.x, v111.x);
  B[1] = tri(v000.y, v100.y, v010.y, v110.y, v001.y, v101.y, v011.y, v111.y);
  B[2] = tri(v000.z, v100.z, v010.z, v110.z, v001.z, v101.z, v011.z, v111.z);
  if (off & 0x7fffffffu) { // (a zero's sign apart)
    auto tri64 = [&](float a000, float a100, float a010, float a110, float a001, float a101,
                     float a011, float a111) {
      const double c00 = mix(widen(a000), widen(a100), f[0]), c10 = mix(widen(a010), widen(a110), f[0]);
      const double c01 = mix(widen(a001), widen(a101), f[0]), c11 = mix(widen(a011), widen(a111), f[0]);
      return mix(mix(c00, c10, f[1]), mix(c01, c11, f[1]), f[2]) * s;
    };
    B[0] = tri64(v000.x, v100.x, v010.x, v110.x, v001.x, v101.x, v011.x, v111.x);
    B[1] = tri64(v000.y, v100.y, v010.y, v110.y, v001.y, v101.y, v011.y, v111.y);
    B[2] = tri64(v000.z, v100.z, v010.z, v110.z, v001.z, v101.z, v011.z, v111.z);
  }
}

// Field map, FP64 stage by stage (EigenStepper.ipp:243-332), with q/p folded
// into the field values.  The three columns (p, v) of the transport Jacobian
// that a leg needs go through the linearised stages
//   dk1 = v x b1, dk2 = (v + h/2 dk1) x b2, dk3 = (v + h/2 dk2) x b2,
//   dk4 = (v + h dk3) x b3, p += h v + h^2/6 (dk1 + dk2 + dk3),
//   v += h/6 (dk1 + 2 (dk2 + dk3) + dk4)
// which is D J on those columns (D: transportMatrix, EigenStepper.ipp:50-124)
// without forming D; the q/p column adds each stage's own k_i / (q/p).
template <bool MAT, class H> __device__ __forceinline__ void rkStep(FitLane<kGrid64, MAT, H> &L, const Params &P) {
  long nTrials = 0;
  double h = ssValue(L);
  double b1[3], b2[3], b3[3], k1[3], k2[3], k3[3], k4[3], t[3];
  fieldScaled(P.field, L.pos, L.qop, b1);
  cross3(L.dir, b1, k1);
  for (;;) {
    L.rkTrials++;
    const double hh = 0.5 * h, h22 = hh * h, h8 = 0.25 * h22;
#pragma unroll
    for (int i = 0; i < 3; ++i) t[i] = fma(h8, k1[i], fma(hh, L.dir[i], L.pos[i]));
    fieldScaled(P.field, t, L.qop, b2);
#pragma unroll
    for (int i = 0; i < 3; ++i) t[i] = fma(hh, k1[i], L.dir[i]);
    cross3(t, b2, k2);
#pragma unroll
    for (int i = 0; i < 3; ++i) t[i] = fma(hh, k2[i], L.dir[i]);
    cross3(t, b2, k3);
#pragma unroll
    for (int i = 0; i < 3; ++i) t[i] = fma(h22, k3[i], fma(h, L.dir[i], L.pos[i]));
    fieldScaled(P.field, t, L.qop, b3);
#pragma unroll
    for (int i = 0; i < 3; ++i) t[i] = fma(h, k3[i], L.dir[i]);
    cross3(t, b3, k4);
    // in FP32 first: the estimate with a bound of its rounding (four values
    // of |k| at 2^-24 each and the sums': below 1e-6 |k|) decides unless it
    // comes near the tolerance
    {
      const float hf = narrow(h);
      float e = 0.f;
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const float a = narrow(k1[i]), b = narrow(k2[i]), c = narrow(k3[i]),
                    d = narrow(k4[i]);
        e += fabsf((a - b) + (d - c)) + 1e-6f * (fabsf(a) + fabsf(b) + fabsf(c) + fabsf(d));
      }
      if (hf * hf * e <= P.tolAcceptF) break;
    }
    const double d0 = k1[0] - k2[0] - k3[0] + k4[0], d1 = k1[1] - k2[1] - k3[1] + k4[1],
                 d2 = k1[2] - k2[2] - k3[2] + k4[2];
    const double e = h * h * (fabs(d0) + fabs(d1) + fabs(d2));
    const double err = (e < 1e-20) ? 1e-20 : e;
    if (err <= P.tol) break;
    if (!rejectTrial(L, P, err, h, nTrials)) return;
  }
  const double hh = 0.5 * h, h6 = h * (1. / 6.), hh6 = h * h6;
  const double iq = rcpFast(L.qop);
  auto &g = L.g;
  auto column = [&](double (&p)[3], double (&v)[3], bool own, double q1) {
    double e1[3], e2[3], e3[3], e4[3], w[3];
    auto src = [&](double e[3], const double k[3]) {
      if (own) {
#pragma unroll
        for (int i = 0; i < 3; ++i) e[i] = fma(k[i], q1, e[i]);
      }
    };
    cross3(v, b1, e1);
    src(e1, k1);
#pragma unroll
    for (int i = 0; i < 3; ++i) w[i] = fma(hh, e1[i], v[i]);
    cross3(w, b2, e2);
    src(e2, k2);
#pragma unroll
    for (int i = 0; i < 3; ++i) w[i] = fma(hh, e2[i], v[i]);
    cross3(w, b2, e3);
    src(e3, k3);
#pragma unroll
    for (int i = 0; i < 3; ++i) w[i] = fma(h, e3[i], v[i]);
    cross3(w, b3, e4);
    src(e4, k4);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const double s23 = e2[i] + e3[i];
      p[i] = fma(hh6, e1[i] + s23, fma(h, v[i], p[i]));
      v[i] = fma(h6, fma(2., s23, e1[i] + e4[i]), v[i]);
    }
  };
  if constexpr (H::kGroup > 1) {
    column(g.p, g.v, true, (threadIdx.x & 7) == 4 ? iq : 0.);
  } else {
    column(g.p[0], g.v[0], false, 0.);
    column(g.p[1], g.v[1], false, 0.);
    column(g.p[2], g.v[2], true, iq);
    if (keepsDirection(L, P)) {
      double p[3], v[3];
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        p[i] = L.stepped ? *recPtr(P, L, L.measStates, i) : 0.;
        v[i] = L.stepped ? *recPtr(P, L, L.measStates, 3 + i) : L.dir[i];
      }
      column(p, v, false, 0.);
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        *recPtr(P, L, L.measStates, i) = p[i];
        *recPtr(P, L, L.measStates, 3 + i) = v[i];
      }
    }
  }
  g.s += h;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const double s23 = k2[i] + k3[i];
    L.pos[i] = fma(hh6, k1[i] + s23, fma(h, L.dir[i], L.pos[i]));
    L.dir[i] = fma(h6, fma(2., s23, k1[i] + k4[i]), L.dir[i]);
    g.k4[i] = k4[i];
  }
  const double f = unitFactor(L.dir);
  L.dir[0] *= f;
  L.dir[1] *= f;
  L.dir[2] *= f;
  L.stepped = true;
  L.rkSteps++;
}

// error estimate of a trial step in FP64 (EigenStepper.ipp:243-269); one
// rejected lane makes its whole warp wait for it
__device__ __forceinline__ double trialErrorUniform(const FieldD &F, const double dir[3], double qop,
                                                    double h) {
  kfa::PolyStep w;
  kfa::polyPrep(dir, F.B, w);
  // no field: the estimate's floor while h^2 is finite, whatever h q/p is
  if (w.beta == 0.) return akey(h) > 0x5fefffffffffffffLL ? DBL_MAX : 1e-20;
  kfa::polyCoef(qop, h, w);
  return w.err;
}
static __device__ __noinline__ double trialError(const FieldD &F, double p0, double p1, double p2,
                                                 double d0, double d1, double d2, double qop, double h) {
  const double pos[3] = {p0, p1, p2}, dir[3] = {d0, d1, d2};
  double b[3], k1[3], k2[3], k3[3], k4[3], t[3];
  const double hh = 0.5 * h, h2 = h * h;
  fieldScaled(F, pos, qop, b);
  cross3(dir, b, k1);
#pragma unroll
  for (int i = 0; i < 3; ++i) t[i] = fma(0.125 * h2, k1[i], fma(hh, dir[i], pos[i]));
  fieldScaled(F, t, qop, b);
#pragma unroll
  for (int i = 0; i < 3; ++i) t[i] = fma(hh, k1[i], dir[i]);
  cross3(t, b, k2);
#pragma unroll
  for (int i = 0; i < 3; ++i) t[i] = fma(hh, k2[i], dir[i]);
  cross3(t, b, k3);
#pragma unroll
  for (int i = 0; i < 3; ++i) t[i] = fma(0.5 * h2, k3[i], fma(h, dir[i], pos[i]));
  fieldScaled(F, t, qop, b);
#pragma unroll
  for (int i = 0; i < 3; ++i) t[i] = fma(h, k3[i], dir[i]);
  cross3(t, b, k4);
  double e = 0.;
#pragma unroll
  for (int i = 0; i < 3; ++i) e += fabs(k1[i] - k2[i] - k3[i] + k4[i]);
  e *= h2;
  return (e < 1e-20) ? 1e-20 : e;
}

// Mixed form: FP32 stage offsets from an FP64 k1, FP32 transport
// (rkTrialDelta, applyTransportOffsets), FP64 position and direction.  The
// FP32 estimate accepts below 99 % of the tolerance; otherwise the FP64 trial
// decides, and a rejection sets the next trial's size from its error
// estimate: the FP32 estimate is a sum of offsets that cancel to ~1 % of
// their size, good to ~1e-5 relative, and rescaled from it the step sizes
// (the RK partition of the path) would drift from the FP64 fit's by ~3e-6,
// so that a later decision near the tolerance could go the other way (1e-4 of
// the perigee's resolution on a few tracks in 1e6).
template <int FORM, bool MAT, class H>
__device__ __forceinline__ typename std::enable_if<isMixed(FORM)>::type
rkStep(FitLane<FORM, MAT, H> &L, const Params &P) {
  constexpr int kMap = FORM == kMixed ? 1 : 0;
  long nTrials = 0;
  double h = ssValue(L);
  const float qopf = L.qopf;
  float posf[3], res[3], hf;
#pragma unroll
  for (int i = 0; i < 3; ++i) split(L.pos[i], posf[i], res[i]);
  const float dirf[3] = {narrow(L.dir[0]), narrow(L.dir[1]), narrow(L.dir[2])};
  StagesDelta S;
  rkFirstDelta<kMap>(P.field, posf, res, L.dir, L.qop, S);
  for (;;) {
    L.rkTrials++;
    hf = narrow(h);
    const float errf = rkTrialDelta<kMap>(P.field, posf, res, dirf, qopf, hf, S);
    if (errf <= P.tolLoF) break;
    const double err = FORM == kMixed
                           ? trialError(P.field, L.pos[0], L.pos[1], L.pos[2], L.dir[0], L.dir[1],
                                        L.dir[2], L.qop, h)
                           : trialErrorUniform(P.field, L.dir, L.qop, h);
    if (err <= P.tol) break;
    if (!rejectTrial(L, P, err, h, nTrials)) return;
  }
  transportUpdate<float>(L, dirf, qopf, hf, L.d37f, S.s);
  L.sTr += h;
  // motion: FP64 state, FP64 k1, FP32 sums of the offsets
  //   pos += h d + h^2/6 (3 k1 + d2 + d3),  dir += h/6 (6 k1 + 2 (d2 + d3) + d4)
  // (finite: any other offset makes either error estimate NaN or infinite)
  const double h6 = h * (1. / 6.), hh6 = h * h6;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const float s23 = S.d2[i] + S.d3[i];
    const float s234 = 2.f * s23 + S.d4[i];
    L.pos[i] = fma(hh6, fma(3., S.k1[i], widenFinite(s23)), fma(h, L.dir[i], L.pos[i]));
    L.dir[i] = fma(h6, fma(6., S.k1[i], widenFinite(s234)), L.dir[i]);
  }
  const double f = unitFactor(L.dir);
  L.dir[0] *= f;
  L.dir[1] *= f;
  L.dir[2] *= f;
#pragma unroll
  for (int i = 0; i < 3; ++i) L.k4[i] = S.s.k4[i];
  L.stepped = true;
  L.rkSteps++;
}

// ---------------------------------------------------------------------------
// Navigation: the plane distance with one short division; magnitudes are
// compared as integers (|path| < tol for the reference's path^2 < tol^2)
// ---------------------------------------------------------------------------
template <int FORM, bool MAT, class H>
__device__ __forceinline__ int updateSurfaceStatus(FitLane<FORM, MAT, H> &L, const Params &P,
                                                   const PlaneD &pl, int k) {
  const double denom = pl.T[0] * L.dir[0] + pl.T[1] * L.dir[1] + pl.T[2] * L.dir[2];
  if (akey(denom) != 0) {
    // along dir; the reference's path is along navDir * dir
    L.idn = rcpFast(denom);
    const double along =
        fma(-pl.T[0], L.pos[0], fma(-pl.T[1], L.pos[1], fma(-pl.T[2], L.pos[2], pl.tc))) * L.idn;
    if (akey(along) < akey(P.surfTol)) {
      ssRelease(L, kActor);
      return kOnSurface;
    }
    const double path = L.navDir < 0 ? -along : along;
    if (okey(path) > okey(-P.overstep) && akey(path) < akey(L.ss[kAborter])) {
      ssUpdate(L, along, kActor, true);
      L.hook.actorSet(L, k);
      return kReachable;
    }
  }
  return kMissed;
}

// LineSurface::intersect (LineSurface.ipp:229-262) along navDir * dir with the
// start's line (axis z)
template <int FORM, bool MAT, class H>
__device__ __forceinline__ void lineIntersect(const FitLane<FORM, MAT, H> &L, const Params &P, double &u,
                                              int &status) {
  using LT = FitLane<FORM, MAT, H>;
  double pg[3], dg[3];
  toGlobal<LT>(P, L.pos, pg);
  toGlobal<LT>(P, L.dir, dg);
  const double ea0 = L.navDir * dg[0], ea1 = L.navDir * dg[1], ea2 = L.navDir * dg[2];
  const double m0 = P.perigee[L.idx] - pg[0], m1 = P.perigee[P.stride + L.idx] - pg[1],
               m2 = P.perigee[2 * P.stride + L.idx] - pg[2];
  const double denom = 1 - ea2 * ea2;
  if (denom * denom > P.surfTol * P.surfTol) {
    u = ((m0 * ea0 + m1 * ea1 + m2 * ea2) - m2 * ea2) * rcpFast(denom);
    status = (u * u < P.surfTol * P.surfTol) ? kOnSurface : kReachable;
  } else {
    u = DBL_MAX;
    status = kMissed;
  }
}

// ---------------------------------------------------------------------------
// Bound-to-bound Jacobian at a surface: J rows 0-3 (loc0, loc1, phi, theta)
// and the time row J5 on columns (loc0, loc1, phi, theta, q/p) of the bound
// parameters at the last surface (CovarianceEngine.hpp:106-125, :269-290)
// ---------------------------------------------------------------------------
// the last surface's local axes (in the lane's frame): a plane's, or the
// start line's X and Y
template <class LT>
__device__ __forceinline__ void lastAxes(const LT &L, const Params &P, const PlaneD *planes,
                                         const Trig &tl, double U[3], double V[3]) {
  if (L.measStates == 0) {
    // LineSurface::referenceFrame at the start direction (LineSurface.ipp:
    // 46-61); the mixed form rounds its start Jacobian to FP32
    double x[3] = {-tl.sP, tl.cP, 0.}, y[3] = {0., 0., 1.};
    if (isMixed(LT::kForm)) {
      x[0] = (double)(float)x[0];
      x[1] = (double)(float)x[1];
    }
    toFrame<LT>(P, x, U);
    toFrame<LT>(P, y, V);
  } else {
    const PlaneD &pl = planes[L.lastPlane];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      U[i] = pl.U[i];
      V[i] = pl.V[i];
    }
  }
}

// position and direction columns of the leg (FP64 forms), c = 2: phi,
// 3: theta, 4: q/p.  At the start, a shift in phi also moves the point at
// distance loc0 from the line (initJacobianToGlobal, LineSurface.ipp:63-112):
// by -loc0 (cos phi, sin phi, 0); loc0 is `o`.
template <int FORM, bool MAT, class H>
__device__ __forceinline__ typename std::enable_if<isUniform(FORM)>::type
legColumn(const FitLane<FORM, MAT, H> &L, const Params &P, const Trig &t, double o, int c, double p[3],
          double v[3]) {
  using LT = FitLane<FORM, MAT, H>;
  LegState<kUniform64> g;
  if constexpr (H::kGroup > 1) { // from the lanes that carry them (the whole group calls)
    const unsigned group = 0xffu << (threadIdx.x & 24);
    double m[4];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      m[i] = __shfl_sync(group, L.g.v[i], c, 8);
      m[2 + i] = __shfl_sync(group, L.g.p[i], c, 8);
    }
    g.g = g.c[0] = m[0];
    g.c[1] = m[1];
    g.b = -m[1];
    g.r = g.a[0] = m[2];
    g.a[1] = m[3];
    g.q1 = -m[3];
    g.s = L.g.s;
  } else {
    g = L.g;
  }
  if (c == 4) {
    p[0] = g.a[0];
    p[1] = g.a[1];
    v[0] = g.c[0];
    v[1] = g.c[1];
    p[2] = v[2] = 0.;
    return;
  }
  double e[3];
  if (c == 2) {
    const double ge[3] = {-t.sT * t.sP, t.sT * t.cP, 0.};
    toFrame<LT>(P, ge, e);
  } else {
    const double ge[3] = {t.cT * t.cP, t.cT * t.sP, -t.sT};
    toFrame<LT>(P, ge, e);
  }
  p[0] = fma(g.r, e[0], g.q1 * e[1]);
  p[1] = fma(g.r, e[1], -g.q1 * e[0]);
  p[2] = g.s * e[2];
  v[0] = fma(g.g, e[0], g.b * e[1]);
  v[1] = fma(g.g, e[1], -g.b * e[0]);
  v[2] = e[2];
  if (c == 2 && L.measStates == 0) {
    const double go[3] = {-o * t.cP, -o * t.sP, 0.};
    double w[3];
    toFrame<LT>(P, go, w);
#pragma unroll
    for (int i = 0; i < 3; ++i) p[i] += w[i];
  }
}
template <bool MAT, class H>
__device__ __forceinline__ void legColumn(const FitLane<kGrid64, MAT, H> &L, const Params &P,
                                          const Trig &t, double o, int c, double p[3], double v[3]) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    if constexpr (H::kGroup > 1) { // from the lane that carries it (the whole group calls)
      const unsigned group = 0xffu << (threadIdx.x & 24);
      p[i] = __shfl_sync(group, L.g.p[i], c, 8);
      v[i] = __shfl_sync(group, L.g.v[i], c, 8);
    } else {
      p[i] = L.g.p[c - 2][i];
      v[i] = L.g.v[c - 2][i];
    }
  }
  if (c == 2 && L.measStates == 0) {
    p[0] -= o * t.cP;
    p[1] -= o * t.sP;
  }
}
// k4 of the last step
template <int FORM, bool MAT, class H>
__device__ __forceinline__ typename std::enable_if<isUniform(FORM)>::type
lastK4(const FitLane<FORM, MAT, H> &L, const Params &P, double k4[3]) {
  const double k = L.qop * P.Bz, y = L.g.y, x = y * y;
  const double w1 = k * fma(x, -0.5, 1.), w2 = k * y * fma(x, -0.25, 1.);
  k4[0] = fma(w1, L.g.dy, -w2 * L.g.dx);
  k4[1] = fma(-w1, L.g.dx, -w2 * L.g.dy);
  k4[2] = 0.;
}
template <bool MAT, class H>
__device__ __forceinline__ void lastK4(const FitLane<kGrid64, MAT, H> &L, const Params &, double k4[3]) {
#pragma unroll
  for (int i = 0; i < 3; ++i) k4[i] = L.g.k4[i];
}
template <int FORM, bool MAT, class H> __device__ __forceinline__ double legPath(const FitLane<FORM, MAT, H> &L) {
  if constexpr (isMixed(FORM)) return L.sTr;
  else return L.g.s;
}

__device__ __forceinline__ double dot3(const double a[3], const double b[3]) {
  return fma(a[0], b[0], fma(a[1], b[1], a[2] * b[2]));
}
// a . b where flat says that the z products vanish (a multiplication by a
// literal 0 costs an FP64 instruction like any other)
__device__ __forceinline__ double dotz(bool flat, const double a[3], const double b[3]) {
  return flat ? fma(a[0], b[0], a[1] * b[1]) : dot3(a, b);
}

// FP64 forms, at a surface with local axes a0, a1, where a parameter's path
// correction is s = (sp . pos column) + (sv . dir column) (sv: line only);
// f0, f1: rows of phi and theta.  All vectors in the lane's frame.
template <bool LINE, class LT>
__device__ __forceinline__ void boundRows(const LT &L, const Params &P, const PlaneD *planes,
                                          const Trig &tl, double o, const double a0[3],
                                          const double a1[3], const double sp[3],
                                          const double sv[3], const double f0[3],
                                          const double f1[3], bool time, double (&J)[4][5],
                                          double (&J5)[5]) {
  // the derivative term (EigenStepper.ipp:320-325): zero right after a reset
  double k4[3] = {0., 0., 0.}, u0 = 0., u1 = 0.;
  if (L.stepped) {
    lastK4(L, P, k4);
    u0 = dot3(a0, L.dir);
    u1 = dot3(a1, L.dir);
  }
  // vectors without a z component: the phi row (but in a turned frame), and in
  // a uniform field along z the k4 and the phi and q/p columns
  constexpr bool kFlatRow = LT::kForm != kUniformAny, kFlat = LT::kForm == kUniform64;
  const double fk0 = dotz(kFlatRow, f0, k4), fk1 = dotz(kFlat, f1, k4);
  const double dt = L.stepped ? L.dtds : 0.;
  double A0[3], A1[3];
  if (!LINE) {
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      A0[i] = fma(-u0, sp[i], a0[i]);
      A1[i] = fma(-u1, sp[i], a1[i]);
    }
  }
  {
    double U[3], V[3];
    lastAxes(L, P, planes, tl, U, V);
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const double *W = c ? V : U;
      const double s = dot3(sp, W);
      J[0][c] = LINE ? fma(-u0, s, dot3(a0, W)) : dot3(A0, W);
      J[1][c] = LINE ? fma(-u1, s, dot3(a1, W)) : dot3(A1, W);
      J[2][c] = -fk0 * s;
      J[3][c] = -fk1 * s;
      if (time) J5[c] = -dt * s;
    }
  }
#pragma unroll
  for (int c = 2; c < 5; ++c) {
    double p[3], v[3];
    legColumn(L, P, tl, o, c, p, v);
    const bool flat = kFlat && c != 3;
    const double s = LINE ? dotz(flat, sp, p) + dotz(flat, sv, v) : dotz(flat, sp, p);
    J[0][c] = LINE ? fma(-u0, s, dotz(flat, a0, p)) : dotz(flat, A0, p);
    J[1][c] = LINE ? fma(-u1, s, dotz(flat, a1, p)) : dotz(flat, A1, p);
    J[2][c] = fma(-fk0, s, dotz(kFlatRow, f0, v));
    J[3][c] = fma(-fk1, s, dotz(flat, f1, v));
    if (time) J5[c] = (c == 4) ? fma(-dt, s, legPath(L) * L.d37) : -dt * s;
  }
}

// the phi and theta rows of jacToLocal (PlaneSurface.ipp:158-189) in the
// lane's frame
template <class LT>
__device__ __forceinline__ void angleRows(const Params &P, const Trig &t, double invS, double f0[3],
                                          double f1[3]) {
  const double a[3] = {-t.sP * invS, t.cP * invS, 0.}, b[3] = {t.cP * t.cT, t.sP * t.cT, -t.sT};
  toFrame<LT>(P, a, f0);
  toFrame<LT>(P, b, f1);
}

// at a plane, FP64 forms; tr: trigonometry of the direction there
template <int FORM, bool MAT, class H>
__device__ __forceinline__ typename std::enable_if<!isMixed(FORM)>::type
boundJacobian(const FitLane<FORM, MAT, H> &L, const Params &P,
                                              const PlaneD *planes, const PlaneD &pl, bool time,
                                              Trig &tr, double (&J)[4][5], double (&J5)[5]) {
  using LT = FitLane<FORM, MAT, H>;
  double dg[3], invS;
  toGlobal<LT>(P, L.dir, dg);
  tr = trigOf(dg, invS);
  const Trig tl = trigLoad(L);
  const double o = L.measStates == 0 ? P.start[L.idx] : 0.;
  double sp[3] = {0., 0., 0.}, f0[3], f1[3];
  if (L.stepped) {
    // (the track is on this plane: idn is its)
#pragma unroll
    for (int i = 0; i < 3; ++i) sp[i] = pl.T[i] * L.idn;
  }
  angleRows<LT>(P, tr, invS, f0, f1);
  boundRows<false>(L, P, planes, tl, o, pl.U, pl.V, sp, sp, f0, f1, time, J, J5);
}

// at a plane, mixed form (boundStatePlaneMixed of the reference's
// CovarianceEngine.hpp:269-290, :106-125): the straight line's bound
// Jacobian in FP64 plus the field-induced remainder in FP32.  With JA = s I +
// dA, JB = I + dB the transported jacToGlobal splits into (G03 + s G46, G46),
// which with the direction's derivative term and the plane's projections
// gives the O(1) entries of J in FP64, and the blocks dA G46, dB G46, Ja, Jc
// with the k4 and dt/ds derivative terms, field-induced, in FP32.  J comes
// out accurate to FP32 rounding of those small terms (an FP32 J moves the
// fitted perigee by up to 3e-6 of its resolution on the 30-plane map
// telescope, mostly through the angle rows).
template <int FORM, bool MAT, class H>
__device__ __forceinline__ typename std::enable_if<isMixed(FORM)>::type
boundJacobian(const FitLane<FORM, MAT, H> &L, const Params &P,
                                              const PlaneD *planes, const PlaneD &pl, bool time,
                                              Trig &tr, double (&J)[4][5], double (&J5)[5]) {
  using LT = FitLane<FORM, MAT, H>;
  double invS;
  tr = trigOf(L.dir, invS);
  const Trig tl = trigLoad(L);
  const bool first = L.measStates == 0;
  const double s = L.sTr;
  const bool st = L.stepped;
  double g46[3][2] = {{(-tl.sT) * tl.sP, tl.cT * tl.cP}, {tl.sT * tl.cP, tl.cT * tl.sP}, {0., -tl.sT}};
  double P0[3][4], s0[4];
  {
    double U[3], V[3], o2[2] = {0., 0.};
    lastAxes(L, P, planes, tl, U, V);
    if (first) { // the mixed form's start Jacobian is rounded to FP32
      const double o = P.start[L.idx];
      o2[0] = (double)(float)(-o * tl.cP);
      o2[1] = (double)(float)(-o * tl.sP);
#pragma unroll
      for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < 2; ++c) g46[r][c] = (double)(float)g46[r][c];
    }
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      P0[r][0] = U[r];
      P0[r][1] = V[r];
      P0[r][2] = r < 2 ? fma(s, g46[r][0], o2[r]) : 0.;
      P0[r][3] = s * g46[r][1];
    }
  }
  // ---- straight-line part, FP64
  const double nv[3] = {pl.T[0] * L.idn, pl.T[1] * L.idn, pl.T[2] * L.idn};
#pragma unroll
  for (int c = 0; c < 4; ++c) { // (the phi column, c = 2, has no z)
    const double col[3] = {P0[0][c], P0[1][c], P0[2][c]};
    s0[c] = dotz(c == 2, nv, col);
  }
  double A0[3], A1[3];
  {
    const double u0 = st ? dot3(pl.U, L.dir) : 0., u1 = st ? dot3(pl.V, L.dir) : 0.;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      A0[i] = fma(-u0, nv[i], pl.U[i]);
      A1[i] = fma(-u1, nv[i], pl.V[i]);
    }
  }
  const double j24 = -tr.sP * invS, j25 = tr.cP * invS;
  const double j34 = tr.cP * tr.cT, j35 = tr.sP * tr.cT, j36 = -tr.sT;
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const double col[3] = {P0[0][c], P0[1][c], P0[2][c]};
    J[0][c] = dotz(c == 2, A0, col);
    J[1][c] = dotz(c == 2, A1, col);
    if (c >= 2) {
      const double g0 = g46[0][c - 2], g1 = g46[1][c - 2], g2 = g46[2][c - 2];
      J[2][c] = fma(j24, g0, j25 * g1);
      J[3][c] = fma(j34, g0, c == 2 ? j35 * g1 : fma(j35, g1, j36 * g2));
    } else {
      J[2][c] = 0.;
      J[3][c] = 0.;
    }
  }
  // ---- field-induced part, FP32
  float G[3][2];
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    G[r][0] = narrow(g46[r][0]);
    G[r][1] = narrow(g46[r][1]);
  }
  float dP[3][5], dD[3][5];
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    dP[r][0] = dP[r][1] = dD[r][0] = dD[r][1] = 0.f;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      dP[r][2 + c] = L.JA[r][0] * G[0][c] + L.JA[r][1] * G[1][c] + L.JA[r][2] * G[2][c];
      dD[r][2 + c] = L.JB[r][0] * G[0][c] + L.JB[r][1] * G[1][c] + L.JB[r][2] * G[2][c];
    }
    dP[r][4] = L.Ja[r];
    dD[r][4] = L.Jc[r];
  }
  const float nvf[3] = {narrow(nv[0]), narrow(nv[1]), narrow(nv[2])};
  float ds[5], sf[5];
#pragma unroll
  for (int c = 0; c < 5; ++c) {
    ds[c] = nvf[0] * dP[0][c] + nvf[1] * dP[1][c] + nvf[2] * dP[2][c];
    sf[c] = (c < 4 ? narrow(s0[c]) : 0.f) + ds[c];
  }
  float R3[5];
  if (st) {
    const float d0 = narrow(L.dir[0]), d1 = narrow(L.dir[1]), d2 = narrow(L.dir[2]);
    const float dt = (float)L.dtds;
#pragma unroll
    for (int c = 0; c < 5; ++c) {
      dP[0][c] -= d0 * ds[c];
      dP[1][c] -= d1 * ds[c];
      dP[2][c] -= d2 * ds[c];
      dD[0][c] -= L.k4[0] * sf[c];
      dD[1][c] -= L.k4[1] * sf[c];
      dD[2][c] -= L.k4[2] * sf[c];
      R3[c] = (c == 4 ? L.Jb : 0.f) - dt * sf[c];
    }
  } else {
#pragma unroll
    for (int c = 0; c < 5; ++c) R3[c] = (c == 4 ? L.Jb : 0.f);
  }
  const float *U = pl.Uf, *V = pl.Vf;
  float bad = 0.f; // NaN where an entry is not finite
  const float f24 = narrow(j24), f25 = narrow(j25), f34 = narrow(j34), f35 = narrow(j35), f36 = narrow(j36);
#pragma unroll
  for (int c = 0; c < 5; ++c) {
    const float e0 = U[0] * dP[0][c] + U[1] * dP[1][c] + U[2] * dP[2][c];
    const float e1 = V[0] * dP[0][c] + V[1] * dP[1][c] + V[2] * dP[2][c];
    const float e2 = f24 * dD[0][c] + f25 * dD[1][c];
    const float e3 = f34 * dD[0][c] + f35 * dD[1][c] + f36 * dD[2][c];
    bad = fmaf(e0, 0.f, fmaf(e1, 0.f, fmaf(e2, 0.f, fmaf(e3, 0.f, bad))));
    const double w0 = widenFinite(e0), w1 = widenFinite(e1), w2 = widenFinite(e2), w3 = widenFinite(e3);
    if (c >= 2) { // (a shift on the last plane has no field-induced part)
      J[0][c] = c < 4 ? J[0][c] + w0 : w0;
      J[1][c] = c < 4 ? J[1][c] + w1 : w1;
    }
    J[2][c] = c >= 2 && c < 4 ? J[2][c] + w2 : w2;
    J[3][c] = c >= 2 && c < 4 ? J[3][c] + w3 : w3;
    if (time) J5[c] = (double)R3[c];
  }
  if (bad != 0.f) J[0][0] = __longlong_as_double(0x7ff8000000000000LL); // and with it the gain
}

// ---------------------------------------------------------------------------
// o = A C A^T for A's rows 0-3 (columns 0-4), row 4 = e4 and time row
// (A5, 1): C the 5x5 block (upper triangle), Ct its time column (6)
// ---------------------------------------------------------------------------
__device__ __forceinline__ void sandwich(const double (&A)[4][5], const double (&A5)[5],
                                         const double (&C)[15], const double (&Ct)[6],
                                         double (&o)[21]) {
  double M[4][5];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 5; ++j) {
      double v = A[i][0] * C[u5(0, j)];
#pragma unroll
      for (int k = 1; k < 5; ++k) v = fma(A[i][k], C[u5(k, j)], v);
      M[i][j] = v;
    }
  double N[6];
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    double v = Ct[k];
#pragma unroll
    for (int l = 0; l < 5; ++l) v = fma(C[u5(k, l)], A5[l], v);
    N[k] = v;
  }
  {
    double v = Ct[5];
#pragma unroll
    for (int l = 0; l < 5; ++l) v = fma(Ct[l], A5[l], v);
#pragma unroll
    for (int k = 0; k < 5; ++k) v = fma(A5[k], N[k], v);
    N[5] = v;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
#pragma unroll
    for (int j = i; j < 4; ++j) {
      double v = M[i][0] * A[j][0];
#pragma unroll
      for (int k = 1; k < 5; ++k) v = fma(M[i][k], A[j][k], v);
      o[ut(i, j)] = v;
    }
    o[ut(i, 4)] = M[i][4];
    double v = A[i][0] * N[0];
#pragma unroll
    for (int k = 1; k < 5; ++k) v = fma(A[i][k], N[k], v);
    o[ut(i, 5)] = v;
  }
  o[ut(4, 4)] = C[u5(4, 4)];
  o[ut(4, 5)] = N[4];
  o[ut(5, 5)] = N[5];
}

// EigenStepper::update (EigenStepper.ipp:554-564) to bound parameters on a
// plane given as loc0, loc1, corrections of the angles from the direction
// with trigonometry t, and q/p: the angles' new sines and cosines (left in t)
// by angle addition, with the corrections' from Taylor series (|delta| <=
// 0.02: truncation below 1e-20 absolute); larger corrections, and directions
// within 1e-6 of the z axis, by sincos of the angles.
template <class LT>
__device__ __forceinline__ void updateState(LT &L, const Params &P, const PlaneD &pl, double loc0,
                                            double loc1, Trig &t, double dphi, double dth,
                                            double qop, bool time) {
#pragma unroll
  for (int r = 0; r < 3; ++r) L.pos[r] = fma(pl.U[r], loc0, fma(pl.V[r], loc1, pl.c[r]));
  double cP, sP, cT, sT;
  // (comparisons as integers: 0.02 and 1e-6 by their bits; NaN compares large)
  if (akey(dphi) > 0x3f947ae147ae147bLL || akey(dth) > 0x3f947ae147ae147bLL ||
      !(okey(t.sT) > 0x3eb0c6f7a0b5ed8dLL) || akey(t.sT) > 0x7ff0000000000000LL) {
    sincos(atan2(t.sP, t.cP) + dphi, &sP, &cP);
    sincos(atan2(t.sT, t.cT) + dth, &sT, &cT);
  } else {
    auto sinCosSmall = [](double d, double &sn, double &cs) {
      const double d2 = d * d;
      sn = fma(d * d2, fma(d2, fma(d2, -1. / 5040., 1. / 120.), -1. / 6.), d);
      cs = fma(d2, fma(d2, fma(d2, fma(d2, 1. / 40320., -1. / 720.), 1. / 24.), -0.5), 1.);
    };
    if constexpr (LT::kCoop) { // phi in the even lanes, theta in the odd ones
      const unsigned group = 0xffu << (threadIdx.x & 24);
      const bool odd = threadIdx.x & 1;
      const double c0 = odd ? t.cT : t.cP, s0 = odd ? t.sT : t.sP;
      double sd, cd;
      sinCosSmall(odd ? dth : dphi, sd, cd);
      const double cn = c0 * cd - s0 * sd, sn = s0 * cd + c0 * sd;
      cP = __shfl_sync(group, cn, 0, 8);
      sP = __shfl_sync(group, sn, 0, 8);
      cT = __shfl_sync(group, cn, 1, 8);
      sT = __shfl_sync(group, sn, 1, 8);
    } else {
      double sdp, cdp, sdt, cdt;
      sinCosSmall(dphi, sdp, cdp);
      sinCosSmall(dth, sdt, cdt);
      cP = t.cP * cdp - t.sP * sdp;
      sP = t.sP * cdp + t.cP * sdp;
      sT = t.sT * cdt + t.cT * sdt;
      cT = t.cT * cdt - t.sT * sdt;
    }
  }
  const double d[3] = {cP * sT, sP * sT, cT};
  toFrame<LT>(P, d, L.dir);
  t = {cP, sP, cT, sT};
  setMomentum(L, P, fabs(qop), time);
}

// The material interaction at a plane (kfm::interact's formulas for charge
// +-1), the direction's trigonometry in t, from 1/p: no square roots but
// those of E and of the new momentum, one logarithm for the energy loss
// (above beta gamma 10 the density correction's log(beta gamma) joins it) and
// one for the scattering.  Returns 1/p after the crossing.
__device__ __forceinline__ double crossMaterial(const kfm::Slab &sl, int flags, double nd, const Trig &t,
                                                double ip, double m, double &varPhi, double &varTheta,
                                                double &varQop) {
  varPhi = varTheta = varQop = 0.;
  const double pc = rcpFast(fabs(nd)); // path correction
  const double p = rcpFast(ip), x = m * ip, q2b = fma(x, x, 1.);
  if (flags & 1) {
    const double t2 = sl.x0frac * pc * q2b, a = 13.6e-3 * ip;
    const double f = fma((double)0.038f, log(t2), 1.);
    varTheta = a * a * t2 * (f * f);
    varPhi = varTheta * rcpFast(t.sT * t.sT);
  }
  if (!(flags & 2)) return ip;
  const double eps = 0.5 * kfm::kBetheK * sl.Ne * sl.t0 * pc * q2b;
  const double bg = p * (1. / m), bg2 = bg * bg, g2 = 1. + bg2;
  const double gamma = g2 * rsqrtFast(g2);
  const double mf = kfm::kElectronMass / m;
  // u wmax = (2 m_e)^2 bg^4 / (1 + 2 gamma mf + mf^2)
  double arg = (4. * kfm::kElectronMass * kfm::kElectronMass) * bg2 *
               rcpFast(fma(2. * mf, gamma, fma(mf, mf, 1.)));
  double c = sl.logI + rcpFast(q2b); // + beta^2
  if (bg < 10.0) arg *= bg2;
  else c += sl.plasma - 0.5;
  const double loss = eps * fma(0.5, log(arg), -c);
  const double k = ip * ip * (4. / kfm::kFwhmOverSigma) * eps;
  varQop = q2b * (k * k);
  const double E = m * gamma;
  if (!(m < E - loss)) return 1. / 0.; // stopped
  return rsqrtFast(fma(-loss, 2. * E - loss, p * p));
}

// any of a Jacobian's entries infinite or NaN (the smoother's NaN gain), on
// the integer pipe
template <int FORM> __device__ __forceinline__ bool anyBad(const double (&J)[4][5]) {
  // (boundJacobian's own check of the mixed form's)
  if (isMixed(FORM)) return ((unsigned)__double2hiint(J[0][0]) & 0x7fffffffu) >= 0x7ff00000u;
  unsigned m = 0;
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 5; ++c) m = max(m, (unsigned)__double2hiint(J[r][c]) & 0x7fffffffu);
  return m >= 0x7ff00000u;
}

// the 2x2 measurement update by successive scalars: with w_i = C h_i,
// S = [h_i . w_j] + V = L diag(S00, 1/i1) L^T
struct Gain {
  double l, i0, i1, e0, e1, chi2; // e: S^-1 r
};
__device__ __forceinline__ Gain gain(double S00, double S01, double S11, double r0, double r1) {
  Gain g;
  g.i0 = rcpFast(S00);
  g.l = S01 * g.i0;
  g.i1 = rcpFast(fma(-g.l, S01, S11));
  const double rp = fma(-g.l, r0, r1);
  g.e1 = rp * g.i1;
  g.e0 = fma(-g.l, g.e1, r0 * g.i0);
  // r S^-1 r as the reference forms it: with an infinite residual infinite or
  // NaN as there (GainMatrixUpdater.hpp:84-93), which decides about an outlier
  g.chi2 = fma(r0, g.e0, r1 * g.e1);
  return g;
}

// chi2 above the cut, if there is one (as integers; NaN is no outlier)
__device__ __forceinline__ bool isOutlier(const Params &P, double chi2) {
  const long long k = okey(chi2);
  return P.cutKey >= 0 && k > P.cutKey && k <= 0x7ff0000000000000LL;
}

// ---------------------------------------------------------------------------
// Actor::filter (KalmanFitter.hpp:284-350, GainMatrixUpdater.hpp:34-106) at a
// plane with a hit
// ---------------------------------------------------------------------------
template <int FORM, bool MAT, class H>
__device__ __forceinline__ void filterHit(FitLane<FORM, MAT, H> &L, const Params &P,
                                          const PlaneD *planes, int k) {
  const PlaneD &pl = planes[k];
  const int s = L.measStates;
  const bool first = s == 0;
  using LT = FitLane<FORM, MAT, H>;
  const bool states = !MAT && !LT::kTape && P.oSmoothed != nullptr; // (with material: kf_device.cuh's lane)
  const bool time = (first || states) && !LT::kTape;
  double J[4][5], J5[5] = {0., 0., 0., 0., 0.};
  Trig tr;
  boundJacobian(L, P, planes, pl, time, tr, J, J5);
  if (!first && anyBad<FORM>(J)) L.badJ = true;
  if (time) L.t = fma(legPath(L), L.dtds, L.t);
  const double d0 = L.pos[0] - pl.c[0], d1 = L.pos[1] - pl.c[1], d2 = L.pos[2] - pl.c[2];
  const double x0 = pl.U[0] * d0 + pl.U[1] * d1 + pl.U[2] * d2;
  const double x1 = pl.V[0] * d0 + pl.V[1] * d1 + pl.V[2] * d2;
  const double *mp = P.meas + (size_t)k * 5 * P.stride + L.idx;
  const double m0 = mp[0], m1 = mp[P.stride], v00 = mp[2 * P.stride], v01 = mp[3 * P.stride],
               v11 = mp[4 * P.stride];
  if (first) L.firstPlane = k;
  Trig tn = tr;
  bool outlier;
  if constexpr (!MAT) {
    // F <- J F, column by column; its time row in the state's record
    double h0[5], h1[5], T5[5];
    if (first) {
#pragma unroll
      for (int c = 0; c < 5; ++c) {
#pragma unroll
        for (int r = 0; r < 4; ++r) L.F(r, c) = J[r][c];
        h0[c] = J[0][c];
        h1[c] = J[1][c];
        T5[c] = J5[c];
      }
    } else {
#pragma unroll
      for (int c = 0; c < 5; ++c) {
        const double f0 = L.F(0, c), f1 = L.F(1, c), f2 = L.F(2, c), f3 = L.F(3, c);
        double n[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          double v = c == 4 ? fma(J[r][0], f0, J[r][4]) : J[r][0] * f0;
          v = fma(J[r][1], f1, v);
          v = fma(J[r][2], f2, v);
          n[r] = fma(J[r][3], f3, v);
          L.F(r, c) = n[r];
        }
        h0[c] = n[0];
        h1[c] = n[1];
        if (states) {
          double v = *recPtr(P, L, s - 1, kRecT + c);
          if (c == 4) v += J5[4];
          T5[c] = v + J5[0] * f0 + J5[1] * f1 + J5[2] * f2 + J5[3] * f3;
        }
      }
    }
    if constexpr (LT::kTape) L.hook.event(L, k, tr, J, x0, x1);
    if (time) {
      // x_p - F D, F
      double x[6] = {x0, x1, 0., 0., L.qop, L.t};
      if (states) {
        x[2] = atan2(tr.sP, tr.cP);
        x[3] = atan2(tr.sT, tr.cT);
        if (!first) {
#pragma unroll
          for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int c = 0; c < 5; ++c) x[r] = fma(-L.F(r, c), L.D(c), x[r]);
          x[4] -= L.D(4);
          x[5] -= L.D(5);
#pragma unroll
          for (int c = 0; c < 5; ++c) x[5] = fma(-T5[c], L.D(c), x[5]);
        }
      }
#pragma unroll
      for (int e = 0; e < 6; ++e) *recPtr(P, L, s, kRecX + e) = x[e];
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 5; ++c) *recPtr(P, L, s, kRecF + 5 * r + c) = L.F(r, c);
#pragma unroll
      for (int c = 0; c < 5; ++c) *recPtr(P, L, s, kRecT + c) = T5[c];
      if (first) {
        *recPtr(P, L, 0, kRecTrig + 0) = tr.cP;
        *recPtr(P, L, 0, kRecTrig + 1) = tr.sP;
        *recPtr(P, L, 0, kRecTrig + 2) = tr.cT;
        *recPtr(P, L, 0, kRecTrig + 3) = tr.sT;
      }
    }
    double C[15], w0[5], w1[5];
#pragma unroll
    for (int e = 0; e < 15; ++e) C[e] = L.C0(e);
#pragma unroll
    for (int i = 0; i < 5; ++i) {
      double a = C[u5(i, 0)] * h0[0], b = C[u5(i, 0)] * h1[0];
#pragma unroll
      for (int j = 1; j < 5; ++j) {
        a = fma(C[u5(i, j)], h0[j], a);
        b = fma(C[u5(i, j)], h1[j], b);
      }
      w0[i] = a;
      w1[i] = b;
    }
    double a00 = h0[0] * w0[0], a01 = h1[0] * w0[0], a11 = h1[0] * w1[0];
#pragma unroll
    for (int i = 1; i < 5; ++i) {
      a00 = fma(h0[i], w0[i], a00);
      a01 = fma(h1[i], w0[i], a01);
      a11 = fma(h1[i], w1[i], a11);
    }
    const Gain g = gain(a00 + v00, a01 + v01, a11 + v11, m0 - x0, m1 - x1);
    outlier = isOutlier(P, g.chi2);
    if constexpr (LT::kTape) L.hook.update(w0, w1, g);
    if (!outlier) {
      double dl[5];
#pragma unroll
      for (int i = 0; i < 5; ++i) {
        dl[i] = fma(w0[i], g.e0, w1[i] * g.e1);
        L.D(i) += dl[i];
      }
      double w50 = 0., w51 = 0.;
      if (L.timeCorr) {
#pragma unroll
        for (int j = 0; j < 5; ++j) {
          w50 = fma(L.Ct(j), h0[j], w50);
          w51 = fma(L.Ct(j), h1[j], w51);
        }
      }
      double dphi = L.F(2, 0) * dl[0], dth = L.F(3, 0) * dl[0];
#pragma unroll
      for (int c = 1; c < 5; ++c) {
        dphi = fma(L.F(2, c), dl[c], dphi);
        dth = fma(L.F(3, c), dl[c], dth);
      }
      if (states) { // the state's filtered time
#pragma unroll
        for (int c = 0; c < 5; ++c) L.t = fma(T5[c], dl[c], L.t);
        L.t += w50 * g.e0 + w51 * g.e1;
      }
      double a0[5], a1[5];
#pragma unroll
      for (int i = 0; i < 5; ++i) {
        w1[i] = fma(-g.l, w0[i], w1[i]);
        a0[i] = w0[i] * g.i0;
        a1[i] = w1[i] * g.i1;
      }
#pragma unroll
      for (int i = 0; i < 5; ++i)
#pragma unroll
        for (int j = i; j < 5; ++j)
          L.C0(u5(i, j)) = fma(-a0[i], w0[j], fma(-a1[i], w1[j], C[u5(i, j)]));
      if (L.timeCorr) {
        L.D(5) += w50 * g.e0 + w51 * g.e1;
        const double z = fma(-g.l, w50, w51);
#pragma unroll
        for (int i = 0; i < 5; ++i) L.Ct(i) = fma(-a0[i], w50, fma(-a1[i], z, L.Ct(i)));
        L.Ct(5) = L.Ct(5) - w50 * g.i0 * w50 - z * g.i1 * z;
      }
      L.chi2 += g.chi2;
      updateState(L, P, pl, x0 + fma(a00, g.e0, a01 * g.e1), x1 + fma(a01, g.e0, a11 * g.e1), tn,
                  dphi, dth, L.qop + dl[4], states);
    }
  } else {
    // ---- process noise: current covariance C (5x5) and X = cov(first state,
    // current state)
    double C[15];
    if (first) {
      double S[15], St[6], o[21];
#pragma unroll
      for (int i = 0; i < 6; ++i)
#pragma unroll
        for (int j = i; j < 6; ++j) {
          const double v = P.scov[(size_t)ut(i, j) * P.stride + L.idx];
          if (j < 5) S[u5(i, j)] = v;
          else St[i] = v;
        }
      sandwich(J, J5, S, St, o);
#pragma unroll
      for (int e = 0; e < 21; ++e) L.P1(e) = o[e];
#pragma unroll
      for (int i = 0; i < 6; ++i)
#pragma unroll
        for (int j = 0; j < 5; ++j) L.X(i, j) = o[sidx(i, j)];
#pragma unroll
      for (int i = 0; i < 5; ++i)
#pragma unroll
        for (int j = i; j < 5; ++j) C[u5(i, j)] = o[ut(i, j)];
      *recPtr(P, L, 0, kRecX + 0) = x0;
      *recPtr(P, L, 0, kRecX + 1) = x1;
      *recPtr(P, L, 0, kRecX + 4) = L.qop;
      *recPtr(P, L, 0, kRecX + 5) = L.t;
      *recPtr(P, L, 0, kRecTrig + 0) = tr.cP;
      *recPtr(P, L, 0, kRecTrig + 1) = tr.sP;
      *recPtr(P, L, 0, kRecTrig + 2) = tr.cT;
      *recPtr(P, L, 0, kRecTrig + 3) = tr.sT;
    } else {
      double O[15];
#pragma unroll
      for (int e = 0; e < 15; ++e) O[e] = L.C(e);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        double M[5];
#pragma unroll
        for (int j = 0; j < 5; ++j) {
          double v = J[i][0] * O[u5(0, j)];
#pragma unroll
          for (int l = 1; l < 5; ++l) v = fma(J[i][l], O[u5(l, j)], v);
          M[j] = v;
        }
#pragma unroll
        for (int j = i; j < 4; ++j) {
          double v = M[0] * J[j][0];
#pragma unroll
          for (int l = 1; l < 5; ++l) v = fma(M[l], J[j][l], v);
          C[u5(i, j)] = v;
        }
        C[u5(i, 4)] = M[4];
      }
      C[u5(4, 4)] = O[u5(4, 4)];
#pragma unroll
      for (int r = 0; r < 6; ++r) {
        double x[5];
#pragma unroll
        for (int j = 0; j < 5; ++j) x[j] = L.X(r, j);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          double v = x[0] * J[i][0];
#pragma unroll
          for (int j = 1; j < 5; ++j) v = fma(x[j], J[i][j], v);
          L.X(r, i) = v;
        }
      }
    }
    const Gain g = gain(C[0] + v00, C[1] + v01, C[u5(1, 1)] + v11, m0 - x0, m1 - x1);
    outlier = isOutlier(P, g.chi2);
    if (!outlier) {
      double w0[5], w1[5], a0[5], a1[5], dl[5];
#pragma unroll
      for (int i = 0; i < 5; ++i) {
        w0[i] = C[u5(i, 0)];
        const double b = C[u5(i, 1)];
        dl[i] = fma(w0[i], g.e0, b * g.e1);
        w1[i] = fma(-g.l, w0[i], b);
        a0[i] = w0[i] * g.i0;
        a1[i] = w1[i] * g.i1;
      }
      double y0[6], y1[6], b0[6], b1[6];
#pragma unroll
      for (int r = 0; r < 6; ++r) {
        y0[r] = L.X(r, 0);
        const double b = L.X(r, 1);
        L.D(r) += fma(y0[r], g.e0, b * g.e1);
        y1[r] = fma(-g.l, y0[r], b);
        b0[r] = y0[r] * g.i0;
        b1[r] = y1[r] * g.i1;
#pragma unroll
        for (int j = 0; j < 5; ++j)
          L.X(r, j) = fma(-b0[r], w0[j], fma(-b1[r], w1[j], L.X(r, j)));
      }
#pragma unroll
      for (int i = 0; i < 6; ++i)
#pragma unroll
        for (int j = i; j < 6; ++j)
          L.P1(ut(i, j)) = fma(-b0[i], y0[j], fma(-b1[i], y1[j], L.P1(ut(i, j))));
#pragma unroll
      for (int i = 0; i < 5; ++i)
#pragma unroll
        for (int j = i; j < 5; ++j)
          C[u5(i, j)] = fma(-a0[i], w0[j], fma(-a1[i], w1[j], C[u5(i, j)]));
      L.chi2 += g.chi2;
      updateState(L, P, pl, x0 + dl[0], x1 + dl[1], tn, dl[2], dl[3], L.qop + dl[4], false);
    }
    // the material effects after the filtering (KalmanFitter.hpp:344-345)
    if (P.planeSlab[k].valid) {
      double vPhi, vTheta, vQop;
      const double ip = crossMaterial(P.planeSlab[k], P.materialEffects, dot3(pl.T, L.dir), tn,
                                      fabs(L.qop), P.mass, vPhi, vTheta, vQop);
      setMomentum(L, P, ip, false);
      C[u5(2, 2)] = smax(0., C[u5(2, 2)] + vPhi);
      C[u5(3, 3)] = smax(0., C[u5(3, 3)] + vTheta);
      C[u5(4, 4)] = smax(0., C[u5(4, 4)] + vQop);
    }
#pragma unroll
    for (int e = 0; e < 15; ++e) L.C(e) = C[e];
  }
  // reinitializeJacobians (CovarianceEngine.hpp:169-201): at the predicted
  // direction, or with faithful_jacobian = 0 at the filtered one
  if constexpr (LT::kTape) L.hook.eventEnd(outlier, tn);
  const Trig &tg = (P.faithful || outlier) ? tr : tn;
  trigSave(L, tg);
  legReset(L, tg);
  L.lastPlane = k;
  L.measStates++;
}

// ---------------------------------------------------------------------------
// Actor::finalize (KalmanFitter.hpp:360-393): the smoothed first state
// becomes the stepper's; false where the smoother's gain is NaN
// ---------------------------------------------------------------------------
template <int FORM, bool MAT, class H>
__device__ __forceinline__ bool finalizeSmooth(FitLane<FORM, MAT, H> &L, const Params &P,
                                               const PlaneD *planes) {
  L.smoothed = true;
  if (L.badJ) return false;
  const double r0 = *recPtr(P, L, 0, kRecX), r1 = *recPtr(P, L, 0, kRecX + 1);
  Trig t = {*recPtr(P, L, 0, kRecTrig), *recPtr(P, L, 0, kRecTrig + 1), *recPtr(P, L, 0, kRecTrig + 2),
            *recPtr(P, L, 0, kRecTrig + 3)};
  double x[4] = {r0, r1, 0., 0.};
  double qop = *recPtr(P, L, 0, kRecX + 4) + L.D(4);
  double tm = *recPtr(P, L, 0, kRecX + 5) + L.D(5);
  if constexpr (!MAT) {
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int c = 0; c < 5; ++c) x[r] = fma(*recPtr(P, L, 0, kRecF + 5 * r + c), L.D(c), x[r]);
#pragma unroll
    for (int c = 0; c < 5; ++c) tm = fma(*recPtr(P, L, 0, kRecT + c), L.D(c), tm);
    if (P.oSmoothed) {
      double C[15], Ct[6];
#pragma unroll
      for (int e = 0; e < 15; ++e) C[e] = L.C0(e);
#pragma unroll
      for (int e = 0; e < 6; ++e) Ct[e] = L.Ct(e);
      for (int s = 0; s < L.measStates; ++s) {
        double A[4][5], A5[5], o[21], xs[6];
#pragma unroll
        for (int e = 0; e < 6; ++e) xs[e] = *recPtr(P, L, s, kRecX + e);
        xs[4] += L.D(4);
        xs[5] += L.D(5);
#pragma unroll
        for (int c = 0; c < 5; ++c) {
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            A[r][c] = *recPtr(P, L, s, kRecF + 5 * r + c);
            xs[r] = fma(A[r][c], L.D(c), xs[r]);
          }
          A5[c] = *recPtr(P, L, s, kRecT + c);
          xs[5] = fma(A5[c], L.D(c), xs[5]);
        }
        sandwich(A, A5, C, Ct, o);
        double *out = P.oSmoothed + (size_t)s * 27 * P.stride + L.idx;
#pragma unroll
        for (int e = 0; e < 6; ++e) out[(size_t)e * P.stride] = xs[e];
#pragma unroll
        for (int e = 0; e < 21; ++e) out[(size_t)(6 + e) * P.stride] = o[e];
      }
    }
  } else {
#pragma unroll
    for (int r = 0; r < 4; ++r) x[r] += L.D(r);
  }
  // the time's q/p factor of a leg that has begun: its own momentum's (d37 is
  // kept up only where a surface's Jacobian has a time row)
  double d37 = 0.;
  if (L.stepped) {
    const double m = P.mass * L.qop;
    d37 = P.mass * m * rsqrtFast(fma(m, m, 1.));
    if constexpr (isMixed(FORM)) L.Jb += (float)(L.sTr * (d37 - (double)L.d37f));
  }
  const PlaneD &pl = planes[L.firstPlane];
  updateState(L, P, pl, x[0], x[1], t, x[2], x[3], qop, true);
  if (!P.faithful) {
    // jacToGlobal from the smoothed state's own plane and direction
    const Trig t0 = trigLoad(L);
    trigSave(L, t);
    L.lastPlane = L.firstPlane;
    if constexpr (FORM == kGrid64) {
      if (L.stepped) legRebase(L, P, t0, t);
      else legReset(L, t);
    }
  }
  // (a leg that had begun when the track ran out of planes goes on)
  if constexpr (!isMixed(FORM)) *recPtr(P, L, 0, kRecRest) = L.stepped ? legPath(L) * (d37 - L.d37) : 0.;
  L.t = fma(-legPath(L), L.dtds, tm);
  L.navDir = -1;
  ssInit(L, -1. * DBL_MAX);
  return true;
}

// boundState<LineSurface> towards the perigee line (axis z) and the outputs
template <int FORM, bool MAT, class H>
__device__ __forceinline__ void reachPerigee(FitLane<FORM, MAT, H> &L, const Params &P,
                                             const PlaneD *planes) {
  using LT = FitLane<FORM, MAT, H>;
  const Trig tl = trigLoad(L);
  double pg[3], dg[3], out[6], cov[21];
  toGlobal<LT>(P, L.pos, pg);
  toGlobal<LT>(P, L.dir, dg);
  double pc[3];
#pragma unroll
  for (int e = 0; e < 3; ++e) pc[e] = pg[e] - P.perigee[(size_t)e * P.stride + L.idx];
  double C[15], Ct[6];
  if constexpr (MAT) {
#pragma unroll
    for (int i = 0; i < 6; ++i)
#pragma unroll
      for (int j = i; j < 6; ++j) {
        if (j < 5) C[u5(i, j)] = L.P1(ut(i, j));
        else Ct[i] = L.P1(ut(i, j));
      }
  } else {
#pragma unroll
    for (int e = 0; e < 15; ++e) C[e] = L.C0(e);
#pragma unroll
    for (int e = 0; e < 6; ++e) Ct[e] = L.Ct(e);
  }
  if constexpr (!isMixed(FORM)) {
    double invS;
    const Trig tr = trigOf(dg, invS);
    // X = z x d / |z x d|, Y = z (LineSurface::referenceFrame), the path
    // correction of LineSurface::derivativeFactors (LineSurface.ipp:145-182)
    const double X[3] = {-tr.sP, tr.cP, 0.}, Y[3] = {0., 0., 1.};
    const double nrm = rcpFast(1. - dg[2] * dg[2]);
    const double on = L.stepped ? 1. : 0.;
    const double k = nrm * (1. - pc[2]) * on;
    const double sp[3] = {dg[0] * k, dg[1] * k, 0.};
    const double sv[3] = {pc[0] * nrm * on, pc[1] * nrm * on, pc[2] * nrm * on};
    double f0[3], f1[3], fX[3], fY[3], fs[3], fv[3], J[4][5], J5[5];
    angleRows<LT>(P, tr, invS, f0, f1);
    toFrame<LT>(P, X, fX);
    toFrame<LT>(P, Y, fY);
    toFrame<LT>(P, sp, fs);
    toFrame<LT>(P, sv, fv);
    boundRows<true>(L, P, planes, tl, 0., fX, fY, fs, fv, f0, f1, true, J, J5);
    J5[4] += *recPtr(P, L, 0, kRecRest); // (boundRows gives all of the leg the last momentum)
    if constexpr (MAT) {
      sandwich(J, J5, C, Ct, cov);
    } else {
      // onto the start parameters: J F1
      double A[4][5], A5[5];
#pragma unroll
      for (int c = 0; c < 5; ++c) {
        double f[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) f[r] = *recPtr(P, L, 0, kRecF + 5 * r + c);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          double v = c == 4 ? J[r][4] : 0.;
#pragma unroll
          for (int l = 0; l < 4; ++l) v = fma(J[r][l], f[l], v);
          A[r][c] = v;
        }
        double v = *recPtr(P, L, 0, kRecT + c) + (c == 4 ? J5[4] : 0.);
#pragma unroll
        for (int l = 0; l < 4; ++l) v = fma(J5[l], f[l], v);
        A5[c] = v;
      }
      sandwich(A, A5, C, Ct, cov);
    }
  } else {
    // mixed form: the Jacobian to the line, and the time row and column of
    // the covariance, in FP32 as the transport; the first state's covariance
    // and the 5x5 block in FP64
    double cs[21];
    if constexpr (MAT) {
#pragma unroll
      for (int e = 0; e < 21; ++e) cs[e] = L.P1(e);
    } else {
      double A[4][5], A5[5];
#pragma unroll
      for (int c = 0; c < 5; ++c) {
#pragma unroll
        for (int r = 0; r < 4; ++r) A[r][c] = *recPtr(P, L, 0, kRecF + 5 * r + c);
        A5[c] = *recPtr(P, L, 0, kRecT + c);
      }
      sandwich(A, A5, C, Ct, cs);
    }
    float Pt[3][5], Dd[3][5], R3[5] = {0.f, 0.f, 0.f, 0.f, L.Jb};
    {
      double U[3], V[3];
      lastAxes(L, P, planes, tl, U, V);
      const double g46[3][2] = {{(-tl.sT) * tl.sP, tl.cT * tl.cP}, {tl.sT * tl.cP, tl.cT * tl.sP}, {0., -tl.sT}};
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        Pt[r][0] = (float)U[r];
        Pt[r][1] = (float)V[r];
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const float g0 = (float)g46[0][c], g1 = (float)g46[1][c], g2 = (float)g46[2][c];
          Pt[r][2 + c] = (float)(0. + L.sTr * g46[r][c]) + L.JA[r][0] * g0 + L.JA[r][1] * g1 + L.JA[r][2] * g2;
          Dd[r][2 + c] = (float)g46[r][c] + L.JB[r][0] * g0 + L.JB[r][1] * g1 + L.JB[r][2] * g2;
        }
        Pt[r][4] = L.Ja[r];
        Dd[r][0] = Dd[r][1] = 0.f;
        Dd[r][4] = L.Jc[r];
      }
    }
    double mX[3], mY[3], mD[3];
    lineFrame(dg, mX, mY, mD);
    const float rX[3] = {(float)mX[0], (float)mX[1], (float)mX[2]};
    const float rY[3] = {(float)mY[0], (float)mY[1], (float)mY[2]};
    const float dr[3] = {(float)dg[0], (float)dg[1], (float)dg[2]};
    const float lc = rY[0] * dr[0] + rY[1] * dr[1] + rY[2] * dr[2];
    const float n0 = dr[0] - lc * rY[0], n1 = dr[1] - lc * rY[1], n2 = dr[2] - lc * rY[2];
    const float nrm = 1.f / (1.f - lc * lc);
    const float p0 = (float)pc[0], p1 = (float)pc[1], p2 = (float)pc[2];
    const float x = dr[0], y = dr[1], cosT = dr[2];
    const float sinT = sqrt(x * x + y * y), invS = 1.f / sinT, cosP = x * invS, sinP = y * invS;
    const float j24 = -sinP * invS, j25 = cosP * invS;
    const float j34 = cosP * cosT, j35 = sinP * cosT, j36 = -sinT;
    float J[6][5];
#pragma unroll
    for (int c = 0; c < 5; ++c) {
      const float s = n0 * Pt[0][c] + n1 * Pt[1][c] + n2 * Pt[2][c];
      const float e0 = rY[0] * s - Dd[0][c], e1 = rY[1] * s - Dd[1][c], e2 = rY[2] * s - Dd[2][c];
      const float row = p0 * e0 + p1 * e1 + p2 * e2;
      const float sV = nrm * (s - row);
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        const float der = L.stepped ? dr[r] : 0.f, dk = L.stepped ? L.k4[r] : 0.f;
        Pt[r][c] -= der * sV;
        Dd[r][c] -= dk * sV;
      }
      R3[c] -= (L.stepped ? (float)L.dtds : 0.f) * sV;
      J[0][c] = rX[0] * Pt[0][c] + rX[1] * Pt[1][c] + rX[2] * Pt[2][c];
      J[1][c] = rY[0] * Pt[0][c] + rY[1] * Pt[1][c] + rY[2] * Pt[2][c];
      J[2][c] = j24 * Dd[0][c] + j25 * Dd[1][c];
      J[3][c] = j34 * Dd[0][c] + j35 * Dd[1][c] + j36 * Dd[2][c];
      J[4][c] = (c == 4) ? 1.f : 0.f;
      J[5][c] = R3[c];
    }
    float N[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      float s = (float)cs[sidx(k, 5)];
#pragma unroll
      for (int l = 0; l < 5; ++l) s += (float)cs[sidx(k, l)] * J[5][l];
      N[k] = s;
    }
    float T5[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      float s = (i == 4) ? N[4] : (i == 5 ? N[5] : 0.f);
      if (i != 4) {
#pragma unroll
        for (int k = 0; k < 5; ++k) s += J[i][k] * N[k];
      }
      T5[i] = s;
    }
    double A[4][5], S[15];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int c = 0; c < 5; ++c) A[i][c] = (double)J[i][c];
#pragma unroll
    for (int i = 0; i < 5; ++i)
#pragma unroll
      for (int j = i; j < 5; ++j) S[u5(i, j)] = cs[ut(i, j)];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      double M[5];
#pragma unroll
      for (int j = 0; j < 5; ++j) {
        double v = A[i][0] * S[u5(0, j)];
#pragma unroll
        for (int l = 1; l < 5; ++l) v = fma(A[i][l], S[u5(l, j)], v);
        M[j] = v;
      }
#pragma unroll
      for (int j = i; j < 4; ++j) {
        double v = M[0] * A[j][0];
#pragma unroll
        for (int l = 1; l < 5; ++l) v = fma(M[l], A[j][l], v);
        cov[ut(i, j)] = v;
      }
      cov[ut(i, 4)] = M[4];
    }
    cov[ut(4, 4)] = S[u5(4, 4)];
#pragma unroll
    for (int i = 0; i < 6; ++i) cov[ut(i, 5)] = (double)T5[i];
  }
  // LineSurface::globalToLocal (LineSurface.ipp:200-220) and the angles
  const double r = sqrt(pc[0] * pc[0] + pc[1] * pc[1]);
  out[0] = ((-dg[1]) * pc[0] + dg[0] * pc[1] < 0.) ? -r : r;
  out[1] = pc[2];
  out[2] = atan2(dg[1], dg[0]);
  out[3] = atan2(sqrt(dg[0] * dg[0] + dg[1] * dg[1]), dg[2]);
  out[4] = L.qop;
  out[5] = fma(legPath(L), L.dtds, L.t);
#pragma unroll
  for (int e = 0; e < 6; ++e) P.oParams[(size_t)e * P.stride + L.idx] = out[e];
#pragma unroll
  for (int e = 0; e < 21; ++e) P.oCov[(size_t)e * P.stride + L.idx] = cov[e];
}

// ---------------------------------------------------------------------------
// EigenStepper::State from BoundParameters<LineSurface> (EigenStepper.hpp:40-61)
// and the navigator initialisation
// ---------------------------------------------------------------------------
template <int FORM, bool MAT, class H>
__device__ __forceinline__ void initFit(FitLane<FORM, MAT, H> &L, const Params &P, const PlaneD *planes,
                                        int64_t i, int64_t wsIdx) {
  using LT = FitLane<FORM, MAT, H>;
  L.idx = i;
  L.wsIdx = wsIdx;
  L.pc = PC_DONE;
  L.parked = 0;
  L.steps = 0;
  L.rkSteps = 0;
  L.rkTrials = 0;
  L.chi2 = 0.;
  L.measStates = 0;
  L.firstPlane = L.lastPlane = 0;
  L.next = 0;
  L.current = -1;
  L.navCache = -1;
  L.navCacheSt = 0;
  L.navCacheLim = 0;
  L.targetReached = false;
  L.navBreak = false;
  L.smoothed = false;
  L.finished = false;
  L.result = true;
  L.tn = false;
  L.badJ = false;
  L.timeCorr = false;
  L.status = KF_TRACK_NOT_FITTED;
  if (i < 0 || i >= P.n) return;
  double sp[6], per[3];
#pragma unroll
  for (int e = 0; e < 6; ++e) sp[e] = P.start[(size_t)e * P.stride + i];
#pragma unroll
  for (int e = 0; e < 3; ++e) per[e] = P.perigee[(size_t)e * P.stride + i];
  int ns = P.nplanes ? P.nplanes[i] : P.nSurf;
  L.nSeq = min(max(ns, 0), P.nSurf);
  L.mask = P.mask ? P.mask[i] : ~0ull;
  L.nHits = __popcll(L.mask & ((L.nSeq >= 64) ? ~0ull : ((1ull << L.nSeq) - 1ull)));
  bool ok = isfinite(sp[4]) && sp[4] != 0.;
#pragma unroll
  for (int e = 0; e < 6; ++e) ok = ok && isfinite(sp[e]);
  if (!ok) {
    L.status = KF_TRACK_BAD_INPUT;
    return;
  }
  if (L.nHits == 0) {
    L.status = KF_TRACK_NO_HITS;
    return;
  }
  // momentum and position on the line (coordinate_transformations.hpp:45-76,
  // LineSurface.ipp:184-198)
  double sph, cph, sth, cth;
  sincos(sp[2], &sph, &cph);
  sincos(sp[3], &sth, &cth);
  const double ip = fabs(sp[4]);
  const double dg[3] = {sth * cph, sth * sph, cth};
  // the radial axis (0,0,1) x d / |...|, undefined (NaN) along the line
  const double sg = sth > 0. ? 1. : (sth < 0. ? -1. : __longlong_as_double(0x7ff8000000000000LL));
  const double r = sp[0] * sg;
  const double pg[3] = {fma(-r, sph, per[0]), fma(r, cph, per[1]), (sp[1] + per[2]) + 0. * r};
  toFrame<LT>(P, pg, L.pos);
  toFrame<LT>(P, dg, L.dir);
  L.q = (sp[4] > 0) ? 1. : -1.;
  L.t = sp[5];
  L.navDir = 1;
  ssInit(L, DBL_MAX);
#pragma unroll
  for (int r = 0; r < 6; ++r) {
#pragma unroll
    for (int c = r; c < 6; ++c) {
      const double v = MAT ? 0. : P.scov[(size_t)ut(r, c) * P.stride + i];
      if (!MAT) {
        if (c < 5) L.C0(u5(r, c)) = v;
        else L.Ct(r) = v;
        if (c == 5 && r < 5 && v != 0.) L.timeCorr = true;
      }
    }
    L.D(r) = 0.;
  }
  setMomentum(L, P, ip, true);
  double invS;
  const Trig t = trigOf(dg, invS);
  trigSave(L, t);
  legReset(L, t);
  L.pc = PC_PRE;
  navStatus(L, P, planes);
}

// ---------------------------------------------------------------------------
// The Kalman actor (KalmanFitter.hpp:216-273), as kf_device.cuh's: with heavy
// == false it only runs between surfaces, where no filter update, smoothing or
// final transport can be due, and returns false without touching the state
// otherwise.  With heavy == true it runs the stage L.parked and returns false
// where another stage of the same call is left (then in L.parked).
// ---------------------------------------------------------------------------
// Stages, in the order in which a warp takes them up: a lane past its last hit
// waits for the lanes that still have planes, so that a warp smooths, steps
// back and reaches the line once, and not once for each last plane among its
// tracks (a lane stepping back early also kept the others waiting at their
// next plane for all of its way).  1M tracks of 5-30 planes with 10 % holes
// 24.9 -> 22.4 ms, 65537 of them mixed 1.76 -> 1.63 ms, 20011 with their
// smoothed states 2.13 -> 1.60 ms; tracks of equal length the same.
enum EventStage { kAtPlane = 1, kAtSmoothing = 2, kAtLine = 3 };

// whether this lane's pending event is of the stage that the warp runs next
// (the whole warp calls)
template <class LT> __device__ __forceinline__ bool eventDue(const LT &L) {
  const unsigned stage = L.parked ? L.parked : kAtLine + 1;
  return __reduce_min_sync(0xffffffffu, stage) == stage && L.parked;
}

template <int FORM, bool MAT, class H>
__device__ __forceinline__ bool actor(FitLane<FORM, MAT, H> &L, const Params &P, const PlaneD *planes,
                                      bool heavy) {
  const bool onPlane = L.current >= 0 && !L.smoothed && !L.finished;
  const bool hit = onPlane && ((L.mask >> L.current) & 1ull);
  if (!heavy) {
    // every plane, hit or not, is a meeting point of the warp (see fitWarp)
    const bool fin = (L.measStates == L.nHits || (L.measStates > 0 && L.navBreak)) && !L.smoothed &&
                     !L.finished && P.smoothing;
    if (onPlane || fin) return false;
    if (L.smoothed && !L.finished) {
      if (L.targetReached || L.current == -2) return false;
      double u;
      int st;
      lineIntersect(L, P, u, st);
      if (st == kOnSurface) return false;
      ssUpdate(L, L.navDir * u, kAborter, false);
    } else if ((L.measStates == L.nHits || (L.measStates > 0 && L.navBreak)) && !L.smoothed &&
               !L.finished) {
      L.finished = true; // no smoothing asked for
    }
    return true;
  }
  if (L.parked == kAtPlane) {
    if (hit) filterHit(L, P, planes, L.current);
    if ((L.measStates == L.nHits || (L.measStates > 0 && L.navBreak)) && !L.smoothed &&
        !L.finished) {
      if (P.smoothing) {
        L.parked = kAtSmoothing;
        return false;
      }
      L.finished = true;
    }
    if (L.smoothed && !L.finished) { // (no plane: the line is reached)
      L.parked = kAtLine;
      return false;
    }
    return true;
  }
  if (L.parked == kAtSmoothing && !finalizeSmooth(L, P, planes)) L.result = false;
  // SurfaceReached (StandardAborters.hpp:88-132)
  bool reached = true;
  if (L.current == -2) {
    L.targetReached = true;
  } else if (!L.targetReached) {
    double u;
    int st;
    lineIntersect(L, P, u, st);
    reached = (st == kOnSurface);
    if (reached) {
      L.current = -2;
      L.targetReached = true;
    } else {
      ssUpdate(L, L.navDir * u, kAborter, false);
    }
  }
  if (reached) {
    if (L.parked == kAtSmoothing) {
      L.parked = kAtLine;
      return false;
    }
    reachPerigee(L, P, planes);
    L.finished = true;
  }
  return true;
}

// Kalman aborter (KalmanFitter.hpp:682-694); the path limit
// (StandardAborters.hpp:37-56) is DBL_MAX here and never reached
template <int FORM, bool MAT, class H>
__device__ __forceinline__ bool aborters(FitLane<FORM, MAT, H> &L, const Params &) {
  return !L.result || L.finished || L.targetReached;
}

// the pending actor call, or the stage of it that is due, and after its last
// the rest of its iteration (see advance)
template <int FORM, bool MAT, class H>
__device__ __forceinline__ void runEvent(FitLane<FORM, MAT, H> &L, const Params &P, const PlaneD *planes) {
  if (!actor(L, P, planes, true)) return;
  L.parked = 0;
  if (L.pc == PC_POST) {
    finish(L, P);
    L.pc = PC_DONE;
  } else if (aborters(L, P)) {
    if (L.pc == PC_ACT) L.tn = true;
    L.pc = PC_POST;
  } else {
    navTarget(L, P, planes);
    if (L.pc == PC_ACT) L.steps++;
    L.pc = PC_LOOP;
  }
}

} // namespace kfd
