// kf_adjoint_z.cu — the chi2 adjoint for a uniform field along z: the fit's
// own formulation (kf_fit.cuh), differentiated by hand.
//
// Objective (see kf_adjoint.cu): chi2 = sum over non-outlier states k of
// rho^T V^-1 rho, rho = m - H x_s.  In the start frame x_s = x_p + F E with
// E_k = sum over hits j >= k of dl_j, dl_j the update's K0 r, so
// rho_k = r_k - (h_0 . E_k, h_1 . E_k) with r the predicted residual and h the
// first two rows of F: the smoother's adjoint is the running sum
// G_j = sum over k <= j of dchi2/dE_k that each hit's dl receives.  The time
// is part of no measurement and does not occur.
//
// A. forward: the fit's lane, whose hook stores per state (F, C0, the update
//    dl, the predicted state, the leg's transport scalars; 70 words) and
//    tapes the RK steps and step constraints (13 and 2 words) and per hit the
//    Jacobian, C0 h and the gain (36);
// B. chi2 and sum of dchi2/dE over the states;
// C. backwards over the tape: reverseStep (the RK step and its transport
//    scalars) and reverseEvent (update, F <- J F, Jacobian from the leg).
// A track whose tape runs over its capacity is left to adjointKernel.
//
// Bound by the FP64 pipe, as the fit.  Against adjointKernel (whose forward
// stores and differentiates J C J^T per plane and whose step records carry the
// transport Jacobian as 25 words) a plane costs a third of the FP64
// instructions and a quarter of the tape: 65536 tracks of 20 planes, call and
// results on the host, 16.1 -> 6.3 ms.

#include <cuda_runtime.h>

#include "kf_adjoint.cuh"
#include "kf_fit.cuh"
#include "kf_host.h"

namespace kfd {
namespace adj {

// a state's record: word e in P.ws (e < 37) or A.stateBar
enum {
  zH = 0,     // F rows 0, 1 (10)
  zD = 10,    // the update's dl, later the sum G (5)
  zX = 15,    // predicted loc0, loc1
  zF2 = 17,   // F rows 2, 3 (10)
  zC = 27,    // C0 before the update (15)
  zPos = 42,  // predicted position, direction, q/p
  zDir = 45,
  zQop = 48,
  zLeg = 49,  // leg scalars g, b, r, q1, s, c0, c1, a0, a1
  zK4 = 58,   // last step: y, dx, dy
  zTr = 61,   // trigonometry of the predicted direction
  zTn = 65,   // ... and of the filtered one
  zStep = 69, // a step since the last surface
  zRho = 70,  // 2 V^-1 rho (written by chi2States)
  zWords = 72
};
// a hit's tape record: J (20), W = C0 [h0 h1] (10), the gain's l, i0, i1, e0, e1
enum { tJ = 0, tW = 20, tGain = 30, tWords = 35 };
static_assert(zWords <= 2 * kStateStride, "state record");

struct ZHook {
  static constexpr bool kTape = true;
  static constexpr int kGroup = 1;
  double *tape;       // this lane's word 0; word k at tape[k * n]
  double *recA, *recB;
  int32_t *info;
  int64_t n;
  int top, head, state, plane, cap;
  bool rec, full, over; // recording; a step failed; the tape ran over its capacity

  __device__ __forceinline__ void put(double v) {
    if (top < cap) __stcs(tape + (int64_t)top * n, v); // written once, read once
    else over = true;
    ++top;
  }
  __device__ __forceinline__ void word(int e, double v) const {
    double *p = e < kStateStride ? recA + ((int64_t)state * kStateStride + e) * n
                                 : recB + ((int64_t)state * kStateStride + e - kStateStride) * n;
    __stcs(p, v);
  }
  template <class LT> __device__ __forceinline__ void stepBegin(const LT &L) {
    if (!rec) return;
    head = top;
    for (int i = 0; i < 3; ++i) put(L.pos[i]);
    for (int i = 0; i < 3; ++i) put(L.dir[i]);
    put(L.g.g);
    put(L.g.b);
    put(L.g.c[0]);
    put(L.g.c[1]);
  }
  // the constraint that sets h: the first minimum of the step constraints
  // (ssMin order, forward direction)
  template <class LT> __device__ __forceinline__ void trial(const LT &L, double h) {
    if (!rec) return;
    int idx = 0;
    long long km = okey(L.ss[0]);
    for (int i = 1; i < 4; ++i) {
      const long long k = okey(L.ss[i]);
      if (k < km) {
        km = k;
        idx = i;
      }
    }
    put(h);
    put((double)idx);
  }
  template <class LT> __device__ __forceinline__ void stepEnd(const LT &, bool ok) {
    if (!rec) return;
    if (!ok) full = true; // a failed step has no derivative: the track is dropped
    put(hdr(REC_STEP, top + 1 - head));
  }
  // set from the state that the next RK step starts from: the plane suffices
  template <class LT> __device__ __forceinline__ void actorSet(const LT &, int k) {
    if (!rec) return;
    put((double)k);
    put(hdr(REC_ACT, 2));
  }
  template <class LT>
  __device__ __forceinline__ void event(const LT &L, int k, const Trig &tr, const double (&J)[4][5],
                                        double x0, double x1) {
    state = L.measStates;
    plane = k;
#pragma unroll
    for (int c = 0; c < 5; ++c) {
      word(zH + c, L.F(0, c));
      word(zH + 5 + c, L.F(1, c));
    }
    word(zX, x0);
    word(zX + 1, x1);
    if (!rec) return;
#pragma unroll
    for (int c = 0; c < 5; ++c) {
      word(zF2 + c, L.F(2, c));
      word(zF2 + 5 + c, L.F(3, c));
    }
#pragma unroll
    for (int e = 0; e < 15; ++e) word(zC + e, L.C0(e));
#pragma unroll
    for (int e = 0; e < 3; ++e) {
      word(zPos + e, L.pos[e]);
      word(zDir + e, L.dir[e]);
    }
    word(zQop, L.qop);
    word(zLeg + 0, L.g.g);
    word(zLeg + 1, L.g.b);
    word(zLeg + 2, L.g.r);
    word(zLeg + 3, L.g.q1);
    word(zLeg + 4, L.g.s);
    word(zLeg + 5, L.g.c[0]);
    word(zLeg + 6, L.g.c[1]);
    word(zLeg + 7, L.g.a[0]);
    word(zLeg + 8, L.g.a[1]);
    word(zK4 + 0, L.g.y);
    word(zK4 + 1, L.g.dx);
    word(zK4 + 2, L.g.dy);
    word(zTr + 0, tr.cP);
    word(zTr + 1, tr.sP);
    word(zTr + 2, tr.cT);
    word(zTr + 3, tr.sT);
    word(zStep, L.stepped ? 1. : 0.);
    head = top;
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int c = 0; c < 5; ++c) put(J[r][c]);
  }
  __device__ __forceinline__ void update(const double (&w0)[5], const double (&w1)[5], const Gain &g) {
#pragma unroll
    for (int c = 0; c < 5; ++c) word(zD + c, fma(w0[c], g.e0, w1[c] * g.e1));
    if (!rec) return;
#pragma unroll
    for (int c = 0; c < 5; ++c) put(w0[c]);
#pragma unroll
    for (int c = 0; c < 5; ++c) put(w1[c]);
    put(g.l);
    put(g.i0);
    put(g.i1);
    put(g.e0);
    put(g.e1);
  }
  __device__ __forceinline__ void eventEnd(bool outlier, const Trig &tn) {
    info[(int64_t)state * n] = plane | (outlier ? 256 : 0);
    if (!rec) return;
    word(zTn + 0, tn.cP);
    word(zTn + 1, tn.sP);
    word(zTn + 2, tn.cT);
    word(zTn + 3, tn.sT);
    put(hdr(REC_HIT, top + 1 - head));
  }
};

using ZLane = FitLane<kUniform64, false, ZHook>;

// ---- the running adjoint ----------------------------------------------------
// In the lane's shared-memory column, once the forward pass is done: F(r, c)
// and C0(e) hold the adjoints of F and of C0 (B: the symmetric matrix, off-
// diagonal entries halved), D(c) the sum E of the updates passed so far.
struct ZAdj {
  double pos[3], dir[3], qop, Bz;
  double g, b, r, q1, s, c0, c1, a0, a1; // leg scalars
  double k40, k41;                       // k4 of the leg's last step
  double ssAcc, ssAct;                   // accuracy and navigation constraints
  double ph, th;                         // angles of the jacToGlobal in use
  double U[3], V[3];                     // axes of its plane
  kfa::FrameBar fb;                      // frame of plane `plane`, not yet added
  int plane;
};

__device__ __forceinline__ void toFrameZ(const PlaneD &pl, kfa::Frame &f) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    f.c[i] = pl.c[i];
    f.U[i] = pl.U[i];
    f.V[i] = pl.V[i];
    f.T[i] = pl.T[i];
  }
}
__device__ __forceinline__ void flushPlane(ZAdj &R, const PlaneD *sp, const AdjParams &A, int64_t n,
                                           int64_t i) {
  if (R.plane >= 0) {
    kfa::Frame f;
    toFrameZ(sp[R.plane], f);
    double g[6];
    kfa::alignmentGrad(f, R.fb, g);
#pragma unroll
    for (int a = 0; a < 6; ++a) A.alignPart[((int64_t)R.plane * 6 + a) * n + i] += g[a];
  }
  kfa::frameBarZero(R.fb);
}
__device__ __forceinline__ void usePlane(ZAdj &R, int k, const PlaneD *sp, const AdjParams &A,
                                         int64_t n, int64_t i) {
  if (R.plane == k) return;
  flushPlane(R, sp, A, n, i);
  R.plane = k;
}

// reverse of one RK step (stepUniform) of a leg with q/p qop; dn: the direction
// it ended with
__device__ void reverseStepZ(TapeRef w, int len, ZAdj &R, const Params &P, double qop,
                             const double dn[3]) {
  const double dx = w[3], dy = w[4], dz = w[5], G = w[6], Bc = w[7], c0 = w[8], c1 = w[9];
  const int T = (len - 11) / 2;
  const double h = w[10 + 2 * (T - 1)];
  const double k = qop * P.Bz, y = h * k, x = y * y, hy = h * y;
  const double m = fma(x, -1. / 24., 0.5), n = fma(x, -1. / 6., 1.);
  const double al = y * n, be1 = fma(-x, m, 1.);
  const double mu = hy * m, nu = h * x * (1. / 6.), hn = h - nu;
  const double hb = h * P.Bz, hhb = h * hb;
  const double t1 = fma(x, -0.5, 1.), t2 = fma(x, -0.125, 0.5);
  const double al1 = hb * t1, be2 = hb * al, mu1 = hhb * t2, nu1 = hhb * y * (1. / 3.);
  // dir' = w / |w| (|w| = 1 where stepUniform does not normalise)
  const double rad = R.dir[0] * dn[0] + R.dir[1] * dn[1] + R.dir[2] * dn[2];
  double wx = fma(-rad, dn[0], R.dir[0]), wy = fma(-rad, dn[1], R.dir[1]),
         wz = fma(-rad, dn[2], R.dir[2]);
  if (!(akey(x) < 0x3ee4f8b588e368f1LL)) {
    const double e0 = fma(be1, dx, al * dy), e1 = fma(be1, dy, -al * dx);
    const double in = rsqrtFast(e0 * e0 + e1 * e1 + dz * dz);
    wx *= in;
    wy *= in;
    wz *= in;
  }
  const double px = R.pos[0], py = R.pos[1], pz = R.pos[2];
  const double a0 = R.a0, a1 = R.a1, q0 = R.c0, q1 = R.c1;
  // coefficients
  const double hnb = a0 * c0 + a1 * c1 + R.r * G + R.q1 * Bc + px * dx + py * dy;
  const double mub = a0 * c1 - a1 * c0 - R.r * Bc + R.q1 * G + px * dy - py * dx;
  const double mu1b = a0 * dy - a1 * dx, nu1b = -(a0 * dx) - a1 * dy;
  const double be1b = q0 * c0 + q1 * c1 + R.g * G + R.b * Bc + wx * dx + wy * dy;
  double alb = q0 * c1 - q1 * c0 - R.g * Bc + R.b * G + wx * dy - wy * dx;
  const double al1b = q0 * dy - q1 * dx, be2b = -(q0 * dx) - q1 * dy;
  double h_ = R.s + pz * dz;
  // the step's start
  double dxb = hn * px - mu * py + be1 * wx - al * wy - nu1 * a0 - mu1 * a1 - be2 * q0 - al1 * q1;
  double dyb = mu * px + hn * py + al * wx + be1 * wy + mu1 * a0 - nu1 * a1 + al1 * q0 - be2 * q1;
  const double dzb = fma(h, pz, wz);
  R.c0 = hn * a0 - mu * a1 + be1 * q0 - al * q1;
  R.c1 = mu * a0 + hn * a1 + al * q0 + be1 * q1;
  const double gb = hn * R.r + mu * R.q1 + be1 * R.g + al * R.b;
  R.b = hn * R.q1 - mu * R.r + be1 * R.b - al * R.g;
  R.g = gb;
  // scalars
  double xb = 0., yb = 0., kb = 0.;
  if (R.k40 != 0. || R.k41 != 0.) { // k4 of the leg's last step (lastK4)
    const double w1 = t1, u = fma(x, -0.25, 1.), w2 = y * u;
    const double e0 = R.k40 * dy - R.k41 * dx, e1 = -(R.k40 * dx) - R.k41 * dy;
    kb = w1 * e0 + w2 * e1;
    const double w1b = k * e0, w2b = k * e1;
    dxb -= k * (w2 * R.k40 + w1 * R.k41);
    dyb += k * (w1 * R.k40 - w2 * R.k41);
    xb = -0.5 * w1b - 0.25 * y * w2b;
    yb = u * w2b;
    R.k40 = R.k41 = 0.;
  }
  alb += hb * be2b;
  double hbb = al * be2b + t1 * al1b;
  const double hhbb = t2 * mu1b + y * (1. / 3.) * nu1b;
  const double nub = -hnb;
  const double mb = hy * mub - x * be1b;
  xb -= 0.5 * hb * al1b + 0.125 * hhb * mu1b;
  xb += h * (1. / 6.) * nub - m * be1b - mb * (1. / 24.) - y * alb * (1. / 6.);
  yb += hhb * (1. / 3.) * nu1b + h * m * mub + n * alb;
  h_ += hnb + x * (1. / 6.) * nub + y * m * mub + hb * hhbb;
  hbb += h * hhbb;
  yb += 2. * y * xb;
  h_ += P.Bz * hbb + k * yb;
  kb += h * yb;
  R.Bz += h * hbb + qop * kb;
  R.qop += P.Bz * kb;
  auto route = [&](int idx, double v) { // to the constraint that set the step
    if (idx == kAccuracy) R.ssAcc += v;
    else if (idx == kActor) R.ssAct += v; // navDir = +1 on the forward leg
  };
  route((int)w[10 + 2 * (T - 1) + 1], h_);
  R.dir[0] = dxb;
  R.dir[1] = dyb;
  R.dir[2] = dzb;
  // rejected trials, last first: each set the accuracy constraint from its
  // error estimate
  for (int t = T - 2; t >= 0; --t) {
    const double gacc = R.ssAcc;
    R.ssAcc = 0.;
    if (gacc == 0.) continue;
    const double ht = w[10 + 2 * t], d[3] = {dx, dy, dz};
    const double *B = P.field.B;
    kfa::PolyStep ps;
    kfa::polyPrep(d, B, ps);
    kfa::polyCoef(qop, ht, ps);
    double dsde, Bb[3] = {0., 0., 0.};
    const double sc = kfa::accScale(ps.err, P.tol, &dsde);
    double htb = gacc * sc;
    kfa::polyErrVjp(d, qop, ht, B, ps, gacc * ht * dsde, R.dir, R.qop, htb, Bb);
    R.Bz += Bb[2];
    route((int)w[10 + 2 * t + 1], htb);
  }
}

// reverse of a hit: state s of track i (tape record J)
__device__ void reverseEvent(TapeRef Jt, int s, ZAdj &R, ZLane &L, const Params &P,
                             const PlaneD *planes, const AdjParams &A, int64_t u, int64_t i,
                             double q, double &qop, double (&dn)[3], double &locb) {
  const int64_t n = P.n;
  auto rec = [&](int st, int e) {
    return __ldcs((e < kStateStride ? P.ws + ((int64_t)st * kStateStride + e) * n
                                    : A.stateBar + ((int64_t)st * kStateStride + e - kStateStride) * n) + u);
  };
  const int inf = A.info[(int64_t)s * n + u];
  const int k = inf & 255;
  const bool outlier = (inf & 256) != 0;
  usePlane(R, k, planes, A, n, i);
  const PlaneD &pl = planes[k];
  kfa::FrameBar &fb = R.fb;
  // the next leg's use of this plane's axes and of the predicted angles
#pragma unroll
  for (int e = 0; e < 3; ++e) {
    fb.U[e] += R.U[e];
    fb.V[e] += R.V[e];
    R.U[e] = R.V[e] = 0.;
  }
  double phb = R.ph, thb = R.th;
  R.ph = R.th = 0.;
  const Trig tr = {rec(s, zTr), rec(s, zTr + 1), rec(s, zTr + 2), rec(s, zTr + 3)};
  qop = rec(s, zQop);
  double x0b = 0., x1b = 0., qopb = R.qop;
  if (!outlier) {
    const double x0 = rec(s, zX), x1 = rec(s, zX + 1);
    double h0[5], h1[5], w0[5], w1[5], C[15];
#pragma unroll
    for (int c = 0; c < 5; ++c) {
      h0[c] = rec(s, zH + c);
      h1[c] = rec(s, zH + 5 + c);
    }
#pragma unroll
    for (int e = 0; e < 15; ++e) C[e] = rec(s, zC + e);
    // chi2's own term
    const double p0 = rec(s, zRho), p1 = rec(s, zRho + 1);
    const Gain g = {Jt[tGain], Jt[tGain + 1], Jt[tGain + 2], Jt[tGain + 3], Jt[tGain + 4], 0.};
    double dl[5], D0 = 0., D1 = 0.; // h . dl: the shift of the predicted position
#pragma unroll
    for (int c = 0; c < 5; ++c) {
      w0[c] = Jt[tW + c];
      w1[c] = Jt[tW + 5 + c];
      dl[c] = fma(w0[c], g.e0, w1[c] * g.e1);
      const double E = L.D(c) += dl[c];
      L.F(0, c) = fma(-p0, E, L.F(0, c));
      L.F(1, c) = fma(-p1, E, L.F(1, c));
      D0 = fma(h0[c], dl[c], D0);
      D1 = fma(h1[c], dl[c], D1);
    }
    // the stepper's new direction and position
    double ph1, th1, X0b, X1b;
    {
      const Trig tn = {rec(s, zTn), rec(s, zTn + 1), rec(s, zTn + 2), rec(s, zTn + 3)};
      ph1 = tn.sT * (tn.cP * R.dir[1] - tn.sP * R.dir[0]);
      th1 = tn.cT * (tn.cP * R.dir[0] + tn.sP * R.dir[1]) - tn.sT * R.dir[2];
      phb += ph1;
      thb += th1;
      const double X0 = x0 + D0, X1 = x1 + D1;
      X0b = dot3(pl.U, R.pos);
      X1b = dot3(pl.V, R.pos);
#pragma unroll
      for (int e = 0; e < 3; ++e) {
        fb.c[e] += R.pos[e];
        fb.U[e] = fma(X0, R.pos[e], fb.U[e]);
        fb.V[e] = fma(X1, R.pos[e], fb.V[e]);
      }
    }
    if ((qop + dl[4]) * q < 0.) qopb = -qopb; // the stepper takes |q/p|
    double dlb[5];
#pragma unroll
    for (int c = 0; c < 5; ++c) {
      const double f2 = rec(s, zF2 + c), f3 = rec(s, zF2 + 5 + c);
      dlb[c] = rec(s, zD + c) + ph1 * f2 + th1 * f3 + X0b * h0[c] + X1b * h1[c] + (c == 4 ? qopb : 0.);
      L.F(2, c) = fma(ph1, dl[c], L.F(2, c));
      L.F(3, c) = fma(th1, dl[c], L.F(3, c));
    }
    // dl = W S^-1 r, C' = C - W S^-1 W^T, W = C [h0 h1], S = [h_i . w_j] + V
    double P0[5], P1[5], Q0[5], Q1[5];
    double s00 = 0., s01 = 0., s11 = 0., r0 = 0., r1 = 0.;
#pragma unroll
    for (int c = 0; c < 5; ++c) {
      P1[c] = fma(-g.l, w0[c], w1[c]) * g.i1;
      P0[c] = fma(w0[c], g.i0, -g.l * P1[c]);
    }
#pragma unroll
    for (int a = 0; a < 5; ++a) {
      double e = 0., f = 0.;
#pragma unroll
      for (int j = 0; j < 5; ++j) {
        const double Bj = L.C0(u5(a, j));
        e = fma(Bj, P0[j], e);
        f = fma(Bj, P1[j], f);
      }
      s00 = fma(P0[a], e, s00);
      s01 = fma(P0[a], f, s01);
      s11 = fma(P1[a], f, s11);
      r0 = fma(P0[a], dlb[a], r0);
      r1 = fma(P1[a], dlb[a], r1);
      Q0[a] = fma(-2., e, dlb[a] * g.e0);
      Q1[a] = fma(-2., f, dlb[a] * g.e1);
    }
    s00 = fma(-r0, g.e0, s00);
    s11 = fma(-r1, g.e1, s11);
    s01 = fma(-0.5, r0 * g.e1 + r1 * g.e0, s01);
#pragma unroll
    for (int c = 0; c < 5; ++c) {
      const double y0 = Q0[c] + h0[c] * s00 + h1[c] * s01, y1 = Q1[c] + h0[c] * s01 + h1[c] * s11;
      Q0[c] = y0;
      Q1[c] = y1;
    }
#pragma unroll
    for (int a = 0; a < 5; ++a) {
      double e = fma(w0[a], s00, w1[a] * s01), f = fma(w0[a], s01, w1[a] * s11);
#pragma unroll
      for (int j = 0; j < 5; ++j) {
        e = fma(C[u5(a, j)], Q0[j], e);
        f = fma(C[u5(a, j)], Q1[j], f);
      }
      L.F(0, a) += fma(X0b, dl[a], e);
      L.F(1, a) += fma(X1b, dl[a], f);
    }
#pragma unroll
    for (int a = 0; a < 5; ++a)
#pragma unroll
      for (int j = a; j < 5; ++j) {
        double v = h0[a] * Q0[j] + h1[a] * Q1[j];
        if (j == a) {
          L.C0(u5(a, a)) += v;
        } else {
          v = fma(h0[j], Q0[a], fma(h1[j], Q1[a], v));
          L.C0(u5(a, j)) = fma(0.5, v, L.C0(u5(a, j)));
        }
      }
    x0b = X0b - (p0 + r0);
    x1b = X1b - (p1 + r1);
#pragma unroll
    for (int e = 0; e < 3; ++e) R.pos[e] = R.dir[e] = 0.;
  }
  R.qop = qopb;
  // predicted local position
  double dir[3];
#pragma unroll
  for (int e = 0; e < 3; ++e) {
    const double d = rec(s, zPos + e) - pl.c[e], v = x0b * pl.U[e] + x1b * pl.V[e];
    dir[e] = dn[e] = rec(s, zDir + e);
    R.pos[e] += v;
    fb.c[e] -= v;
    fb.U[e] = fma(x0b, d, fb.U[e]);
    fb.V[e] = fma(x1b, d, fb.V[e]);
  }
  // F = J F_old + J(:, 4) e4^T
  double Jb[4][5];
  if (s == 0) {
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int c = 0; c < 5; ++c) Jb[r][c] = L.F(r, c);
  } else {
    double J[4][4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        J[r][c] = Jt[tJ + 5 * r + c];
        Jb[r][c] = 0.;
      }
      Jb[r][4] = L.F(r, 4);
    }
#pragma unroll
    for (int c = 0; c < 5; ++c) {
      double f[4], o[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) f[r] = L.F(r, c);
      o[0] = rec(s - 1, zH + c);
      o[1] = rec(s - 1, zH + 5 + c);
      o[2] = rec(s - 1, zF2 + c);
      o[3] = rec(s - 1, zF2 + 5 + c);
#pragma unroll
      for (int l = 0; l < 4; ++l) {
        double v = J[0][l] * f[0];
#pragma unroll
        for (int r = 1; r < 4; ++r) v = fma(J[r][l], f[r], v);
        L.F(l, c) = v;
#pragma unroll
        for (int r = 0; r < 4; ++r) Jb[r][l] = fma(f[r], o[l], Jb[r][l]);
      }
    }
  }
  // ---- the bound Jacobian (boundRows)
  const bool st = rec(s, zStep) != 0.;
  const double is = rcpFast(tr.sT);
  double f0[2] = {-tr.sP * is, tr.cP * is}, f1[3] = {tr.cP * tr.cT, tr.sP * tr.cT, -tr.sT};
  double sp[3] = {0., 0., 0.}, k4[2] = {0., 0.}, u0 = 0., u1 = 0., idn = 0.;
  const double K = qop * P.Bz, ky = rec(s, zK4), kdx = rec(s, zK4 + 1), kdy = rec(s, zK4 + 2);
  if (st) {
    idn = rcpFast(dot3(pl.T, dir));
    const double kx = ky * ky, e1 = K * fma(kx, -0.5, 1.), e2 = K * ky * fma(kx, -0.25, 1.);
    k4[0] = fma(e1, kdy, -e2 * kdx);
    k4[1] = fma(-e1, kdx, -e2 * kdy);
    u0 = dot3(pl.U, dir);
    u1 = dot3(pl.V, dir);
  }
  double A0[3], A1[3];
#pragma unroll
  for (int e = 0; e < 3; ++e) {
    sp[e] = pl.T[e] * idn;
    A0[e] = fma(-u0, sp[e], pl.U[e]);
    A1[e] = fma(-u1, sp[e], pl.V[e]);
  }
  const double fk0 = f0[0] * k4[0] + f0[1] * k4[1], fk1 = f1[0] * k4[0] + f1[1] * k4[1];
  double A0b[3] = {0., 0., 0.}, A1b[3] = {0., 0., 0.}, spb[3] = {0., 0., 0.}, f0b[2] = {0., 0.},
         f1b[3] = {0., 0., 0.}, fk0b = 0., fk1b = 0.;
  // one column: position part p (flat: no z), its adjoint pb
  auto column = [&](int c, const double *p, bool flat, double *pb) {
    const double sc = dotz(flat, sp, p);
    const double scb = -(fk0 * Jb[2][c]) - fk1 * Jb[3][c];
    fk0b = fma(-sc, Jb[2][c], fk0b);
    fk1b = fma(-sc, Jb[3][c], fk1b);
    const int m = flat ? 2 : 3;
#pragma unroll
    for (int e = 0; e < 3; ++e) {
      if (e >= m) break;
      pb[e] = Jb[0][c] * A0[e] + Jb[1][c] * A1[e] + scb * sp[e];
      A0b[e] = fma(Jb[0][c], p[e], A0b[e]);
      A1b[e] = fma(Jb[1][c], p[e], A1b[e]);
      spb[e] = fma(scb, p[e], spb[e]);
    }
  };
  // the last surface: its trigonometry and axes
  Trig tl;
  double o = 0.;
  if (s == 0) {
    double sp_, cp_, st_, ct_;
    sincos(P.start[2 * P.stride + i], &sp_, &cp_);
    sincos(P.start[3 * P.stride + i], &st_, &ct_);
    const double sg = st_ < 0. ? -1. : 1.;
    tl = {sg * cp_, sg * sp_, ct_, sg * st_};
    o = P.start[i];
  } else {
    tl = {rec(s - 1, zTr), rec(s - 1, zTr + 1), rec(s - 1, zTr + 2), rec(s - 1, zTr + 3)};
  }
  {
    double U[3], V[3], pb[3];
    const int kl = s == 0 ? 0 : (A.info[(int64_t)(s - 1) * n + u] & 255);
#pragma unroll
    for (int e = 0; e < 3; ++e) {
      U[e] = s == 0 ? (e == 0 ? -tl.sP : (e == 1 ? tl.cP : 0.)) : planes[kl].U[e];
      V[e] = s == 0 ? (e == 2 ? 1. : 0.) : planes[kl].V[e];
    }
    column(0, U, false, pb);
    if (s == 0) {
      R.ph -= pb[0] * tl.cP + pb[1] * tl.sP;
    } else {
#pragma unroll
      for (int e = 0; e < 3; ++e) R.U[e] = pb[e];
    }
    column(1, V, false, pb);
    if (s != 0) {
#pragma unroll
      for (int e = 0; e < 3; ++e) R.V[e] = pb[e];
    }
  }
  const double lg = rec(s, zLeg), lb = rec(s, zLeg + 1), lr = rec(s, zLeg + 2), lq = rec(s, zLeg + 3),
               ls = rec(s, zLeg + 4);
  R.g = R.b = R.r = R.q1 = R.s = 0.;
  // direction columns phi (c = 2: flat) and theta (c = 3): e -> (p, v)
  auto dircol = [&](int c, const double (&e)[3], double (&eb)[3]) {
    const bool flat = c == 2;
    double p[3] = {fma(lr, e[0], lq * e[1]), fma(lr, e[1], -lq * e[0]), 0.}, pb[3] = {0., 0., 0.};
    const double v[2] = {fma(lg, e[0], lb * e[1]), fma(lg, e[1], -lb * e[0])};
    if (!flat) p[2] = ls * e[2];
    double off[2] = {0., 0.};
    if (flat && s == 0) { // (the point at distance loc0 from the line)
      off[0] = -tl.cP;
      off[1] = -tl.sP;
      p[0] = fma(o, off[0], p[0]);
      p[1] = fma(o, off[1], p[1]);
    }
    column(c, p, flat, pb);
    if (flat && s == 0) {
      locb += pb[0] * off[0] + pb[1] * off[1];
      R.ph += o * (pb[0] * tl.sP - pb[1] * tl.cP);
    }
    const double v0b = Jb[2][c] * f0[0] + Jb[3][c] * f1[0], v1b = Jb[2][c] * f0[1] + Jb[3][c] * f1[1];
    f0b[0] = fma(Jb[2][c], v[0], f0b[0]);
    f0b[1] = fma(Jb[2][c], v[1], f0b[1]);
    f1b[0] = fma(Jb[3][c], v[0], f1b[0]);
    f1b[1] = fma(Jb[3][c], v[1], f1b[1]);
    R.r += pb[0] * e[0] + pb[1] * e[1];
    R.q1 += pb[0] * e[1] - pb[1] * e[0];
    R.g += v0b * e[0] + v1b * e[1];
    R.b += v0b * e[1] - v1b * e[0];
    eb[0] = lr * pb[0] - lq * pb[1] + lg * v0b - lb * v1b;
    eb[1] = lq * pb[0] + lr * pb[1] + lb * v0b + lg * v1b;
    eb[2] = 0.;
    if (!flat) {
      f1b[2] = fma(Jb[3][c], e[2], f1b[2]);
      R.s += pb[2] * e[2];
      eb[2] = fma(ls, pb[2], Jb[3][c] * f1[2]);
    }
  };
  {
    double eb[3];
    const double e2[3] = {-tl.sT * tl.sP, tl.sT * tl.cP, 0.}, e3[3] = {tl.cT * tl.cP, tl.cT * tl.sP, -tl.sT};
    dircol(2, e2, eb);
    R.ph -= eb[0] * e2[1] - eb[1] * e2[0];
    R.th += tl.cT * (eb[1] * tl.cP - eb[0] * tl.sP);
    dircol(3, e3, eb);
    R.ph += eb[1] * e3[0] - eb[0] * e3[1];
    R.th -= tl.sT * (eb[0] * tl.cP + eb[1] * tl.sP) + eb[2] * tl.cT;
  }
  {
    const double p[3] = {rec(s, zLeg + 7), rec(s, zLeg + 8), 0.};
    const double v[2] = {rec(s, zLeg + 5), rec(s, zLeg + 6)};
    double pb[3];
    column(4, p, true, pb);
    R.a0 = pb[0];
    R.a1 = pb[1];
    R.c0 = Jb[2][4] * f0[0] + Jb[3][4] * f1[0];
    R.c1 = Jb[2][4] * f0[1] + Jb[3][4] * f1[1];
    f0b[0] = fma(Jb[2][4], v[0], f0b[0]);
    f0b[1] = fma(Jb[2][4], v[1], f0b[1]);
    f1b[0] = fma(Jb[3][4], v[0], f1b[0]);
    f1b[1] = fma(Jb[3][4], v[1], f1b[1]);
  }
  // ---- rows
  R.k40 = R.k41 = 0.;
  if (st) {
    const double u0b = -dot3(A0b, sp), u1b = -dot3(A1b, sp);
    double idb = 0.;
#pragma unroll
    for (int e = 0; e < 3; ++e) {
      spb[e] -= u0 * A0b[e] + u1 * A1b[e];
      fb.U[e] = fma(u0b, dir[e], fb.U[e]);
      fb.V[e] = fma(u1b, dir[e], fb.V[e]);
      R.dir[e] += u0b * pl.U[e] + u1b * pl.V[e];
      idb = fma(spb[e], pl.T[e], idb);
    }
    const double t = -(idn * idn) * idb;
#pragma unroll
    for (int e = 0; e < 3; ++e) {
      fb.T[e] += spb[e] * idn + t * dir[e];
      R.dir[e] = fma(t, pl.T[e], R.dir[e]);
    }
    R.k40 = fk0b * f0[0] + fk1b * f1[0];
    R.k41 = fk0b * f0[1] + fk1b * f1[1];
    f0b[0] = fma(fk0b, k4[0], f0b[0]);
    f0b[1] = fma(fk0b, k4[1], f0b[1]);
    f1b[0] = fma(fk1b, k4[0], f1b[0]);
    f1b[1] = fma(fk1b, k4[1], f1b[1]);
  }
#pragma unroll
  for (int e = 0; e < 3; ++e) {
    fb.U[e] += A0b[e];
    fb.V[e] += A1b[e];
  }
  // angles of the predicted direction
  phb += -is * (f0b[0] * tr.cP + f0b[1] * tr.sP) + tr.cT * (f1b[1] * tr.cP - f1b[0] * tr.sP);
  thb += -(tr.cT * is) * (f0b[0] * f0[0] + f0b[1] * f0[1]) -
         tr.sT * (f1b[0] * tr.cP + f1b[1] * tr.sP) - tr.cT * f1b[2];
  R.dir[0] += phb * f0[0] + thb * f1[0];
  R.dir[1] += phb * f0[1] + thb * f1[1];
  R.dir[2] += thb * f1[2];
}

// chi2 of a track with ns states, backwards with the sum E of the updates; with
// grad each state's 2 V^-1 rho into its record, and then, forwards, the sum G
// of dchi2/dE in place of its update (sums of their own: differences of running
// sums cancel)
__device__ double chi2States(const Params &P, const AdjParams &A, int64_t u, int64_t i, int ns) {
  const int64_t n = P.n;
  double chi2 = 0., E[5] = {0., 0., 0., 0., 0.};
  for (int s = ns - 1; s >= 0; --s) {
    const int inf = A.info[(int64_t)s * n + u];
    if (inf & 256) continue;
    const double *rc = P.ws + (int64_t)s * kStateStride * n + u;
    const double *mp = P.meas + (size_t)(inf & 255) * 5 * P.stride + i;
    const double v00 = mp[2 * P.stride], v01 = mp[3 * P.stride], v11 = mp[4 * P.stride];
    double f0 = mp[0] - rc[zX * n], f1 = mp[P.stride] - rc[(zX + 1) * n];
#pragma unroll
    for (int c = 0; c < 5; ++c) {
      E[c] += rc[(zD + c) * n];
      f0 = fma(-rc[(zH + c) * n], E[c], f0);
      f1 = fma(-rc[(zH + 5 + c) * n], E[c], f1);
    }
    const double id = 1. / (v00 * v11 - v01 * v01); // (0 where large variances' product overflows)
    const double w0 = (v11 * f0 - v01 * f1) * id, w1 = (v00 * f1 - v01 * f0) * id;
    chi2 += f0 * w0 + f1 * w1;
    if (A.grad) {
      double *rb = A.stateBar + ((int64_t)s * kStateStride + zRho - kStateStride) * n + u;
      rb[0] = 2. * w0;
      rb[n] = 2. * w1;
    }
  }
  if (!A.grad) return chi2;
  double G[5] = {0., 0., 0., 0., 0.};
  for (int s = 0; s < ns; ++s) {
    if (A.info[(int64_t)s * n + u] & 256) continue;
    double *rc = P.ws + (int64_t)s * kStateStride * n + u;
    const double *rb = A.stateBar + ((int64_t)s * kStateStride + zRho - kStateStride) * n + u;
    const double p0 = rb[0], p1 = rb[n];
#pragma unroll
    for (int c = 0; c < 5; ++c) {
      G[c] -= p0 * rc[(zH + c) * n] + p1 * rc[(zH + 5 + c) * n];
      rc[(zD + c) * n] = G[c];
    }
  }
  return chi2;
}

__device__ void zeroTrackZ(const Params &P, const AdjParams &A, int64_t i) {
  A.chi2[i] = 0.;
  A.trackFs[i] = 0.;
  for (int64_t k = 0; k < (int64_t)P.nSurf * 6; ++k) A.alignPart[k * P.n + i] = 0.;
  if (A.gradStart)
    for (int e = 0; e < 6; ++e) A.gradStart[(int64_t)e * P.stride + i] = 0.;
}

constexpr int kZBlock = 32; // one-warp blocks spread over the SMs most evenly

__global__ void __launch_bounds__(kZBlock, 8) adjointZ(const __grid_constant__ Params P,
                                                       const __grid_constant__ AdjParams A) {
  PlaneD *sp = reinterpret_cast<PlaneD *>(kfColdSmem + (size_t)blockDim.x * coldSlots<false>() * sizeof(double));
  for (int k = threadIdx.x; k < P.nSurf; k += blockDim.x) sp[k] = P.planes[k];
  __syncthreads();
  // every lane stays to the end: the lane program and the reverse sweep run
  // warp-synchronously (idle lanes carry no work)
  const int64_t u = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; // queue position
  const bool valid = u < P.n;
  const int64_t i = valid ? (int64_t)A.perm[u] : 0; // track
  ZLane L;
  L.hook.tape = A.tape + (valid ? u : 0);
  L.hook.recA = P.ws + (valid ? u : 0);
  L.hook.recB = A.stateBar + (valid ? u : 0);
  L.hook.info = A.info + (valid ? u : 0);
  L.hook.n = P.n;
  L.hook.top = L.hook.head = L.hook.state = L.hook.plane = 0;
  L.hook.cap = A.tapeCap;
  L.hook.rec = valid && A.grad != 0;
  L.hook.full = L.hook.over = false;
  if (valid) zeroTrackZ(P, A, i);
  // ---- A: forward (recording from before initFit, which already sets the
  // step constraint towards the first plane)
  initFit(L, P, sp, valid ? i : -1, valid ? u : 0);
  for (;;) {
    if (!L.parked && L.pc != PC_DONE) advance(L, P, sp);
    const bool waiting = L.parked || L.pc == PC_DONE;
    if (__all_sync(0xffffffffu, waiting)) {
      if (eventDue(L)) runEvent(L, P, sp);
      if (__all_sync(0xffffffffu, L.pc == PC_DONE)) break;
    }
  }
  const int ns = L.measStates;
  bool ok = valid && L.status == KF_TRACK_OK && ns > 0;
  const bool left = ok && A.grad && L.hook.over && !L.hook.full;
  if (valid) A.status[i] = left ? kLeft : (ok && L.hook.full ? KF_TRACK_ADJOINT_FAILED : L.status);
  ok = ok && !left && !L.hook.full;
  // ---- B
  if (ok) A.chi2[i] = chi2States(P, A, u, i, ns);
  if (!A.grad) return;
  // ---- C
  ZAdj R;
  for (int e = 0; e < 3; ++e) R.pos[e] = R.dir[e] = R.U[e] = R.V[e] = 0.;
  R.qop = R.Bz = R.g = R.b = R.r = R.q1 = R.s = R.c0 = R.c1 = R.a0 = R.a1 = R.k40 = R.k41 = 0.;
  R.ssAcc = R.ssAct = R.ph = R.th = 0.;
  R.plane = -1;
  kfa::frameBarZero(R.fb);
  for (int r = 0; r < 4; ++r)
    for (int c = 0; c < 5; ++c) L.F(r, c) = 0.;
  for (int e = 0; e < 15; ++e) L.C0(e) = 0.;
  for (int c = 0; c < 5; ++c) L.D(c) = 0.;
  const TapeRef tape = {L.hook.tape, P.n};
  int top = ok ? L.hook.top : 0, state = ns;
  const double q = L.q;
  double qop = 0., cpos[3] = {0., 0., 0.}, cdir[3] = {0., 0., 0.}, locb = 0.;
  bool bad = false;
  // steps and constraints whenever a lane has one on top, hits once every lane
  // with work has one on top
  for (;;) {
    int type = 0, len = 0;
    if (top > 0 && !bad) {
      const int h = (int)tape[top - 1];
      type = h >> 16;
      len = h & 0xffff;
      if (len < 2 || len > top || type < REC_STEP || type > REC_HIT) {
        bad = true;
        type = 0;
      }
    }
    if (__any_sync(0xffffffffu, type == REC_STEP || type == REC_ACT)) {
      if (type == REC_STEP) {
        const TapeRef w = tape + (top - len);
        reverseStepZ(w, len, R, P, qop, cdir);
        for (int e = 0; e < 3; ++e) {
          cpos[e] = w[e];
          cdir[e] = w[3 + e];
        }
        top -= len;
      } else if (type == REC_ACT) {
        if (R.ssAct != 0.) {
          const int k = (int)tape[top - len];
          usePlane(R, k, sp, A, P.n, i);
          kfa::pathVjp(cpos, cdir, sp[k].c, sp[k].T, R.ssAct, R.pos, R.dir, R.fb.c, R.fb.T);
          R.ssAct = 0.;
        }
        top -= len;
      }
    } else {
      if (!__any_sync(0xffffffffu, type == REC_HIT)) break;
      if (type == REC_HIT) {
        --state;
        reverseEvent(tape + (top - len), state, R, L, P, sp, A, u, i, q, qop, cdir, locb);
        top -= len;
      }
    }
  }
  if (!ok) return;
  if (bad) {
    A.status[i] = KF_TRACK_ADJOINT_FAILED;
    zeroTrackZ(P, A, i);
    return;
  }
  flushPlane(R, sp, A, P.n, i);
  // ---- start parameters
  if (A.gradStart) {
    double sph, cph, sth, cth;
    const double l0 = P.start[i];
    sincos(P.start[2 * P.stride + i], &sph, &cph);
    sincos(P.start[3 * P.stride + i], &sth, &cth);
    const double sg = sth < 0. ? -1. : 1.;
    const Trig t = {sg * cph, sg * sph, cth, sg * sth};
    const double out[6] = {
        locb + t.cP * R.pos[1] - t.sP * R.pos[0], R.pos[2],
        R.ph - l0 * (R.pos[0] * t.cP + R.pos[1] * t.sP) + t.sT * (t.cP * R.dir[1] - t.sP * R.dir[0]),
        sg * (R.th + t.cT * (t.cP * R.dir[0] + t.sP * R.dir[1]) - t.sT * R.dir[2]), R.qop, 0.};
    for (int e = 0; e < 6; ++e) A.gradStart[(int64_t)e * P.stride + i] = out[e];
  }
  A.trackFs[i] = R.Bz * A.B0[2];
}

cudaError_t launchAdjointZ(const Params &P_, const AdjParams &A, cudaStream_t s) {
  Params P = P_;
  P.Bz = P.field.B[2];
  P.rotated = 0;
  P.lanes = 32;
  const size_t smem = fitSmemBytes<false>(kZBlock, P.nSurf);
  const unsigned grid = (unsigned)((P.n + kZBlock - 1) / kZBlock);
  adjointZ<<<grid, kZBlock, smem, s>>>(P, A);
  return cudaGetLastError();
}

} // namespace adj
} // namespace kfd
