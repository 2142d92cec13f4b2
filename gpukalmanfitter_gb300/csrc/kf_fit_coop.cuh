// kf_fit_coop.cuh — a track on eight lanes of a warp, for batches too small to
// fill the chip.
//
// One FP64 instruction of a warp takes its SM sub-partition 64 cycles whatever
// the lanes it has active (measured), so a small batch's time is the number of
// FP64 instructions of one warp, and lanes are free.  The eight lanes of a
// group run the same track, each with the whole state; what a hit does per
// column of the five bound parameters is shared out: lane c forms column c of
// the bound Jacobian and of F <- J F, entry c of C h and row c of the
// covariance update; the three sums of h C h^T, and the two angles' updates,
// go to one lane each.  In a field map lane c transports column c through the
// RK stages; in a uniform field the track, the leg's scalars and its q/p
// column, which a step turns alike, are a lane's each.  About 200 instead of
// 430 FP64 instructions a hit, in a field map 340 instead of 450 a step, in a
// uniform field 55 instead of 70 (the last two and the sums: 5 tracks of 10
// planes 205 -> 189 us, 1000 tracks 339 -> 310 us).  Every sum keeps its
// order, so that the results have the bits of the one-lane form (kf_fit.cuh),
// which serves larger batches: four tracks a warp are the better use of a warp
// only while warps are short (launchFit).
//
// The lanes of a group take every branch together; shared-memory exchange is
// separated by __syncwarp of the group.
#pragma once

#include "kf_fit.cuh"

namespace kfd {

template <int FORM> using CoopLane = FitLane<FORM, false, CoopHook>;

constexpr int kCoopScratch = 10; // shared-memory words 10 ... 13 of a lane's column: exchange

// column c of the bound Jacobian, and of its time row (boundJacobian)
template <int FORM>
__device__ __forceinline__ void boundColumn(const CoopLane<FORM> &L, const Params &P,
                                            const PlaneD *planes, const PlaneD &pl, int c, bool time,
                                            Trig &tr, double (&J)[4], double &J5) {
  using LT = CoopLane<FORM>;
  if constexpr (isMixed(FORM)) {
    double A[4][5], A5[5] = {0., 0., 0., 0., 0.};
    boundJacobian(L, P, planes, pl, time, tr, A, A5);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      J[r] = A[r][0];
#pragma unroll
      for (int l = 1; l < 5; ++l) J[r] = c == l ? A[r][l] : J[r];
    }
    J5 = A5[0];
#pragma unroll
    for (int l = 1; l < 5; ++l) J5 = c == l ? A5[l] : J5;
  } else {
    double invS;
    tr = trigOf(L.dir, invS);
    const Trig tl = trigLoad(L);
    const bool first = L.measStates == 0;
    const double o = first ? P.start[L.idx] : 0.;
    double sp[3] = {0., 0., 0.}, f0[3], f1[3], k4[3] = {0., 0., 0.}, u0 = 0., u1 = 0.;
    angleRows<LT>(P, tr, invS, f0, f1);
    if (L.stepped) {
      lastK4(L, P, k4);
      u0 = dot3(pl.U, L.dir);
      u1 = dot3(pl.V, L.dir);
#pragma unroll
      for (int i = 0; i < 3; ++i) sp[i] = pl.T[i] * L.idn;
    }
    const double fk0 = dotz(true, f0, k4), fk1 = dotz(FORM == kUniform64, f1, k4);
    double A0[3], A1[3], U[3], V[3], p[3], v[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      A0[i] = fma(-u0, sp[i], pl.U[i]);
      A1[i] = fma(-u1, sp[i], pl.V[i]);
    }
    lastAxes(L, P, planes, tl, U, V);
    // this lane's column: position and direction parts
    if constexpr (FORM == kUniform64) {
      const auto &g = L.g;
      const bool th = c == 3;
      const double e0 = th ? tl.cT * tl.cP : -tl.sT * tl.sP, e1 = th ? tl.cT * tl.sP : tl.sT * tl.cP,
                   e2 = th ? -tl.sT : 0.;
      p[0] = fma(g.p[0], e0, -g.p[1] * e1);
      p[1] = fma(g.p[0], e1, g.p[1] * e0);
      p[2] = g.s * e2;
      v[0] = fma(g.v[0], e0, -g.v[1] * e1);
      v[1] = fma(g.v[0], e1, g.v[1] * e0);
      v[2] = e2;
      if (c == 4) {
        p[0] = g.p[0];
        p[1] = g.p[1];
        v[0] = g.v[0];
        v[1] = g.v[1];
        p[2] = v[2] = 0.;
      }
      if (first && c == 2) {
        p[0] += -o * tl.cP;
        p[1] += -o * tl.sP;
      }
    } else {
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        p[i] = L.g.p[i];
        v[i] = L.g.v[i];
      }
      if (first && c == 2) {
        p[0] -= o * tl.cP;
        p[1] -= o * tl.sP;
      }
    }
    if (c < 2) {
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        p[i] = c ? V[i] : U[i];
        v[i] = 0.;
      }
    }
    const double s = dot3(sp, p);
    J[0] = dot3(A0, p);
    J[1] = dot3(A1, p);
    J[2] = fma(-fk0, s, dotz(true, f0, v));
    J[3] = fma(-fk1, s, dot3(f1, v));
    if (time) {
      const double dt = L.stepped ? L.dtds : 0.;
      J5 = (c == 4) ? fma(-dt, s, legPath(L) * L.d37) : -dt * s;
    }
  }
}

// Actor::filter at a plane with a hit (filterHit of kf_fit.cuh, no process
// noise, no smoothed states returned)
template <int FORM>
__device__ __forceinline__ void filterHit(CoopLane<FORM> &L, const Params &P, const PlaneD *planes,
                                          int k) {
  const unsigned group = 0xffu << (threadIdx.x & 24);
  const int c = min((int)(threadIdx.x & 7), 4);
  const bool own = (threadIdx.x & 7) < 5; // lanes 5 ... 7 follow lane 4, storing nothing
  const PlaneD &pl = planes[k];
  const bool first = L.measStates == 0;
  double J[4], J5 = 0.;
  Trig tr;
  boundColumn(L, P, planes, pl, c, first, tr, J, J5);
  if (!first) {
    unsigned m = 0;
#pragma unroll
    for (int r = 0; r < 4; ++r) m = max(m, (unsigned)__double2hiint(J[r]) & 0x7fffffffu);
    if (__any_sync(group, m >= 0x7ff00000u)) L.badJ = true;
  }
  if (first) L.t = fma(legPath(L), L.dtds, L.t);
  const double d0 = L.pos[0] - pl.c[0], d1 = L.pos[1] - pl.c[1], d2 = L.pos[2] - pl.c[2];
  const double x0 = pl.U[0] * d0 + pl.U[1] * d1 + pl.U[2] * d2;
  const double x1 = pl.V[0] * d0 + pl.V[1] * d1 + pl.V[2] * d2;
  const double *mp = P.meas + (size_t)k * 5 * P.stride + L.idx;
  const double m0 = mp[0], m1 = mp[P.stride], v00 = mp[2 * P.stride], v01 = mp[3 * P.stride],
               v11 = mp[4 * P.stride];
  if (first) L.firstPlane = k;
  // F <- J F, this lane's column
  double n[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    n[r] = J[r];
    L.cold(kCoopScratch + r) = J[r];
  }
  __syncwarp(group);
  if (!first) {
    const double f0 = L.F(0, c), f1 = L.F(1, c), f2 = L.F(2, c), f3 = L.F(3, c);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      // (a product plus -0 rounds as the product)
      double v = fma(L.coldOf(kCoopScratch + r, 0), f0, c == 4 ? J[r] : -0.);
      v = fma(L.coldOf(kCoopScratch + r, 1), f1, v);
      v = fma(L.coldOf(kCoopScratch + r, 2), f2, v);
      n[r] = fma(L.coldOf(kCoopScratch + r, 3), f3, v);
    }
  }
  __syncwarp(group);
  if (own) {
#pragma unroll
    for (int r = 0; r < 4; ++r) L.F(r, c) = n[r];
  }
  if (first) {
    if (own) {
#pragma unroll
      for (int r = 0; r < 4; ++r) *recPtr(P, L, 0, kRecF + 5 * r + c) = n[r];
      *recPtr(P, L, 0, kRecT + c) = J5;
    }
    if ((threadIdx.x & 7) == 0) {
      const double x[6] = {x0, x1, 0., 0., L.qop, L.t};
#pragma unroll
      for (int e = 0; e < 6; ++e) *recPtr(P, L, 0, kRecX + e) = x[e];
      *recPtr(P, L, 0, kRecTrig + 0) = tr.cP;
      *recPtr(P, L, 0, kRecTrig + 1) = tr.sP;
      *recPtr(P, L, 0, kRecTrig + 2) = tr.cT;
      *recPtr(P, L, 0, kRecTrig + 3) = tr.sT;
    }
  }
  __syncwarp(group);
  // w = C h: this lane's entry
  double h0[5], h1[5], w0[5], w1[5], wc[2], Cr[5];
#pragma unroll
  for (int l = 0; l < 5; ++l) {
    h0[l] = L.F(0, l);
    h1[l] = L.F(1, l);
    Cr[l] = l >= c ? L.coldOf(4 + l - c, c) : L.coldOf(4 + c - l, l);
  }
  {
    double a = Cr[0] * h0[0], b = Cr[0] * h1[0];
#pragma unroll
    for (int j = 1; j < 5; ++j) {
      a = fma(Cr[j], h0[j], a);
      b = fma(Cr[j], h1[j], b);
    }
    L.cold(kCoopScratch) = wc[0] = a;
    L.cold(kCoopScratch + 1) = wc[1] = b;
  }
  __syncwarp(group);
#pragma unroll
  for (int l = 0; l < 5; ++l) {
    w0[l] = L.coldOf(kCoopScratch, l);
    w1[l] = L.coldOf(kCoopScratch + 1, l);
  }
  // h0 . w0, h1 . w0, h1 . w1: lanes 0, 1, 2 (the others as lane 2)
  const int l8 = threadIdx.x & 7;
  double a00, a01, a11;
  {
    double hw = (l8 == 0 ? h0[0] : h1[0]) * (l8 < 2 ? w0[0] : w1[0]);
#pragma unroll
    for (int i = 1; i < 5; ++i)
      hw = fma(l8 == 0 ? h0[i] : h1[i], l8 < 2 ? w0[i] : w1[i], hw);
    a00 = __shfl_sync(group, hw, 0, 8);
    a01 = __shfl_sync(group, hw, 1, 8);
    a11 = __shfl_sync(group, hw, 2, 8);
  }
  const Gain g = gain(a00 + v00, a01 + v01, a11 + v11, m0 - x0, m1 - x1);
  const bool outlier = isOutlier(P, g.chi2);
  Trig tn = tr;
  if (!outlier) {
    // this lane's entries
    const double w0c = wc[0], w1c = fma(-g.l, w0c, wc[1]), dlc = fma(w0c, g.e0, wc[1] * g.e1);
    double dl[5];
#pragma unroll
    for (int i = 0; i < 5; ++i) dl[i] = __shfl_sync(group, dlc, i, 8);
    double w50 = 0., w51 = 0.;
    if (L.timeCorr) {
#pragma unroll
      for (int j = 0; j < 5; ++j) {
        w50 = fma(L.Ct(j), h0[j], w50);
        w51 = fma(L.Ct(j), h1[j], w51);
      }
    }
    // phi in the even lanes, theta in the odd ones
    const int r = 2 + (l8 & 1);
    double da = L.F(r, 0) * dl[0];
#pragma unroll
    for (int l = 1; l < 5; ++l) da = fma(L.F(r, l), dl[l], da);
    const double dphi = __shfl_sync(group, da, 0, 8), dth = __shfl_sync(group, da, 1, 8);
#pragma unroll
    for (int i = 0; i < 5; ++i) w1[i] = __shfl_sync(group, w1c, i, 8);
    const double a0 = w0c * g.i0, a1 = w1c * g.i1;
    if (own) {
      L.D(c) += dlc;
#pragma unroll
      for (int j = 0; j < 5; ++j)
        if (j >= c) L.coldOf(4 + j - c, c) = fma(-a0, w0[j], fma(-a1, w1[j], Cr[j]));
    }
    if (L.timeCorr) { // every lane its own copy
      L.D(5) += w50 * g.e0 + w51 * g.e1;
      const double z = fma(-g.l, w50, w51);
#pragma unroll
      for (int i = 0; i < 5; ++i)
        L.Ct(i) = fma(-(w0[i] * g.i0), w50, fma(-(w1[i] * g.i1), z, L.Ct(i)));
      L.Ct(5) = L.Ct(5) - w50 * g.i0 * w50 - z * g.i1 * z;
    }
    L.chi2 += g.chi2;
    updateState(L, P, pl, x0 + fma(a00, g.e0, a01 * g.e1), x1 + fma(a01, g.e0, a11 * g.e1), tn, dphi,
                dth, L.qop + dl[4], false);
  }
  const Trig &tg = (P.faithful || outlier) ? tr : tn;
  trigSave(L, tg);
  legReset(L, tg);
  L.lastPlane = k;
  L.measStates++;
  __syncwarp(group);
}

} // namespace kfd
