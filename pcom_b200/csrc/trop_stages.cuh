// trop_stages.cuh -- the barotropic substep's four stages (mod_int.f90:184-274)
// at one point of a tile's (TX+4) x (TY+4) region, shared by the resident
// kernel (k_trop.cu) and the multi-tile kernel (k_trop_multi.cu).
//
// The stages run straight through for every thread, whatever its point
// belongs to: values at points a stage does not cover are formed from
// whatever is there and are never read by a point it does cover.  With a
// branch per part the parts' latencies added up (a substep of 4 to 20 warps
// on an SM is bound by its dependency chains, not by issue).  The caller puts
// a CTA barrier between stages.
//
// Divisions by a metric, a bottom pressure or the Coriolis denominator go
// through dvr.  A scaling by 2 is exact, so the halves of the means, of
// sqrt(ter()) and of the pressure-gradient terms are folded into constants:
// twice dxx[1] and dxy[1] and half their reciprocals, half prh_u and
// bgraphi, twice graphih; masks are 0 or 1, so mask * x * dtbt = x * (mask * dtbt).
#pragma once
#include "pcom_dev.cuh"

// region fields in shared memory; what a later stage needs at the thread's
// own point only stays in registers
enum {
  X_CH, X_UB, X_VB,
  X_S1, X_X2,  // supb1, supb2*rh3 (reused for the corrector's supb)
  X_PRED,
  X_A1U, X_A1V, X_A2U, X_A2V,
  X_COUNT
};
// doubles before the first field and after the last (+ 32 for the last
// warp's threads past the region): reads outside the region are discarded
__host__ __device__ constexpr int x_pad(int W) { return W + 1; }

// metric vectors over lx and ly (1-D copies, folded as above)
constexpr int kXVecs = 8, kYVecs = 19;
// vector n (0-based) of column i and of row j
PD double trop_xvec(const DevCommon &P, int n, int i) {
  return n == 0 ? 2.0 * __ldg(P.dxx1d[1] + i - 1) : n == 4 ? 0.5 * __ldg(P.rdxx1d[1] + i - 1)
         : n < 4 ? __ldg(P.dxx1d[n + 1] + i - 1) : __ldg(P.rdxx1d[n - 3] + i - 1);
}
PD double trop_yvec(const DevCommon &P, int n, int j) {
  switch (n) {
  case 0: return 2.0 * __ldg(P.dxy1d[1] + j - 1);
  case 1: case 2: case 3: return __ldg(P.dxy1d[n + 1] + j - 1);
  case 4: return 0.5 * __ldg(P.rdxy1d[1] + j - 1);
  case 5: case 6: case 7: return __ldg(P.rdxy1d[n - 3] + j - 1);
  case 8: case 9: case 10: case 11: return __ldg(P.rh1d[n - 7] + j - 1);
  case 12: return __ldg(P.arh1d[1] + j - 1);
  case 13: return __ldg(P.rarh1d[1] + j - 1);
  case 14: return __ldg(P.arh1d[2] + j - 1);
  case 15: return __ldg(P.rarh1d[2] + j - 1);
  case 16: return __ldg(P.rrh1d[4] + j - 1);
  case 17: return __ldg(P.aarh3 + j - 1);
  default: return __ldg(P.raarh3 + j - 1);
  }
}

// a point's coefficients (shifted where the reference's formulas shift them)
struct TropCoef {
  double prh_uh, prh_t, rprh_t, rden;     // 0.5 prh_u; 1 / prh_t; 1 / (1 + (0.5 cor dtbt)^2)
  double sam1, cor, ut, vt;               // lev_u mask x am(1)
  double bxn, bxs, bye, byw;              // bphi
  double gxn, gxs, gye, gyw, ghx, ghy;    // 0.5 bgraphi, 2 graphih
  bool sea_u, sea_t;
};

// where a thread's point is, its fields and its metrics.  MREG: the metrics
// are kept in registers (27 pairs; tiles whose threads can have the
// registers): from shared memory they were half of a small tile's loads (int_trop
// of the 128 x 64 box 278 -> 272 us)
template <bool MREG>
struct TropPoint {
  double *f;              // &field[0][point]
  const double *vx, *vy;  // this column's and this row's metrics in shared memory
  int W, RS;              // row length of the region, size of a field
  int XS, YS, YR;         // from one column vector to the next, one row vector to the next, one row to the next
  bool inR;               // the thread has a point of the region
  bool nrow, srow;        // j <= njm, j >= 2
  bool s2sea, s6sea, s2zero;  // sqrt(ter()) of ch / of pred is formed; it is 0 (row nj)
  double xr[MREG ? kXVecs : 1], yr[MREG ? kYVecs : 1], yn[MREG ? 2 : 1];
  PD double &S(int F, int o) const { return f[F * RS + o]; }
  PD double X(int n) const { return MREG ? xr[n] : vx[n * XS]; }
  PD double Y(int n) const { return MREG ? yr[n] : vy[n * YS]; }
  // vectors 14 and 15 of the next row
  PD double Yn(int n) const { return MREG ? yn[n - 14] : vy[n * YS + YR]; }
  PD void load_metrics() {
    if constexpr (MREG) {
      #pragma unroll
      for (int n = 0; n < kXVecs; ++n) xr[n] = vx[n * XS];
      #pragma unroll
      for (int n = 0; n < kYVecs; ++n) yr[n] = vy[n * YS];
      yn[0] = vy[14 * YS + YR];
      yn[1] = vy[15 * YS + YR];
    }
  }
};

struct TropState {
  double c0, u0, v0;                  // ch, ub, vb as staged for this substep
  double s1, x2;                      // supb
  double a1u, a1v, a2u, a2v;          // the viscosity's differences
  double pred, dvu, dvv;
  double ubc, vbc;
};

// S2: sch = sqrt(ter(ch)) on U and the fluxes supb; the viscosity's
// differences p1(ub)/rh4 on N and p2(ub) rh2 on E
template <class Pt>
PD void trop_s2(const Pt &T, const TropCoef &K, TropState &s) {
  const int W = T.W;
  const double w = s.c0 + T.S(X_CH, W) + T.S(X_CH, 1) + T.S(X_CH, W + 1);
  double sch = sqrt(T.s2sea ? w : 4.0);
  if (T.s2zero) sch = 0.0;
  const double ps = K.prh_uh * sch;
  s.s1 = ps * s.u0;
  s.x2 = ps * s.v0 * T.Y(10);
  const double dx4 = T.X(3), rdx4 = T.X(7), rh4 = T.Y(11), rrh4 = T.Y(16);
  s.a1u = dvr(dvr(s.u0 - T.S(X_UB, -1), dx4, rdx4), rh4, rrh4);
  s.a1v = dvr(dvr(s.v0 - T.S(X_VB, -1), dx4, rdx4), rh4, rrh4);
  const double dy2 = T.Y(1), rdy2 = T.Y(5), rh2 = T.Y(9);
  s.a2u = dvr(s.u0 - T.S(X_UB, -W), dy2, rdy2) * rh2;
  s.a2v = dvr(s.v0 - T.S(X_VB, -W), dy2, rdy2) * rh2;
  if (!T.srow) s.a2u = s.a2v = 0.0;
  if (T.inR) {
    T.S(X_S1, 0) = s.s1;
    T.S(X_X2, 0) = s.x2;
    T.S(X_A1U, 0) = s.a1u;
    T.S(X_A1V, 0) = s.a1v;
    T.S(X_A2U, 0) = s.a2u;
    T.S(X_A2V, 0) = s.a2v;
  }
}

// divergence of the staged fluxes (the ter U->E and U->N means formed here;
// rows >= 2)
template <class Pt>
PD double trop_div(const Pt &T, const TropState &s) {
  const int W = T.W;
  double A = dvr((T.S(X_S1, -W) + s.s1) - (T.S(X_S1, -W - 1) + T.S(X_S1, -1)), T.X(0), T.X(4));
  double B = dvr((T.S(X_X2, -1) + s.x2) - (T.S(X_X2, -W - 1) + T.S(X_X2, -W)), T.Y(0), T.Y(4));
  if (!T.srow) A = B = 0.0;
  return dvr(A + B, T.Y(12), T.Y(13));
}

// S4: predictor ch (land_ch: ch on land); the viscosity's change since the
// first substep (vs0u, vs0v; set where `first`)
template <class Pt>
PD void trop_s4(const Pt &T, const TropCoef &K, TropState &s, double bt, double gamma_b, double land_ch, bool first,
                double &vs0u, double &vs0v) {
  const int W = T.W;
  const double div = trop_div(T, s);
  s.pred = s.c0 - dvr(div * bt * gamma_b, K.prh_t, K.rprh_t);
  if (!K.sea_t) s.pred = land_ch;
  const double dx3 = T.X(2), rdx3 = T.X(6), dy3 = T.Y(2), rdy3 = T.Y(6), aarh = T.Y(17), raarh = T.Y(18);
  const double L1u = dvr(T.S(X_A1U, 1) - s.a1u, dx3, rdx3), L1v = dvr(T.S(X_A1V, 1) - s.a1v, dx3, rdx3);
  double L2u = dvr(T.S(X_A2U, W) - s.a2u, dy3, rdy3), L2v = dvr(T.S(X_A2V, W) - s.a2v, dy3, rdy3);
  if (!T.nrow) L2u = L2v = 0.0;
  const double vsu = K.sam1 * dvr(L1u + L2u, aarh, raarh), vsv = K.sam1 * dvr(L1v + L2v, aarh, raarh);
  if (first) { vs0u = vsu; vs0v = vsv; }
  s.dvu = vsu - vs0u;
  s.dvv = vsv - vs0v;
  if (T.inR) T.S(X_PRED, 0) = s.pred;
}

// S6: sqrt(ter(pred)), the gradients and means of pred on E (rows j and
// j + 1) and N (columns i and i + 1), all from the same four values, and the
// corrector velocity (pressure gradient, Coriolis adjustment); its fluxes
template <class Pt>
PD void trop_s6(const Pt &T, const TropCoef &K, TropState &s, double bt, double a, double ra) {
  const int W = T.W;
  const double pe = T.S(X_PRED, 1), pn = T.S(X_PRED, W), pne = T.S(X_PRED, W + 1), pred = s.pred;
  const double w = pred + pn + pe + pne;
  double sch = sqrt(T.s6sea ? w : 4.0);
  if (T.s2zero) sch = 0.0;
  const double dx2 = T.X(1), rdx2 = T.X(5), dy4 = T.Y(3), rdy4 = T.Y(7);
  const double gx0 = dvr(dvr(pe - pred, dx2, rdx2), T.Y(14), T.Y(15));
  const double gx1 = dvr(dvr(pne - pn, dx2, rdx2), T.Yn(14), T.Yn(15));
  const double gy0 = dvr(dvr(pn - pred, dy4, rdy4), a, ra), gy1 = dvr(dvr(pne - pe, dy4, rdy4), a, ra);
  double t1 = (gx0 * K.bxn + gx1 * K.bxs) + ((pred + pe) * K.gxn + (pn + pne) * K.gxs);
  double t2 = (gy0 * K.bye + gy1 * K.byw) + ((pred + pn) * K.gye + (pe + pne) * K.gyw);
  if (!T.nrow) t1 = t2 = 0.0;
  const double sbt = K.sea_u ? bt : 0.0, sea4 = K.sea_u ? 0.25 : 0.0;
  const double cb = 0.5 * K.cor * bt, den = 1 + cb * cb;
  const double pg1 = (t1 + K.ghx) * sea4 * sch, pg2 = (t2 + K.ghy) * sea4 * sch;
  const double w1 = (s.dvu + K.ut - pg1 + 0.5 * K.cor * s.v0) * sbt + s.u0;
  const double w2 = (s.dvv + K.vt - pg2 - 0.5 * K.cor * s.u0) * sbt + s.v0;
  const double u1 = 0.5 * (dvr(w1 + cb * w2, den, K.rden) + s.u0);
  const double v1 = 0.5 * (dvr(w2 - cb * w1, den, K.rden) + s.v0);
  s.ubc = (s.dvu - pg1 + K.ut + K.cor * v1) * sbt + s.u0;
  s.vbc = (s.dvv - pg2 + K.vt - K.cor * u1) * sbt + s.v0;
  const double ps = K.prh_uh * sch;
  s.s1 = ps * s.ubc;
  s.x2 = ps * s.vbc * T.Y(10);
  if (T.inR) {
    T.S(X_S1, 0) = s.s1;
    T.S(X_X2, 0) = s.x2;
  }
}

// S8: corrector ch
template <class Pt>
PD double trop_s8(const Pt &T, const TropCoef &K, const TropState &s, double bt) {
  return s.c0 - dvr(trop_div(T, s) * (K.sea_t ? bt : 0.0), K.prh_t, K.rprh_t);
}
