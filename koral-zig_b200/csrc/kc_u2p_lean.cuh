// kc_u2p_lean.cuh — the W inversion (koral/solve/invert.zig:240) with each
// residual evaluated once.
//
// kp::u2p_solver_w evaluates the residual of an accepted W twice: as the trial
// of one Newton step and again as the start of the next (and the first W a
// third time, in the bounds loop). The residual is a pure function of W, so
// this form carries the accepted trial's value over; every value formed is the
// one the plain form has, in the same order of operations, and the loops are
// merged into one so that the residual stands in the code once. A Newton step
// is a serial chain of some ten divisions and a square root, which is what
// bounds the inversion on a small grid.
// Host and device: the CPU test compares it bit for bit with the plain form.
#pragma once
#include "../../include/koral/kinvert.h"

namespace kc {
namespace lean {

using namespace kp;

// kmath::pow for a positive exponent below 3.5 and a base whose powers stay in the
// normal range: exp(yf log x) times x, x x or x (x x), the products pow's loop
// forms from x's fraction and exponent apart; pow itself for anything else.
KC_HD double pow_pos(double x, double y) {
  if (!(x > 0x1p-200 && x < 0x1p+200 && y > 0.0 && y < 3.5 && y != 0.5)) return kmath::pow(x, y);
  double yi = kmath::trunc(y);
  double yf = y - yi;
  double a = 1.0;
  if (yf != 0.0) {
    if (yf > 0.5) {
      yf -= 1.0;
      yi += 1.0;
    }
    a = kmath::exp(yf * kmath::log(x));
  }
  const int n = (int)yi;
  if (n & 1) a *= x;
  if (n & 2) a *= x * x;
  return a;
}
// kp::s_from_u (hydro.zig:31)
KC_HD double entropy(double rho, double u, double gam) {
  const double gammam1 = gam - 1.0;
  const double indexn = 1.0 / gammam1;
  const double pre = gammam1 * u;
  return rho * kmath::log(pow_pos(pre, indexn) / pow_pos(rho, indexn + 1.0));
}

struct WRes {
  double f, df, den;  // err = |f| / den
};
// kp::f_u2p_hot / f_u2p_entropy (invert.zig:121, :170)
KC_HD WRes w_residual(int etype, double W, double D, double Qn, double Qtsq, double QdotBsq, double Bsq, double Sc,
                      double pgamma) {
  const double Wp = W - D;
  W = Wp + D;  // the residual's own W (it takes W - D)
  const double x = Bsq + W;
  const double wsq = W * W;
  const double w3 = wsq * W;
  const double x3 = x * x * x;
  double v2, gamma, gamma2, rho0, wmrho0;
  w_kinematics(W, Wp, D, Qtsq, QdotBsq, Bsq, v2, gamma, gamma2, rho0, wmrho0);
  const double dvsq = -2.0 / x3 * (Qtsq + QdotBsq * (3.0 * W * x + Bsq * Bsq) / w3);
  const double dwmrho0dvsq = D * (gamma * 0.5 - 1.0) - Wp;
  WRes r;
  if (etype == ETYPE_HOT) {
    const double u = wmrho0 / pgamma;
    const double p = (pgamma - 1.0) * u;
    const double half = 0.5 * Bsq * (1.0 + v2), q2 = QdotBsq / 2.0 / wsq;
    r.f = Qn + W - p + half - q2;
    r.den = kmath::fabs(Qn) + kmath::fabs(W) + kmath::fabs(p) + kmath::fabs(half) + kmath::fabs(q2);
    const double dp1 = (pgamma - 1.0) * (1.0 - v2) / pgamma;
    const double idwmrho0dp = (pgamma - 1.0) / pgamma;
    const double dp2 = dwmrho0dvsq * idwmrho0dp;
    const double dpdW = dp1 + dp2 * dvsq;
    r.df = 1.0 - dpdW + QdotBsq / w3 + 0.5 * Bsq * dvsq;
  } else {
    const double pressure = (pgamma - 1.0) / pgamma * wmrho0;
    const double indexn = 1.0 / (pgamma - 1.0);
    const double ssofchi = kmath::log(pow_pos(pressure, indexn) / pow_pos(rho0, indexn + 1.0));
    r.f = -Sc + D * ssofchi;
    r.den = kmath::fabs(Sc) + kmath::fabs(D * ssofchi);
    const double dssdrho = pgamma / ((1.0 - pgamma) * rho0);
    const double dssdchi = 1.0 / ((pgamma - 1.0) * wmrho0);
    const double dwmrho0dw = 1.0 / (gamma * gamma);
    const double drho0dvsq = -D * gamma * 0.5;
    const double dssdw = dwmrho0dw * dssdchi;
    const double dssdvsq = drho0dvsq * dssdrho + dwmrho0dvsq * dssdchi;
    r.df = D * (dssdw + dssdvsq * dvsq);
  }
  return r;
}
// the part of kp::w_out_of_bounds (invert.zig:224) that reads W alone
KC_HD bool w_outside(double W, double Qtsq, double QdotBsq, double Bsq) {
  return (W * W * W * (W + 2.0 * Bsq) - QdotBsq * (2.0 * W + Bsq)) <= W * W * (Qtsq - Bsq * Bsq);
}

// kp::u2p_solver_w. Reads uu[RHO..VZ], uu[B1..B3] and, for the entropy solve,
// uu[ENTR]; the entropy of the result (pp[ENTR]) is written when with_entropy.
KC_HD int u2p_w(const double uu[NV], double pp[NV], const Geom& g, int etype, double pgamma, bool with_entropy) {
  const double conv = 1.0e-10;
  const double big = 1.0 / 1.0e-80;
  const double gdetu_inv = 1.0 / g.gdet;
  const double alpha = g.alpha;
  const double D = uu[RHO] * gdetu_inv * alpha;
  const double Sc = (etype == ETYPE_ENTROPY || with_entropy) ? uu[ENTR] * gdetu_inv * alpha : 0.0;
  double Qcov[4] = {(uu[UU] * gdetu_inv - uu[RHO] * gdetu_inv) * alpha, uu[VX] * gdetu_inv * alpha,
                    uu[VY] * gdetu_inv * alpha, uu[VZ] * gdetu_inv * alpha};
  double Qcon[4];
  raise_vec(Qcov, g, Qcon);
  double Bcon[4] = {0.0, uu[B1] * gdetu_inv * alpha, uu[B2] * gdetu_inv * alpha, uu[B3] * gdetu_inv * alpha};
  double Bcov[4];
  lower_vec(Bcon, g, Bcov);
  const double Bsq = dot(Bcon, Bcov);
  const double QdotB = dot(Qcov, Bcon);
  const double QdotBsq = QdotB * QdotB;
  double ncov[4] = {-alpha, 0.0, 0.0, 0.0};
  double ncon[4];
  raise_vec(ncov, g, ncon);
  const double Qn = Qcon[0] * ncov[0];
  double Qtcon[4];
  for (int i = 0; i < 4; ++i) {
    Qtcon[i] = 0.0;
    for (int j = 0; j < 4; ++j) Qtcon[i] += (kron(i, j) + ncon[i] * ncov[j]) * Qcon[j];
  }
  double Qtcov[4];
  lower_vec(Qtcon, g, Qtcov);
  const double Qtsq = dot(Qtcon, Qtcov);

  double qsq = 0.0;
  {
    const double ut[4] = {0.0, pp[VX], pp[VY], pp[VZ]};
    for (int i = 1; i < 4; ++i)
      for (int j = 1; j < 4; ++j) qsq += ut[i] * ut[j] * g.gg[i][j];
  }
  double W = (pp[RHO] + pgamma * pp[UU]) * (1.0 + qsq);

  // mode 0: the bounds loop; 1: a damped Newton trial; 2: W moved off a zero slope.
  // A W outside the bounds is moved without forming its residual; a damped trial
  // of a state that has no solution is moved so a hundred times an iteration.
  double Wt = W, f0 = 0.0, df = 1.0, q0 = 0.0, errr = 0.0, dumpfac = 1.0;
  bool q_exact = false;
  int mode = 0, grow = 0, idump = 0, iter = 0;
  KC_ROLLED
  for (;;) {
    WRes r;
    bool bad = mode != 2 && w_outside(Wt, Qtsq, QdotBsq, Bsq);
    if (!bad) {
      r = w_residual(etype, Wt, D, Qn, Qtsq, QdotBsq, Bsq, Sc, pgamma);
      bad = !kmath::isfinite(r.f) || !kmath::isfinite(r.df);
    }
    if (mode == 0) {
      if (bad && grow < 50) {
        Wt *= 10.0;
        grow += 1;
        continue;
      }
      if (grow >= 50) return -150;
      W = Wt;
    } else if (mode == 1) {
      if (bad && idump < 100) {
        idump += 1;
        dumpfac /= 2.0;
        Wt = W - (q_exact ? dumpfac * q0 : dumpfac * f0 / df);
        continue;
      }
      if (idump >= 100) return -101;
      const double Wprev = W;
      W = Wt;
      if (kmath::fabs(W) > big) return -103;
      if (kmath::fabs((W - Wprev) / Wprev) < conv && errr < 1.0e-1) break;
    } else {
      W = Wt;
    }
    if (iter >= 50) break;
    iter += 1;
    errr = kmath::fabs(r.f) / r.den;
    if (errr < conv) break;
    if (r.df == 0.0) {
      Wt = W * 1.1;
      mode = 2;
      continue;
    }
    f0 = r.f;
    df = r.df;
    q0 = f0 / df;
    Wt = W - q0;
    // a power of two times f0, over df, is that power times f0 / df while neither
    // leaves the normal range
    q_exact = kmath::fabs(f0) > 0x1p-900 && kmath::fabs(q0) > 0x1p-900 && kmath::fabs(q0) < kmath::inf();
    idump = 0;
    dumpfac = 1.0;
    mode = 1;
  }
  if (iter >= 50) return -102;
  if (!kmath::isfinite(W)) return -103;

  const double wsq = W * W;
  const double xsq = (Bsq + W) * (Bsq + W);
  const double v2 = (wsq * Qtsq + QdotBsq * (Bsq + 2.0 * W)) / (wsq * xsq);
  const double gamma2 = 1.0 / (1.0 - v2);
  const double gamma = kmath::sqrt(gamma2);
  const double rho = D / gamma;
  const double uint_ = 1.0 / pgamma * (W / gamma2 - rho);
  double utcon[4];
  for (int i = 1; i < 4; ++i) utcon[i] = gamma / (W + Bsq) * (Qtcon[i] + QdotB * Bcon[i] / W);
  if (!kmath::isfinite(utcon[1])) return -120;
  if (uint_ < 0.0 || gamma2 < 0.0 || kmath::isnan(W) || !kmath::isfinite(W)) return -104;
  pp[RHO] = rho;
  pp[UU] = uint_;
  pp[VX] = utcon[1];
  pp[VY] = utcon[2];
  pp[VZ] = utcon[3];
  if (rho < 0.0) return -105;
  if (with_entropy) pp[ENTR] = Sc / gamma;
  pp[B1] = uu[B1] * gdetu_inv;
  pp[B2] = uu[B2] * gdetu_inv;
  pp[B3] = uu[B3] * gdetu_inv;
  return 0;
}

// kp::u2p_mhd (invert.zig:422): the hot solve and, where it fails, the entropy
// solve, through one copy of the code
KC_HD U2pMhdRes u2p_mhd(const double uu_in[NV], double pp[NV], const Geom& g, double pgamma, const FloorParams& fl) {
  double uu[NV], ppmhd[NV];
  for (int i = 0; i < NV; ++i) {
    uu[i] = uu_in[i];
    ppmhd[i] = pp[i];
  }
  U2pMhdRes r;
  r.ret = 0;
  r.entropy_used = false;
  if (uu[RHO] * g.alpha / g.gdet < 0.0) {
    ppmhd[RHO] = fl.rhofloor;
    uu[RHO] = fl.rhofloor * g.gdet / g.alpha;
    r.ret = -2;
  }
  int ret, etype = ETYPE_HOT;
  KC_ROLLED
  for (;;) {
    ret = u2p_w(uu, ppmhd, g, etype, pgamma, true);
    if (ret >= 0 || etype == ETYPE_ENTROPY) break;
    r.ret = -1;
    r.entropy_used = true;
    etype = ETYPE_ENTROPY;
  }
  if (ret >= 0) {
    for (int i = 0; i < NV; ++i) pp[i] = ppmhd[i];
  } else {
    r.ret = -3;
  }
  r.fixup = r.ret < -1;
  return r;
}

}  // namespace lean
}  // namespace kc
