// kc_init_lean.cuh — the limotorus profile of one (x1, x2) column by a warp
// (include/koral/kinit.h init_dsandvels_s; puffy.zig:572).
//
// A column is a bisection inside a bisection (the radius of the maximum: ~60
// outer steps of ~60 inner ones) and an adaptive GK21 quadrature whose every
// point bisects too: some 15 million dependent operations for one thread. Here
// the warp's lanes take
//  - the 31 midpoints that the next five outer bisection steps can meet (a binary
//    tree of outcomes): each lane forms its node's midpoint by the very updates
//    the serial loop would make on the way there, and the warp then walks the
//    tree by the signs found: five steps a round, the same midpoints, the same
//    stop;
//  - the 21 nodes of a quadrature rule, summed afterwards in the serial order.
// The angular momentum outside its broken-power-law range is a constant, formed
// once, and without spin its two powers are multiplied by zero: 1 - 0/x + 0 and
// 1 - 2/r + 0/x are formed without x. All values are the serial code's bits.
// Measured at 192x180 columns: 205 ms one thread per column.
#pragma once
#include "../../include/koral/kinit.h"

namespace kc {
namespace lean {

// kcinit::l3d with the constants beyond its range
struct TorusL {
  double a, lb1, lb2, xi;
  double l1, l2;  // xi lK(lb1), xi lK(lb2)
  KC_HD double lk(double r) const {
    if (a == 0.0 && r > 0x1p-100 && r < 0x1p+100) return kmath::sqrt(r) / (1.0 - 2.0 / r);
    return kcinit::lK(r, a);
  }
  KC_HD double l3d(double lam) const { return lam <= lb1 ? l1 : (lam >= lb2 ? l2 : xi * lk(lam)); }
  // kcinit::lam_bl
  KC_HD double lam_bl(double R, const kcinit::Gd& gd) const {
    const double x1 = R, x2 = 10.0 * R;
    double dx, rtb;
    if (at(x1, gd) < 0.0) {
      dx = x2 - x1;
      rtb = x1;
    } else {
      dx = x1 - x2;
      rtb = x2;
    }
    for (int j = 1; j <= 100; ++j) {
      dx *= 0.5;
      const double xmid = rtb + dx;
      const double fmid = at(xmid, gd);
      if (fmid <= 0.0) rtb = xmid;
      if (kmath::fabs(dx) < kcinit::kXacc || fmid == 0.0) return rtb;
    }
    return 0.0;
  }
  KC_HD double at(double lam, const kcinit::Gd& gd) const {
    const double l = l3d(lam);
    return lam * lam + l * (l * gd.gdtp + gd.gdpp) / (l * gd.gdtt + gd.gdtp);
  }
  // the outer function of kcinit::find_rml
  KC_HD double rml_at(double x, double lamsq) const {
    const kcinit::Gd gd = kcinit::compute_gd(x, kcinit::kPi2, a);
    const double lx = lam_bl(x, gd);
    return lamsq - lx * lx;
  }
  // kcinit::LnfIntegrand
  KC_HD double lnf(double r) const {
    const double r2 = r * r, r3 = r2 * r, a2 = a * a;
    const kcinit::Gd gd = kcinit::compute_gd(r, kcinit::kPi2, a);
    const double lam = lam_bl(r, gd);
    const double lam2 = lam * lam;
    const double l = l3d(lam);
    const double term1 = (r - 2.0) * l, term2 = 2.0 * a, term3 = r3 + a2 * (r + 2.0), term4 = term2 * l;
    const double om_num = term1 + term2, om_den = term3 - term4;
    const double om = om_num / om_den;
    double dl_dr = 0.0;
    if (!(lam <= lb1 || lam >= lb2)) {
      const double oneplusx = 1.0 - 2.0 / lam + a * kmath::pow(lam, -1.5);
      const double dx_dlam = 2.0 * kmath::pow(lam, -2.0) - 1.5 * a * kmath::pow(lam, -2.5);
      const double lamroot = kmath::sqrt(lam);
      const double dlk_dlam = (oneplusx * 0.5 * (1.0 / lamroot) + (a - lamroot) * dx_dlam) / (oneplusx * oneplusx);
      const double dd = term3 - 2.0 * term4 - lam2 * (r - 2.0);
      const double ee = l * (3.0 * r2 + a2 - lam2);
      dl_dr = ee / (2.0 * lam * om_num / (xi * dlk_dlam) - dd);
    }
    const double dom_dr =
        (om_den * (l + (r - 2.0) * dl_dr) - om_num * (3.0 * r2 + a2 + 2.0 * a * dl_dr)) / (om_den * om_den);
    return -l / (1.0 - om * l) * dom_dr;
  }
};
KC_HD TorusL torus_l(double a, double lb1, double lb2, double xi) {
  TorusL t = {a, lb1, lb2, xi, xi * kcinit::lK(lb1, a), xi * kcinit::lK(lb2, a)};
  return t;
}

// The node of the outcome tree that lane (0..30) of a round looks at: starting
// from the bracket (rtb, dx), its midpoint after the steps that lead there. Nodes
// are numbered from 1 (the root), 2n after a positive value, 2n + 1 after f <= 0.
KC_HD double tree_midpoint(int node, double rtb, double dx) {
  int top = 16;
  while (top > node) top >>= 1;
  for (top >>= 1; top; top >>= 1) {
    dx *= 0.5;
    const double xmid = rtb + dx;
    if (node & top) rtb = xmid;
  }
  return rtb + dx * 0.5;
}

#if defined(__CUDACC__)
// kcinit::find_rml
__device__ double find_rml_warp(const TorusL& t, double lam) {
  const unsigned all = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const double lamsq = lam * lam;
  const double x1 = 6.0, x2 = 10.0 * lamsq;
  double dx, rtb;
  if (t.rml_at(x1, lamsq) < 0.0) {
    dx = x2 - x1;
    rtb = x1;
  } else {
    dx = x1 - x2;
    rtb = x2;
  }
  for (int j = 0; j < 100; j += 5) {
    const double f = t.rml_at(tree_midpoint(lane < 31 ? lane + 1 : 1, rtb, dx), lamsq);
    for (int node = 1; node < 32;) {
      dx *= 0.5;
      const double xmid = rtb + dx;
      const double fmid = __shfl_sync(all, f, node - 1);
      if (fmid <= 0.0) rtb = xmid;
      if (kmath::fabs(dx) < kcinit::kXacc || fmid == 0.0) return rtb;
      node = 2 * node + (fmid <= 0.0);
    }
  }
  return 0.0;
}
// kcinit::gk21 of the torus integrand
__device__ void gk21_warp(const TorusL& t, double a, double b, double& value, double& abserr) {
  const double kXgk[11] = {
      0.995657163025808080735527280689003, 0.973906528517171720077964012084452,
      0.930157491355708226001207180059508, 0.865063366688984510732096688423493,
      0.780817726586416897063717578345042, 0.679409568299024406234327365114874,
      0.562757134668604683339000099272694, 0.433395394129247190799265943165784,
      0.294392862701460198131126603103866, 0.148874338981631210884826001129720,
      0.000000000000000000000000000000000};
  const double kWgk[11] = {
      0.011694638867371874278064396062192, 0.032558162307964727478818972459390,
      0.054755896574351996031381300244580, 0.075039674810919952767043140916190,
      0.093125454583697605535465065083366, 0.109387158802297641899210590325805,
      0.123491976262065851077958109831074, 0.134709217311473325928054001771707,
      0.142775938577060080797094273138717, 0.147739104901338491374841515972068,
      0.149445554002916905664936468389821};
  const double kWg[5] = {
      0.066671344308688137593568809893332, 0.149451349150580593145776339657697,
      0.219086362515982043995534934228163, 0.269266719309996355091226921569469,
      0.295524224714752870173892994651338};
  const unsigned all = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const double c = 0.5 * (a + b), h = 0.5 * (b - a);
  // lanes 2k and 2k+1: c -+ h kXgk[k]; the others the centre
  double xg = 0.0;
#pragma unroll
  for (int k = 0; k < 10; ++k)
    if (lane / 2 == k) xg = kXgk[k];
  const double x = h * xg;
  const double f = t.lnf(lane >= 20 ? c : (lane & 1) ? c + x : c - x);
  const double fc = __shfl_sync(all, f, 20);
  double resg = 0.0, resk = kWgk[10] * fc;
#pragma unroll
  for (int j = 0; j < 5; ++j) {
    const int jtw = 2 * j + 1;
    const double fsum = __shfl_sync(all, f, 2 * jtw) + __shfl_sync(all, f, 2 * jtw + 1);
    resg += kWg[j] * fsum;
    resk += kWgk[jtw] * fsum;
  }
#pragma unroll
  for (int j = 0; j < 5; ++j) {
    const int jtw = 2 * j;
    resk += kWgk[jtw] * (__shfl_sync(all, f, 2 * jtw) + __shfl_sync(all, f, 2 * jtw + 1));
  }
  value = resk * h;
  abserr = kmath::fabs((resk - resg) * h);
}
// kcinit::integrate of the torus integrand; seg: the warp's 4 kMaxSeg doubles
__device__ bool integrate_warp(const TorusL& t, double a, double b, double epsrel, double& out, double* seg) {
  using kcinit::kMaxSeg;
  if (a == b) {
    out = 0.0;
    return true;
  }
  const int lane = threadIdx.x & 31;
  double *sa = seg, *sb = seg + kMaxSeg, *sv = seg + 2 * kMaxSeg, *se = seg + 3 * kMaxSeg;
  auto put = [&](int i, double lo, double hi, double v, double e) {
    if (lane == 0) {
      sa[i] = lo;
      sb[i] = hi;
      sv[i] = v;
      se[i] = e;
    }
  };
  int nseg = 1;
  {
    double v, e;
    gk21_warp(t, a, b, v, e);
    put(0, a, b, v, e);
  }
  for (;;) {
    __syncwarp();
    double total = 0.0, toterr = 0.0, most = 0.0;
    int worst = 0;
    for (int i = 0; i < nseg; ++i) {
      const double e = se[i];
      total += sv[i];
      toterr += e;
      if (i == 0 || e > most) {
        most = e;
        worst = i;
      }
    }
    out = total;
    if (toterr <= kmath::fmax(0.0, epsrel * kmath::fabs(total))) return true;
    if (nseg == kMaxSeg) return false;
    const double lo = sa[worst], hi = sb[worst];
    const double mid = 0.5 * (lo + hi);
    double lv, le, rv, re;
    gk21_warp(t, lo, mid, lv, le);
    gk21_warp(t, mid, hi, rv, re);
    __syncwarp();
    put(worst, lo, mid, lv, le);
    put(nseg, mid, hi, rv, re);
    nseg += 1;
  }
}
// kcinit::init_dsandvels_s, by a whole warp
__device__ kcinit::DsVels init_column_warp(double r, double th, const TorusL& t, const kcinit::TorusConsts& tc,
                                           const kcinit::PuffyPhysics& ph, double* seg) {
  kcinit::DsVels o = {-1.0, 0.0, 0.0};
  const double R = r * kmath::sin(th);
  if (R < ph.lt_rin) return o;
  const kcinit::Gd gd = kcinit::compute_gd(r, th, t.a);
  const double lam = t.lam_bl(R, gd);
  const double l = t.l3d(lam);
  const double om = kcinit::omega3d(l, gd);
  const double agrav = kcinit::compute_agrav(om, gd);
  const double rml = find_rml_warp(t, lam);
  double q;
  const bool conv = integrate_warp(t, ph.lt_rin, rml, 1.0e-12, q, seg);
  const double lnf3d = conv ? q : -kmath::inf();
  const double f3d = kmath::exp(-lnf3d);
  const double f3din = 1.0;
  const double hh = f3din * agrav / (f3d * tc.agravin);
  const double eps = (-1.0 + hh) * (1.0 / ph.lt_gamma);
  const double rho = (eps < 0.0) ? -1.0
                                 : kmath::pow((-1.0 + ph.lt_gamma) * eps * (1.0 / ph.lt_kappa), 1.0 / (-1.0 + ph.lt_gamma));
  o.rho = rho;
  o.ell = l;
  o.uu = ph.lt_kappa * kmath::pow(rho, ph.lt_gamma) / (ph.lt_gamma - 1.0);
  return o;
}
#endif

}  // namespace lean
}  // namespace kc
