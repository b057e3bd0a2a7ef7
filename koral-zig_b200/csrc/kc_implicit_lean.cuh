// kc_implicit_lean.cuh — the implicit radiation-gas solve
// (koral/solve/implicit.zig:927) with only the values that reach its result.
//
// kp::solve_implicit_lab (include/koral/kimplicit.h) is the reference's solve as
// it stands: each trial state fills the whole radiation state. Most of that fill
// is never read, or is the same in every trial of a cell. Here
//  - the 1-D bisection forms the velocities, b^2 and the radiation frame once
//    (its trials share them) and no Rosseland mean (it reads the absorption
//    opacities and the Compton term only: 2 of the 8 powers of a full fill);
//  - the constraints leave out the entropy (two powers and a logarithm each),
//    which only the accepted state and the entropy fallback read; it is formed
//    there from the same operands;
//  - the gas velocities and b^2 of the constrained state serve its radiation
//    state too, and an accepted trial is filled only when another iteration
//    starts from it (most solves end there);
//  - powers of one argument share its logarithm;
//  - the constraints and the residual each stand in the code once: the start,
//    the finite-difference columns and the damped trials go through one loop,
//    so lanes in different stages share the instructions, and the loop of a
//    solve fits the instruction cache;
//  - the gas inversion evaluates each residual once (kc_u2p_lean.cuh).
// Every value formed is formed by the operations of the plain solve in their
// order, so the results are the same bits (host and device; the CPU test compares
// the two over options and states).
//
// The kernels that use it (k_implicit_warm, k_implicit, k_batch_solve) say what
// bounds it and what it measured.
#pragma once
#include "../../include/koral/kimplicit.h"
#include "kc_u2p_lean.cuh"

#if defined(__CUDACC__)
#define KC_UNROLL _Pragma("unroll")
#else
#define KC_UNROLL
#endif

namespace kc {
namespace lean {

using namespace kp;

// ---- powers of a shared logarithm ---------------------------------------------
// kmath::pow(x, y) for a fixed y > 0 is exp(yf log x) times x^yi, formed from x's
// fraction and exponent apart. Inside [2^-200, 2^200] no step of it can leave
// the normal range, the exponent only scales exactly, and the product with x (or
// x x) itself rounds to the same bits; outside (and for NaN) pow is called.
struct PowArg {
  double x, lx;
  bool in;
};
// INL: the transcendentals inline (the warm start, whose loop is short: 6% faster)
// or out of line (the ladder, whose code is larger than the instruction cache
// otherwise: instruction-fetch stalls 2.2 -> 1.4 a warp instruction, 7% faster)
template <bool INL>
KC_HD double exp_(double x) { return INL ? kmath::exp_inl(x) : kmath::exp(x); }
template <bool INL>
KC_HD double cbrt_(double x) { return INL ? kmath::cbrt_inl(x) : kmath::cbrt(x); }
template <bool INL>
KC_HD PowArg pow_arg(double x) {
  PowArg a;
  a.x = x;
  a.in = x > 0x1p-200 && x < 0x1p+200;
  a.lx = INL ? kmath::log_inl(a.in ? x : 1.0) : kmath::log(a.in ? x : 1.0);
  return a;
}
// y in (0, 0.5]: exp(y log x)
template <bool INL>
KC_HD double pow_frac(const PowArg& a, double y) { return a.in ? exp_<INL>(y * a.lx) : kmath::pow(a.x, y); }
// y in (0.5, 1): exp((y - 1) log x) x
template <bool INL>
KC_HD double pow_up1(const PowArg& a, double y) {
  return a.in ? exp_<INL>((y - 1.0) * a.lx) * a.x : kmath::pow(a.x, y);
}
// y in (1.5, 2): exp((y - 1 - 1) log x) (x x)
template <bool INL>
KC_HD double pow_up2(const PowArg& a, double y) {
  return a.in ? exp_<INL>((y - 1.0 - 1.0) * a.lx) * (a.x * a.x) : kmath::pow(a.x, y);
}

// ---- opacities ------------------------------------------------------------------
struct OpacLean {
  double gas_abs, rad_abs, rad_ross;
};
// The channels of kp::calc_opacities (opacities.zig:131) that the four-force
// reads, trad = tradbb; rad_ross only with ROSS (the ladder's form).
template <bool ROSS>
KC_HD OpacLean opacities(const Consts& c, const Channels& ch, double rho, double te, double trad, double ne, double bsq) {
  const double rt_te = kmath::sqrt(te);
  const double rhocgs = c.rhogu2cgs * rho;
  const double nethcgs = ne * c.numdensgu2cgs;
  const double bsqcgs = c.fourpi * (bsq * c.enden_gu2cgs_fac);
  const double bmagcgs = kmath::sqrt(bsqcgs);
  const double bbenergy = (4.0 * c.sigma_rad_cgs) * te * te * te * te;
  double kappagasff = 0, kapparadff = 0, kapparadffross = 0;
  double kappagassyn = 0, kapparadsyn = 0, kapparadsynross = 0;
  if (ch.bremsstrahlung) {
    const double mfrac = 1.0 - c.hfrac - c.hefrac;
    const double emis_ff = 1.4e-27 * nethcgs * ((c.hfrac + c.hefrac + c.z2diva_mean * mfrac) / c.m_proton_cgs) * rt_te *
                           1.2 * (1.0 + 4.4e-10 * te);
    kappagasff = c.kappacgs2gu * (emis_ff / bbenergy) * rho;
    const double zeta = trad / te;
    const double zeta_inv = 1.0 / zeta;
    const double zeta_inv_3 = zeta_inv * zeta_inv * zeta_inv;
    kapparadff = kappagasff * (ROSS ? kmath::log1p(1.6 * zeta) : kmath::log1p_inl(1.6 * zeta)) * c.one_over_log_2p6 * zeta_inv_3;
    if (ROSS) {
      const double zeta_root5 = pow_frac<!ROSS>(pow_arg<!ROSS>(zeta), 0.2);
      const double zeta_root5_inv_4 = 1.0 / (zeta_root5 * zeta_root5 * zeta_root5 * zeta_root5);
      const double zeta_root5_inv_3 = zeta_root5 * zeta_root5_inv_4;
      const double scale_pla_ros_ff =
          14.12 / (432.7 - 106.8 * zeta_root5_inv_3 + 43.17 * zeta_root5_inv_4 + 57.88 * zeta_inv);
      kapparadffross = kappagasff * scale_pla_ros_ff * zeta_inv_3;
    }
  }
  if (ch.synchrotron) {
    const bool bridge = ch.synchrotron_bridge != 0;
    double trad_syn = trad;
    if (bridge) {
      const double trad_lim = kmath::pow(trad, 4.0 / 3.0) / kmath::pow(te, 1.0 / 3.0);
      trad_syn = (trad < trad_lim) ? trad_lim : trad;
    }
    const double ne_rho = nethcgs / rhocgs;
    const double emis_synchro = 3.61e-34 * ne_rho * te * te * bmagcgs * bmagcgs;
    kappagassyn = c.kappacgs2gu * (emis_synchro / bbenergy) * rho;
    const double nu_mbsyn = 1.19e-13 * te * te;
    const double zbr = (c.k_boltz_cgs * trad_syn / c.h_cgs) / nu_mbsyn;
    const double zeta_a_denom_rad =
        1.79 * cbrt_<!ROSS>(zbr * zbr * zbr * zbr * zbr * bmagcgs * bmagcgs * bmagcgs * bmagcgs) +
        1.35 * cbrt_<!ROSS>(zbr * zbr * zbr * zbr * zbr * zbr * zbr * bmagcgs * bmagcgs) + 0.248 * zbr * zbr * zbr;
    const double ia_by_b_rad = bmagcgs * bmagcgs / zeta_a_denom_rad;
    const double te5 = te * te * te * te * te;
    const double synfac = 2.13e39 * ne_rho / te5;
    kapparadsyn = c.kappacgs2gu * (synfac * ia_by_b_rad) * rho;
    if (bridge)
      kapparadsyn += c.kappacgs2gu * (2.35869e-21 * ne_rho * (bmagcgs * bmagcgs) / (trad_syn * trad_syn * trad_syn)) * rho;
    if (ROSS) {
      // a field-free cell (bmag 0) takes pow's values at zero directly
      double bmb = 0.0, b69 = 0.0;
      if (bmagcgs != 0.0) {
        const PowArg ab = pow_arg<!ROSS>(bmagcgs);
        bmb = (bmagcgs > 0.0) ? (ab.in ? 1.0 / exp_<!ROSS>(0.463 * ab.lx) : kmath::pow(bmagcgs, -0.463)) : 0.0;
        b69 = pow_up1<!ROSS>(ab, 0.69);
      }
      const PowArg az = pow_arg<!ROSS>(zbr);
      const double ia_by_b_ross_rad =
          0.13 * b69 / (pow_up2<!ROSS>(az, 1.69) * exp_<!ROSS>(1.6 * pow_frac<!ROSS>(az, 0.463) * bmb));
      kapparadsynross = c.kappacgs2gu * (synfac * ia_by_b_ross_rad) * rho;
    }
    if (bridge) kappagassyn += c.kappacgs2gu * (2.35869e-21 * ne_rho * (bmagcgs * bmagcgs) / (te * te * te)) * rho;
    if (!bridge) {
      const double terel = te * c.k_over_mecsq;
      const double terelfactor = (terel * terel) / (1.0 + terel * terel);
      kappagassyn *= terelfactor;
      kapparadsyn *= terelfactor;
      if (ROSS) kapparadsynross *= terelfactor;
    }
  }
  OpacLean o;
  o.gas_abs = kappagasff + kappagassyn;
  o.rad_abs = kapparadff + kapparadsyn;
  o.rad_ross = ROSS ? kapparadffross + kapparadsynross : 0.0;
  return o;
}
// kp::kappaes_at (opacities.zig:352)
template <bool INL>
KC_HD double kappaes(const OpacParams& op, double rho, double trad) {
  if (op.kappaes_mode == KAPPAES_PUFFY) {
    double opac_correction = 1.0;
    if (op.ch.kleinnishina) opac_correction = 1.0 / (1.0 + pow_up1<INL>(pow_arg<INL>(trad / 4.5e8), 0.86));
    return ((0.2 * (1.0 + op.c.hfrac)) * opac_correction) * op.c.kappa_cgs2gu_fac * rho;
  }
  if (op.kappaes_mode == KAPPAES_GREY) return op.kappaes_grey * rho;
  return 0.0;
}
// absorption of kp::fill_rad_state in either opacity mode
template <bool ROSS>
KC_HD OpacLean absorption(const OpacParams& op, double rho, double te, double trad, double ne, double bsq) {
  if (op.kappa_mode == KAPPA_DEFAULT) return opacities<ROSS>(op.c, op.ch, rho, te, trad, ne, bsq);
  const double kap = op.kappa_grey * rho;
  OpacLean o = {kap, kap, kap};
  return o;
}
// kp::temps_from_urho's electron temperature
KC_HD double te_of(double tgas) {
  const double te = kmath::isfinite(tgas) ? tgas : KP_BIG;
  return (te < KP_TEMPEMINIMAL) ? KP_TEMPEMINIMAL : te;
}
KC_HD double tgas_of(const Consts& c, double uint_, double rho, double gam) {
  const double p = uint_ * (gam - 1.0);
  return c.mugas_mp_over_kb * p / rho;
}
// kp::compton_gi_coeff
KC_HD double compton(const Consts& c, double kes, double ehat, double trad, double te) {
  const double thetae = c.kb_over_me * te;
  return kes * ehat * ((4.0 * c.kb_over_me) * (trad - te)) * (1.0 + 3.683 * thetae + 4.0 * thetae * thetae) /
         (1.0 + 4.0 * thetae);
}
// R^mu nu u_mu u_nu (radforce.zig:241) of the M1 closure with energy erf and
// frame velocity urf
KC_HD double rij_ehat(double erf, const double urf[4], const Geom& g, const double ucov[4]) {
  const double four_third = 4.0 / 3.0, one_third = 1.0 / 3.0;
  double ehat = 0.0;
  for (int i = 0; i < 4; ++i)
    for (int j = 0; j < 4; ++j) {
      const double r = four_third * erf * urf[i] * urf[j] + one_third * erf * g.GG[i][j];
      ehat += r * ucov[i] * ucov[j];
    }
  return ehat;
}

// ---- the warm start (implicit.zig:473, :941-961) ---------------------------------
struct Warm {
  double uu, ee;  // the start state: pp00 with these energies
  double ehat;    // the reference state's radiation energy in the gas frame
  double entr;    // and conserved entropy
  int startwith;
};
// BISECT as ImplicitParams::start_with_bisect
KC_HD Warm warm_start(const double pp00[NV], const Geom& g, double dt, double gam, const OpacParams& op,
                      const ImplicitParams& ip) {
  const Consts& c = op.c;
  Warm w;
  w.uu = pp00[UU];
  w.ee = pp00[EE];
  double ucon[4], ucov[4], urf[4];
  {
    double vin[4] = {0.0, pp00[VX], pp00[VY], pp00[VZ]};
    velr_to_vel4(vin, g, ucon);
    lower_vec(ucon, g, ucov);
    double fin[4] = {0.0, pp00[FX], pp00[FY], pp00[FZ]};
    velr_to_vel4(fin, g, urf);
  }
  w.entr = g.gdet * (pp00[ENTR] * ucon[0]);
  {
    // kp::calc_ff_rtt: the start fluid's own radiation energy (radiation.zig:104)
    const double four_third = 4.0 / 3.0, one_third = 1.0 / 3.0, erf = pp00[EE];
    double rtt = 0.0;
    for (int ia = 0; ia < 4; ++ia) {
      double r[4];
      for (int k = 0; k < 4; ++k) r[k] = four_third * erf * urf[ia] * urf[k] + one_third * erf * g.GG[ia][k];
      for (int ib = 0; ib < 4; ++ib) {
        double s = 0.0;
        for (int k = 0; k < 4; ++k) s += r[k] * g.gg[k][ib];
        rtt += -s * ucon[ib] * ucov[ia];
      }
    }
    w.startwith = (-rtt < ip.threshold * pp00[UU]) ? PRIM_RAD : PRIM_MHD;
  }
  w.ehat = rij_ehat(pp00[EE], urf, g, ucov);
  if (!ip.start_with_bisect) return w;

  const double rho = pp00[RHO];
  const double ne = thermal_ne(c, rho);
  double bsq;
  {
    double B[3] = {pp00[B1], pp00[B2], pp00[B3]}, bcon[4], bcov[4];
    bcon_bcov_bsq(B, ucon, ucov, g, bcon, bcov, bsq);
  }
  // kp::solve_1d_prim
  const double ehat0 = w.ehat;
  const double dtau = dt / ucon[0];
  const double tot = ehat0 + pp00[UU];
  const bool rad = ehat0 < 1.0e-3 * pp00[UU];  // PRIM_RAD
  const double tgas0 = tgas_of(c, pp00[UU], rho, gam);
  const double ratio = ehat0 / pp00[EE];
  const double fac = 3.0, fac1 = fac + 1.0;
  double pp_uu = pp00[UU], pp_ee = pp00[EE];
  if (tgas0 > 1.0e14) {
    pp_uu = pp00[UU] * 1.0e14 / tgas0;
    pp_ee = (tot - pp_uu) / ratio;
  }
  double xlo, xhi;
  if (!rad) {
    xlo = pp_uu / 1.05;
    xhi = kmath::fmin(pp_uu * 1.05, (pp_uu + fac * tot) / fac1);
  } else {
    xlo = pp_ee / 1.05;
    xhi = kmath::fmin(pp_ee * 1.05, (pp_ee + fac * tot / ratio) / fac1);
  }
  const double ee_ratio = pp00[EE] / ratio;
  const int maxiter = 50;
  double errlo = 0.0, errhi = 0.0, x = xlo;
  int iter = 0, phase = 0;  // 0, 1: the bracket's ends; 2, 3: a widened end; 4: a midpoint
  KC_ROLLED
  for (;;) {
    // kp::f1d_err at x (implicit.zig:431)
    double ugas, ehat_x;
    if (rad) {
      ehat_x = x * ratio;
      ugas = tot - ehat_x;
    } else {
      ugas = x;
      ehat_x = tot - ugas;
    }
    const double te = te_of(tgas_of(c, ugas, rho, gam));
    const double ehat = rij_ehat(ehat_x / ratio, urf, g, ucov);
    const double trad = lte_T_from_E(c, ehat);
    const OpacLean o = absorption<false>(op, rho, te, trad, ne, bsq);
    const double b = c.sigma_rad_over_pi * te * te * te * te;
    double gi0 = -o.gas_abs * c.fourpi * b + o.rad_abs * ehat;
    if (op.ch.comptonization) gi0 += compton(c, kappaes<true>(op, rho, trad), ehat, trad, te);
    if (op.opdamp != 1.0) gi0 *= op.opdamp;
    const double err = rad ? ehat_x - ee_ratio + dtau * gi0 : ugas - pp00[UU] - dtau * gi0;

    if (phase == 0) {
      errlo = err;
      x = xhi;
      phase = 1;
      continue;
    }
    if (phase < 4) {
      if (phase == 2) errlo = err;
      else errhi = err;
      if (phase >= 2 && (kmath::isnan(errlo) || kmath::isnan(errhi))) iter = maxiter;
      if (iter >= maxiter) return w;  // no bracket: the pre-solve state
      if (errlo * errhi > 0.0) {
        iter += 1;
        if (errlo > 0.0) {
          xhi = xlo;
          errhi = errlo;
          xlo /= fac;
          x = xlo;
          phase = 2;
        } else {
          xlo = xhi;
          errlo = errhi;
          if (rad) xhi = kmath::fmin(xhi * fac, (xhi + fac * tot / ratio) / fac1);
          else xhi = kmath::fmin(xhi * fac, (xhi + fac * tot) / fac1);
          x = xhi;
          phase = 3;
        }
        continue;
      }
      phase = 4;
    } else {
      if (err * errlo > 0.0) {
        xlo = x;
        errlo = err;
      } else {
        xhi = x;
        errhi = err;
      }
      if (kmath::isnan(x) || kmath::isnan(err)) return w;
      if (!(kmath::fabs((xhi - xlo) / x) > 1.0e-3)) break;
    }
    x = 0.5 * (xlo + xhi);
  }
  if (rad) {
    w.ee = x;
    w.uu = tot - x * ratio;
  } else {
    w.uu = x;
    w.ee = (tot - x) / ratio;
  }
  return w;
}

// ---- the Newton core (implicit.zig:642) ------------------------------------------
// What a solve keeps fixed lives in a cell object: geom() and uu0() give the
// cell's metric and reference conserveds, jac() the Jacobian's entries, ref() the
// scalars that only the later rungs and lag_opac read. A cell kept in shared
// memory (SharedCell) gives fresh loads at each call, so that the metric's 29
// numbers are not live through the whole Newton loop: the loop's registers hold
// the trial state, and nothing of it spills.
enum : int { U_RHO = 0, U_GAS = 1, U_RAD = 5, U_ENTR = 9, NU0 = 10 };  // uu0: rho, u and momenta, R^t_mu, entropy
struct RefScalars {
  double ugas, rho, ehat;  // of the pre-solve state
  double lag[4];           // lag_opac: its kappaes, gas_abs, rad_abs, rad_ross
};
struct CellGeom {
  Geom g;
  double ngtt, gdinv;  // -1 / g^tt, 1 / sqrt(-g): the quotients every trial forms
};
// Velocities of a trial that its constraints and its radiation state share
struct Kin {
  double ucon[4], ucov[4], bsq;  // gas
  double urf[4];                 // radiation frame
};

// kp::velr_to_vel4 with -1/g^tt given
KC_HD void four_velocity(double v1, double v2, double v3, const CellGeom& q, double out[4]) {
  const Geom& g = q.g;
  const double u[4] = {0.0, v1, v2, v3};
  double qsq = 0.0;
  for (int i = 1; i < 4; ++i)
    for (int j = 1; j < 4; ++j) qsq += u[i] * u[j] * g.gg[i][j];
  const double alpgam2 = q.ngtt * (1.0 + qsq);
  const double alpgam = (alpgam2 < 0.0) ? 1.0 : kmath::sqrt(alpgam2);
  out[0] = -alpgam * g.GG[0][0];
  for (int i = 1; i < 4; ++i) out[i] = u[i] - alpgam * g.GG[0][i];
}
KC_HD void gas_kin(const double pp[NV], const CellGeom& q, Kin& k, double bcon[4], double bcov[4]) {
  four_velocity(pp[VX], pp[VY], pp[VZ], q, k.ucon);
  lower_vec(k.ucon, q.g, k.ucov);
  const double B[3] = {pp[B1], pp[B2], pp[B3]};
  bcon_bcov_bsq(B, k.ucon, k.ucov, q.g, bcon, bcov, k.bsq);
}

// absorption<true> out of line, its operands by value: for lag_opac's one fill of
// the reference state
KC_HDN OpacLean absorption_call(const OpacParams& op, double rho, double te, double trad, double ne, double bsq) {
  return absorption<true>(op, rho, te, trad, ne, bsq);
}
// the reference state's opacities, for lag_opac (kp::lag_opac)
KC_HD void lag_reference(const double pp00[NV], double ehat, const Geom& g, double gam, const OpacParams& op,
                         double lag[4]) {
  double ucon[4], ucov[4], bcon[4], bcov[4], bsq, B[3] = {pp00[B1], pp00[B2], pp00[B3]};
  double vin[4] = {0.0, pp00[VX], pp00[VY], pp00[VZ]};
  velr_to_vel4(vin, g, ucon);
  lower_vec(ucon, g, ucov);
  bcon_bcov_bsq(B, ucon, ucov, g, bcon, bcov, bsq);
  const double te = te_of(tgas_of(op.c, pp00[UU], pp00[RHO], gam)), trad = lte_T_from_E(op.c, ehat);
  const OpacLean o = absorption_call(op, pp00[RHO], te, trad, thermal_ne(op.c, pp00[RHO]), bsq);
  lag[0] = kappaes_at(op, pp00[RHO], trad);
  lag[1] = o.gas_abs;
  lag[2] = o.rad_abs;
  lag[3] = o.rad_ross;
}
// What the residuals read of the pre-solve state pp00 (implicit.zig:941): its
// conserveds (NU0 of them) and, with scalars, the rest
KC_HD void reference(const double pp00[NV], double ehat, const Geom& g, double gam, const OpacParams& op,
                     const ImplicitParams& ip, double uu0[NU0], RefScalars& r, bool scalars) {
  double uu[NV];
  p2u(pp00, uu, g, gam);
  uu0[U_RHO] = uu[RHO];
  for (int k = 0; k < 4; ++k) uu0[U_GAS + k] = uu[UU + k];
  for (int k = 0; k < 4; ++k) uu0[U_RAD + k] = uu[EE + k];
  uu0[U_ENTR] = uu[ENTR];
  if (!scalars) return;
  r.ugas = pp00[UU];
  r.rho = pp00[RHO];
  r.ehat = ehat;
  if (ip.lag_opac) lag_reference(pp00, ehat, g, gam, op, r.lag);
}
// a cell held by its thread
struct LocalCell {
  CellGeom q;
  double u0[NU0], jm[16], dt_;
  RefScalars r;
  KC_HD void init(const Geom& g, double dt, const double uu0[NU0], const RefScalars& rs) {
    q.g = g;
    q.ngtt = -1.0 / g.GG[0][0];
    q.gdinv = 1.0 / g.gdet;
    for (int i = 0; i < NU0; ++i) u0[i] = uu0[i];
    r = rs;
    dt_ = dt;
  }
  KC_HD CellGeom geom() const { return q; }
  KC_HD double uu0(int i) const { return u0[i]; }
  KC_HD double gcov(int k) const { return q.g.gg[k][k]; }
  KC_HD double jac(int i, int j) const { return jm[i * 4 + j]; }
  KC_HD void set_jac(int i, int j, double v) { jm[i * 4 + j] = v; }
  KC_HD double dt() const { return dt_; }
  KC_HD RefScalars ref() const { return r; }
};

// The Newton step's matrix (implicit.zig:770-800): the Jacobian, scaled by the
// unknowns' sizes, inverted (kp::invert4, the pivot rows exchanged by selects)
// and scaled back, in the cell's jac()
template <class Cell>
KC_HD void newton_matrix(Cell& cell, double x0, int scale) {
  double lu[4][4];
  double sc0 = 1.0, is0 = 1.0;  // the other three scales are 1
  if (scale) {
    sc0 = (x0 == 0.0) ? 1.0 : x0;
    is0 = 1.0 / sc0;
  }
  int perm[4] = {0, 1, 2, 3};
  for (int i = 0; i < 4; ++i)
    for (int j = 0; j < 4; ++j) {
      lu[i][j] = cell.jac(i, j);
      // off the diagonal jac (scale_j / scale_i)
      if (scale && i != j) lu[i][j] = lu[i][j] * ((j == 0 ? sc0 : 1.0) * (i == 0 ? is0 : 1.0));
    }
KC_UNROLL
  for (int k = 0; k < 4; ++k) {
    int piv = k;
    double pmax = kmath::fabs(lu[k][k]);
KC_UNROLL
    for (int r = k + 1; r < 4; ++r)
      if (kmath::fabs(lu[r][k]) > pmax) {
        pmax = kmath::fabs(lu[r][k]);
        piv = r;
      }
KC_UNROLL
    for (int r = k + 1; r < 4; ++r)
      if (piv == r) {
KC_UNROLL
        for (int cc = 0; cc < 4; ++cc) {
          const double t = lu[k][cc];
          lu[k][cc] = lu[r][cc];
          lu[r][cc] = t;
        }
        const int tp = perm[k];
        perm[k] = perm[r];
        perm[r] = tp;
      }
KC_UNROLL
    for (int r = k + 1; r < 4; ++r) {
      lu[r][k] = lu[r][k] / lu[k][k];
KC_UNROLL
      for (int cc = k + 1; cc < 4; ++cc) lu[r][cc] -= lu[r][k] * lu[k][cc];
    }
  }
  KC_ROLLED
  for (int col = 0; col < 4; ++col) {
    double y[4], x[4];
KC_UNROLL
    for (int r = 0; r < 4; ++r) {
      y[r] = (perm[r] == col) ? 1.0 : 0.0;
KC_UNROLL
      for (int cc = 0; cc < r; ++cc) y[r] -= lu[r][cc] * y[cc];
    }
KC_UNROLL
    for (int r = 3; r >= 0; --r) {
      x[r] = y[r];
KC_UNROLL
      for (int cc = r + 1; cc < 4; ++cc) x[r] -= lu[r][cc] * x[cc];
      x[r] = x[r] / lu[r][r];
    }
KC_UNROLL
    for (int r = 0; r < 4; ++r) {
      if (scale) x[r] = x[r] * (r == 0 ? sc0 : 1.0) * (col == 0 ? is0 : 1.0);
      cell.set_jac(r, col, x[r]);
    }
  }
}

// kp::apply_constraints for the fluid PRIM (implicit.zig:240): pp and the
// conserveds uu of a trial, -2 when it is not admissible. first: no constraint
// was applied to uu before (its entropy is the reference's). Of k the gas part
// (PRIM_MHD) or the radiation frame (PRIM_RAD) is set.
template <int PRIM, class Cell>
KC_HD int constrain(const Cell& cell, double pp[NV], double uu[NV], bool first, double gam, const RadParams& rad,
                    const ImplicitParams& ip, Kin& k) {
  const CellGeom q = cell.geom();
  const Geom& g = q.g;
  const double gdetu = g.gdet;
  if (PRIM == PRIM_MHD) {
    double bcon[4], bcov[4];
    gas_kin(pp, q, k, bcon, bcov);
    pp[RHO] = cell.uu0(U_RHO) * q.gdinv / k.ucon[0];
    // the energy and the momenta of kp::p2u_mhd
    const double rho = pp[RHO], ugas = pp[UU];
    const double vcon[4] = {0.0, pp[VX], pp[VY], pp[VZ]};
    const double pre = (gam - 1.0) * ugas;
    const double w = rho + ugas + pre;
    const double eta = w + k.bsq;
    const double etap = ugas + pre + k.bsq;
    const double ptot = pre + 0.5 * k.bsq;
    const double utp1 = calc_utp1(vcon, g);
    uu[UU] = gdetu * (etap * k.ucon[0] * k.ucov[0] + rho * k.ucon[0] * utp1 + ptot - bcon[0] * bcov[0]);
    for (int i = 1; i < 4; ++i) uu[UU + i] = gdetu * (eta * k.ucon[0] * k.ucov[i] - bcon[0] * bcov[i]);
    for (int i = 0; i < 4; ++i) uu[EE + i] = cell.uu0(U_RAD + i) - (uu[UU + i] - cell.uu0(U_GAS + i));
    const U2pRadRes rr = u2p_rad_inl(uu, pp, g, rad);
    return rr.corrected ? (ip.allow_rad_ceiling ? -1 : -2) : rr.ret;
  }
  four_velocity(pp[FX], pp[FY], pp[FZ], q, k.urf);
  {
    // kp::p2u_rad
    const double four_third = 4.0 / 3.0, one_third = 1.0 / 3.0, erf = pp[EE];
    double rt[4];
    for (int i = 0; i < 4; ++i) rt[i] = four_third * erf * k.urf[0] * k.urf[i] + one_third * erf * g.GG[0][i];
    lower_vec(rt, g, rt);
    for (int i = 0; i < 4; ++i) uu[EE + i] = gdetu * rt[i];
  }
  uu[RHO] = cell.uu0(U_RHO);
  for (int i = 0; i < 4; ++i) uu[UU + i] = cell.uu0(U_GAS + i) - (uu[EE + i] - cell.uu0(U_RAD + i));
  for (int i = 0; i < 3; ++i) uu[B1 + i] = gdetu * pp[B1 + i];
  double pn[NV];
  for (int i = 0; i < NV; ++i) pn[i] = pp[i];
  int ret, etype = ETYPE_HOT;
  KC_ROLLED
  for (;;) {
    ret = u2p_w(uu, pn, g, etype, gam, false);
    if (ret >= 0 || etype == ETYPE_ENTROPY || !ip.allow_entr_in_4dprim) break;
    // the conserved entropy as the last constraint left it: that of the gas state
    // this one started from
    double ucon[4];
    four_velocity(pp[VX], pp[VY], pp[VZ], q, ucon);
    uu[ENTR] = first ? cell.uu0(U_ENTR) : entropy(pp[RHO], pp[UU], gam) * gdetu * ucon[0];
    etype = ETYPE_ENTROPY;
  }
  for (int i = 0; i < EE; ++i) pp[i] = pn[i];
  return (ret < 0) ? -2 : 0;
}
// kp::fill_rad_state of a constrained state and its residual
// (kp::implicit_residual, implicit.zig:337): f and the largest normalised error.
// k holds what the constraints of this state left. One copy for both fluids.
template <class Cell>
KC_HD double residual(const Cell& cell, bool mhd, const double pp[NV], const double uu[NV], Kin& k, double gam,
                      const OpacParams& op, double opdamp, const ImplicitParams& ip, int whicheq, int whichframe,
                      double sgas0, double f[4]) {
  const Consts& c = op.c;
  const CellGeom q = cell.geom();
  const Geom& g = q.g;
  const double gdetu = g.gdet, dt = cell.dt();
  if (mhd) {
    four_velocity(pp[FX], pp[FY], pp[FZ], q, k.urf);
  } else {
    double bcon[4], bcov[4];
    gas_kin(pp, q, k, bcon, bcov);
  }
  const double rho = pp[RHO], erf = pp[EE];
  const double tgas = tgas_of(c, pp[UU], rho, gam);
  const double te = te_of(tgas);
  const double four_third = 4.0 / 3.0, one_third = 1.0 / 3.0;
  double ehat = 0.0, ru[4];
  for (int i = 0; i < 4; ++i) {
    ru[i] = 0.0;
    for (int j = 0; j < 4; ++j) {
      const double r = four_third * erf * k.urf[i] * k.urf[j] + one_third * erf * g.GG[i][j];
      ehat += r * k.ucov[i] * k.ucov[j];
      ru[i] += r * k.ucov[j];
    }
  }
  const double trad = lte_T_from_E(c, ehat);
  double kes, kgas, krad, kross;
  if (ip.lag_opac) {
    const RefScalars r = cell.ref();
    kes = r.lag[0];
    kgas = r.lag[1];
    krad = r.lag[2];
    kross = r.lag[3];
  } else {
    kes = kappaes<false>(op, rho, trad);
    const OpacLean o = absorption<true>(op, rho, te, trad, thermal_ne(c, rho), k.bsq);
    kgas = o.gas_abs;
    krad = o.rad_abs;
    kross = o.rad_ross;
  }
  const double b = c.sigma_rad_over_pi * te * te * te * te;
  double gilab[4], gi[4];
  for (int i = 0; i < 4; ++i)
    gilab[i] = -(kross + kes) * ru[i] - ((kross + kes - krad) * ehat + kgas * c.fourpi * b) * k.ucon[i];
  double giff0 = -kgas * c.fourpi * b + krad * ehat;
  if (op.ch.comptonization) {
    const double coeff = compton(c, kes, ehat, trad, te);
    for (int i = 0; i < 4; ++i) gilab[i] += coeff * k.ucon[i];
    giff0 += coeff;
  }
  if (opdamp != 1.0) {
    for (int i = 0; i < 4; ++i) gilab[i] *= opdamp;
    giff0 *= opdamp;
  }
  lower_vec(gilab, g, gi);
  const double small = 1.0e-80;
  double u[4], u0[4];  // the fluid's energy and momenta
  KC_UNROLL
  for (int i = 0; i < 4; ++i) {
    u[i] = mhd ? uu[UU + i] : uu[EE + i];
    u0[i] = cell.uu0((mhd ? U_GAS : U_RAD) + i);
  }
  const double sg = mhd ? 1.0 : -1.0;  // a - (-x) is a + x exactly
  double err0 = 0.0, e;
  if (whichframe == FRAME_LAB) {
    const double dg = dt * gdetu * gi[0];
    f[0] = u[0] - u0[0] - sg * dg;
    e = (kmath::fabs(f[0]) > small) ? kmath::fabs(f[0]) / (kmath::fabs(u[0]) + kmath::fabs(u0[0]) + kmath::fabs(dg)) : 0.0;
  } else {
    const double dtau = dt / k.ucon[0];
    if (whicheq == EQ_ENERGY) {
      const RefScalars r = cell.ref();
      if (!mhd) {
        f[0] = ehat - r.ehat + dtau * giff0;
        e = kmath::fabs(f[0]) / (kmath::fabs(ehat) + kmath::fabs(r.ehat) + kmath::fabs(dtau * giff0));
      } else {
        f[0] = pp[UU] - r.ugas - dtau * giff0;
        e = kmath::fabs(f[0]) / (kmath::fabs(pp[UU]) + kmath::fabs(r.ugas) + kmath::fabs(dtau * giff0));
      }
    } else {
      const double s = c.kb_over_mugas_mp * entropy(rho, pp[UU], gam);
      f[0] = tgas * (s - sgas0) - dtau * giff0;
      e = kmath::fabs(f[0]) / (kmath::fabs(tgas * s) + kmath::fabs(tgas * sgas0) + kmath::fabs(dtau * giff0));
    }
  }
  err0 = (e > err0) ? e : err0;
  KC_UNROLL
  for (int i = 1; i < 4; ++i) {
    const double dg = dt * gdetu * gi[i];
    f[i] = u[i] - u0[i] - sg * dg;
    e = (kmath::fabs(f[i]) > small)
            ? kmath::fabs(f[i]) / (1.0e-20 * u[0] + kmath::fabs(u[i]) + kmath::fabs(u0[i]) + kmath::fabs(dg))
            : 0.0;
    err0 = (e > err0) ? e : err0;
  }
  return err0;
}

// The solves of a stream of cells: kp::implicit_ladder (implicit.zig:963) over
// kp::solve_4dprim_core for one cell after the other, as one loop whose every
// trip constrains one trial state of the lane's cell and, where the core reads
// it, forms its residual. A lane whose rung or cell ends goes on with the next
// at the next trip, so the lanes of a warp share the trip's code whatever rung,
// iteration, column or damped trial they are in.
// Src: bool take(Cell&, double pp[NV], int& startwith) the next cell, its start
// state in pp (false: none left); void start(const Cell&, double pp[NV]) the start
// state again; void done(Cell&, double pp[NV], const ImplicitResult&) its result
// (pp: the solution, entropy included, when ok).
template <class Src, class Cell>
KC_HD void solve_cells(Src& src, Cell& cell, double gam, const RadParams& rad, const OpacParams& op,
                       const ImplicitParams& ip) {
  const Consts& c = op.c;
  enum { BASE, COLUMN, TRIAL };
  enum { GOING, SOLVED, FAILED };
  // none for a negative number of levels; no run reaches the upper bound
  const int levels = ip.opdamp_maxlevels < 0 ? 0 : ip.opdamp_maxlevels < 1 << 28 ? ip.opdamp_maxlevels + 1 : 1 << 28;
  const int nrung = 6 * levels;
  double pp[NV], uu[NV];
  Kin kin;
  double ppp[4] = {0, 0, 0, 0}, f1[4] = {0, 0, 0, 0};
  double errbase = 0.0, sign = -1.0, del = 1.0, xiapp = 1.0, tgasold = 0.0, tradold = 0.0, sgas0 = 0.0, od = 1.0;
  int stage = BASE, iter = 0, j = 0, rungs = 0, ir = 0, startwith = PRIM_MHD;
  int whicheq = EQ_ENERGY, whichframe = FRAME_LAB;
  bool mhd = true, first = true;  // first: no constraint applied yet in this rung
  if (nrung == 0) {  // a ladder without rungs fails every cell
    const ImplicitResult none = {0, -1, 0, PRIM_RAD, EQ_ENERGY, FRAME_LAB};
    while (src.take(cell, pp, startwith)) src.done(cell, pp, none);
    return;
  }
  if (!src.take(cell, pp, startwith)) return;
  mhd = startwith == PRIM_MHD;
  KC_ROLLED
  for (;;) {
    int out = GOING;
    const int fret = mhd ? constrain<PRIM_MHD>(cell, pp, uu, first, gam, rad, ip, kin)
                         : constrain<PRIM_RAD>(cell, pp, uu, first, gam, rad, ip, kin);
    first = false;
    double x[4];  // the unknowns
    KC_UNROLL
    for (int k = 0; k < 4; ++k) x[k] = mhd ? pp[UU + k] : pp[EE + k];

    if (stage == TRIAL) {
      // ---- a damped Newton step: accept, damp further, or fail ----------------------
      bool okcheck = false;
      {
        const double edenmin = ppp[0] / ip.max_en_change_down;
        const double edenmax = ppp[0] * ip.max_en_change_up;
        if (x[0] > edenmin && x[0] < edenmax && fret >= -1) okcheck = true;
      }
      if (okcheck) {
        const double tgasnew = tgas_of(c, pp[UU], pp[RHO], gam);
        if (tgasnew > tgasold * ip.max_tgas_change || tgasnew < tgasold / ip.max_tgas_change) okcheck = false;
      }
      if (okcheck) {
        const double tradnew = lte_T_from_E(c, pp[EE]);
        if (tradnew > tradold * ip.max_trad_change || tradnew < tradold / ip.max_trad_change) okcheck = false;
      }
      if (!okcheck) {
        if (x[0] <= 0.0) {
          xiapp *= ppp[0] / (ppp[0] + kmath::fabs(x[0]));
          xiapp *= 1.0e-1;
        } else {
          xiapp /= ip.damping_factor;
        }
        if (!(xiapp >= ip.max_damping)) out = FAILED;
      } else {
        const double convrel = (whicheq == EQ_ENTROPY) ? ip.convrelentr : ip.convrel;
        const double convrelerr = (whicheq == EQ_ENTROPY) ? ip.convrelentrerr : ip.convrelerr;
        bool small = !(kmath::fabs((x[0] - ppp[0]) / ppp[0]) > convrel);
        KC_UNROLL
        for (int i = 1; i < 4; ++i)
          if (kmath::fabs((x[i] - ppp[i]) / kmath::fmax(ip.eps, kmath::fabs(ppp[i]))) > convrel) small = false;
        if (small || errbase <= convrelerr) out = SOLVED;
        else if (iter > ip.maxiter) out = FAILED;
        stage = BASE;
      }
    }
    if (stage == BASE && out == GOING) {
      iter += 1;
      KC_UNROLL
      for (int k = 0; k < 4; ++k) ppp[k] = x[k];
      tgasold = tgas_of(c, pp[UU], pp[RHO], gam);
      tradold = lte_T_from_E(c, pp[EE]);
      if (fret < -1) out = FAILED;
    }
    const bool rejected = stage == COLUMN && fret < -1;
    if (rejected) {
      if (sign > 0.0) out = FAILED;  // neither side of the column is admissible
      sign = 1.0;
    }
    if (stage != TRIAL && !rejected && out == GOING) {
      double f[4];
      const double err0 = residual(cell, mhd, pp, uu, kin, gam, op, od, ip, whicheq, whichframe, sgas0, f);
      sign = -1.0;
      if (stage == BASE) {
        errbase = err0;
        if (errbase < ((whicheq == EQ_ENTROPY) ? ip.entrconv : ip.conv)) out = SOLVED;
        KC_UNROLL
        for (int k = 0; k < 4; ++k) f1[k] = f[k];
        j = 0;
        stage = COLUMN;
      } else {
        KC_UNROLL
        for (int i = 0; i < 4; ++i) cell.set_jac(i, j, (f[i] - f1[i]) / del);
        j += 1;
        if (j == 4) {
          newton_matrix(cell, ppp[0], ip.scale_jacobian);
          xiapp = 1.0;
          stage = TRIAL;
        }
      }
    }
    if (out != GOING) {
      // ---- the rung ends: the next one, or the next cell -------------------------------
      if (out == SOLVED && iter > ip.maxiter) out = FAILED;
      rungs += 1;
      if (out == SOLVED || rungs >= nrung) {
        ImplicitResult res;
        res.ok = out == SOLVED;
        res.rung = res.ok ? ir : -1;
        res.iters = res.ok ? iter : 0;
        res.whichprim = res.ok && mhd ? PRIM_MHD : PRIM_RAD;
        res.whicheq = res.ok ? whicheq : EQ_ENERGY;
        res.whichframe = res.ok ? whichframe : FRAME_LAB;
        if (res.ok) pp[ENTR] = entropy(pp[RHO], pp[UU], gam);
        src.done(cell, pp, res);
        if (!src.take(cell, pp, startwith)) return;
        rungs = 0;
        ir = 0;
        od = 1.0;
      } else {
        src.start(cell, pp);
        ir += 1;
        if (ir == 6) {
          ir = 0;
          od /= ip.opdamp_factor;
        }
      }
      int prim;
      implicit_rung(ir, startwith, prim, whicheq, whichframe);
      mhd = prim == PRIM_MHD;
      if (whicheq == EQ_ENTROPY) {
        const RefScalars r = cell.ref();
        sgas0 = c.kb_over_mugas_mp * entropy(r.rho, r.ugas, gam);
      }
      stage = BASE;
      iter = 0;
      sign = -1.0;
      first = true;
    } else {
      // ---- the next state to constrain --------------------------------------------------
      if (stage == TRIAL) {
        KC_UNROLL
        for (int i = 0; i < 4; ++i) {
          x[i] = ppp[i];
          KC_UNROLL
          for (int k = 0; k < 4; ++k) x[i] -= xiapp * cell.jac(i, k) * f1[k];
        }
      } else {
        double pj = ppp[0], gjj = 1.0;
        KC_UNROLL
        for (int k = 1; k < 4; ++k)
          if (k == j) {
            pj = ppp[k];
            gjj = cell.gcov(k);
          }
        if (j == 0) {
          del = sign * ip.eps * pj;
        } else {
          const double veleps = ip.eps * my_sign(pj) * kmath::fmax(1.0e-8 / kmath::sqrt(gjj), kmath::fabs(pj));
          del = (pj >= 0.0) ? sign * veleps : -sign * veleps;
        }
        KC_UNROLL
        for (int k = 0; k < 4; ++k) x[k] = k == j ? pj + del : ppp[k];
      }
      KC_UNROLL
      for (int k = 0; k < 4; ++k) {
        if (mhd) pp[UU + k] = x[k];
        else pp[EE + k] = x[k];
      }
    }
  }
}

// The rung-0 residual of a start state (kp::implicit_start_residual): +1e300
// when the constraints reject it; pp becomes the constrained start
template <class Cell>
KC_HD double start_residual(const Cell& cell, double pp[NV], int prim, double gam, const RadParams& rad,
                            const OpacParams& op, const ImplicitParams& ip) {
  double uu[NV], f[4];
  Kin k;
  if (prim == PRIM_MHD) {
    if (constrain<PRIM_MHD>(cell, pp, uu, true, gam, rad, ip, k) < -1) return 1.0e300;
    return residual(cell, true, pp, uu, k, gam, op, 1.0, ip, EQ_ENERGY, FRAME_LAB, 0.0, f);
  }
  if (constrain<PRIM_RAD>(cell, pp, uu, true, gam, rad, ip, k) < -1) return 1.0e300;
  return residual(cell, false, pp, uu, k, gam, op, 1.0, ip, EQ_ENERGY, FRAME_LAB, 0.0, f);
}

}  // namespace lean
}  // namespace kc
