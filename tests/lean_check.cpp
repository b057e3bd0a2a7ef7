// Compares the engine's lean implicit solve and W inversion
// (koral-zig_b200/csrc/kc_implicit_lean.cuh, kc_u2p_lean.cuh) with the plain
// restatement (include/koral/kimplicit.h, kinvert.h) bit for bit, on the host.
// Input: cells (geom23, dt, pp), an option variant; prints the number of cells
// that differ, the number solved and a histogram of the rungs reached. A fourth
// argument names a file for the plain solve's results (pp, then the six of res).
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <vector>

#include "../include/koral/kparams.h"
#include "../koral-zig_b200/csrc/kc_fold.cuh"
#include "../koral-zig_b200/csrc/kc_implicit_lean.cuh"
#include "../koral-zig_b200/csrc/kc_init_lean.cuh"

using namespace kp;

static void geom_from_record(const double* v, Geom& g) {
  memset(&g, 0, sizeof g);
  int n = 0;
  for (int i = 0; i < 4; ++i)
    for (int j = i; j < 4; ++j) {
      g.gg[i][j] = g.gg[j][i] = v[n];
      g.GG[i][j] = g.GG[j][i] = v[10 + n];
      ++n;
    }
  g.gdet = v[20];
  g.alpha = v[21];
  g.gttpert = v[22];
}
static bool same(const double* a, const double* b, int n) {
  for (int i = 0; i < n; ++i)
    if (memcmp(&a[i], &b[i], 8) != 0 && !(a[i] != a[i] && b[i] != b[i])) return false;
  return true;
}

// bases of powers: field values, extremes and special values in turn
static double k_pow_arg(long c, const double* pp) {
  const double special[8] = {0.0, 1.0, -2.0, kmath::inf(), kmath::nan(), 1e-300, 3e200, 5e-324};
  return c % 16 == 0 ? special[(c / 16) % 8] : c % 3 == 0 ? pp[UU] : c % 3 == 1 ? pp[RHO] : pp[EE] * 1e-40;
}
// The torus functions of the column solve, and the outer bisection by outcome
// trees (its walk as the warp makes it), against the serial code
static int check_init(double a) {
  kcinit::PuffyPhysics ph;
  const kcinit::TorusConsts tc = kcinit::torus_consts(a, ph);
  const kc::lean::TorusL t = kc::lean::torus_l(a, tc.lb1, tc.lb2, ph.lt_xi);
  const kcinit::LnfIntegrand integrand = {a, tc.lb1, tc.lb2, ph.lt_xi};
  long bad = 0, n = 0;
  for (double r = 35.0; r < 499.0; r *= 1.013, ++n) {
    const double th = 0.4 + 1.1 * (double)(n % 23) / 23.0;
    const kcinit::Gd gd = kcinit::compute_gd(r, th, a);
    const double l0 = kcinit::lam_bl(r, gd, a, tc.lb1, tc.lb2, ph.lt_xi), l1 = t.lam_bl(r, gd);
    const double f0 = integrand(r), f1 = t.lnf(r);
    bad += !same(&l0, &l1, 1) + !same(&f0, &f1, 1);
    if (n % 29) continue;
    const double m0 = kcinit::find_rml(l0, a, tc.lb1, tc.lb2, ph.lt_xi);
    const double lamsq = l0 * l0, x1 = 6.0, x2 = 10.0 * lamsq;
    double dx, rtb, m1 = 0.0;
    if (t.rml_at(x1, lamsq) < 0.0) dx = x2 - x1, rtb = x1;
    else dx = x1 - x2, rtb = x2;
    bool found = false;
    for (int j = 0; j < 100 && !found; j += 5) {
      const double rtb0 = rtb, dx0 = dx;
      for (int node = 1; node < 32 && !found;) {
        dx *= 0.5;
        const double xmid = rtb + dx, xt = kc::lean::tree_midpoint(node, rtb0, dx0);
        bad += !same(&xmid, &xt, 1);
        const double fmid = t.rml_at(xt, lamsq);
        if (fmid <= 0.0) rtb = xmid;
        if (kmath::fabs(dx) < kcinit::kXacc || fmid == 0.0) found = true, m1 = rtb;
        node = 2 * node + (fmid <= 0.0);
      }
    }
    bad += !same(&m0, &m1, 1);
  }
  printf("%ld %ld\n", bad, n);
  return 0;
}

// One term beside every multiple of half an ulp (the multiple and its neighbours on
// both sides) added to a sum of either sign and parity, through the term's map and
// as an addition
static long check_fold_ties() {
  using namespace kc;
  long bad = 0;
  for (int sign = -1; sign <= 1; sign += 2)
    for (int e : {-950, -3, 0, 40, 900})
      for (int odd = 0; odd < 2; ++odd)
        for (int h = -9; h <= 9; ++h) {
          const double ulp = ldexp(1.0, e - 52), half = 0.5 * h;
          const double near[] = {half, nextafter(half, -1e9), nextafter(half, 1e9), nextafter(nextafter(half, -1e9), -1e9),
                                 nextafter(nextafter(half, 1e9), 1e9)};
          for (double x : near) {
            const double v = x * ulp, sum0 = sign * (ldexp(1.5, e) + odd * ulp);
            double sum = sum0, acc = sum0;
            sum += v;
            const long long key = fold_key(sum0);
            const FoldRun r = fold_term(v * fold_scale(key));
            const FoldChunk c = {r.m, r.lo, r.hi, r.ok ? key : 0};
            bad += !fold_apply(acc, c) || !same(&sum, &acc, 1);
          }
        }
  return bad;
}
// The ordered fold's maps, chunk by chunk, against the serial sum: sums that grow
// through binades, of one sign and of both, ties (few-bit terms), zeros, a
// non-finite term
static int check_fold() {
  using namespace kc;
  std::mt19937_64 r(3);
  long bad = check_fold_ties(), mapped = 0;
  for (int t = 0; t < 400; ++t) {
    const int kind = t % 8, chunk = 1 << (5 + t % 4);
    std::vector<double> v(2000 + r() % 20000);
    for (double& x : v) {
      const double u = (double)(r() >> 11) * 0x1p-53;
      x = kind == 0 ? u : kind == 1 ? ldexp(u, (int)(r() % 60)) : kind == 2 ? -ldexp(u, (int)(r() % 10))
          : kind == 3 ? (double)(long)(u * 1000) * 0.125 : kind == 4 ? u - 0.3 : kind == 5 ? (r() % 3 ? 0.0 : u * 1e-20)
          : kind == 6 ? ldexp((double)(1 + r() % 7), -3 + (int)(r() % 4)) : u * 1e-30 * (u < 0.001 ? 1e10 : 1.0);
    }
    if (kind == 6) v[0] = ldexp(1.0, 51 + t % 4);
    if (t % 50 == 49) v[v.size() / 2] = kmath::inf();
    double s = 0.0, acc = 0.0, est = 0.0;
    for (double x : v) s += x;
    for (size_t k0 = 0; k0 < v.size(); k0 += chunk) {
      const size_t k1 = k0 + chunk < v.size() ? k0 + chunk : v.size();
      FoldChunk c = {{0, 0}, 0, 0, 0};
      double sum = 0.0;
      if (const long long key = fold_key(est * (1.0 + 1e-14))) {
        std::vector<FoldRun> q;
        for (size_t k = k0; k < k1; ++k) q.push_back(fold_term(v[k] * fold_scale(key)));
        while (q.size() > 1) {  // joined as a tree, as the kernel does
          std::vector<FoldRun> z;
          for (size_t i = 0; i < q.size(); i += 2) z.push_back(i + 1 < q.size() ? fold_join(q[i], q[i + 1]) : q[i]);
          q = z;
        }
        c = {q[0].m, q[0].lo, q[0].hi, q[0].ok ? key : 0};
      }
      if (fold_apply(acc, c)) ++mapped;
      else
        for (size_t k = k0; k < k1; ++k) acc += v[k];
      for (size_t k = k0; k < k1; ++k) sum += v[k];
      est += sum;
    }
    bad += !same(&s, &acc, 1);
  }
  printf("%ld %ld\n", bad, mapped);
  return 0;
}

int main(int argc, char** argv) {
  if (argc == 2 && !strcmp(argv[1], "fold")) return check_fold();
  if (argc == 3 && !strcmp(argv[1], "init")) return check_init(atof(argv[2]));
  if (argc < 4) return 2;
  const long n = atol(argv[2]);
  const int variant = atoi(argv[3]);
  std::vector<double> in(n * 37);
  FILE* f = fopen(argv[1], "rb");
  if (!f || fread(in.data(), 8, in.size(), f) != in.size()) return 3;
  fclose(f);
  const double gam = variant == 9 ? 4.0 / 3.0 : 5.0 / 3.0;
  ImplicitParams ip = implicit_params_puffy();
  RadParams rp = rad_params_puffy();
  OpacParams op = opac_params_puffy();
  if (variant == 1) ip.start_with_bisect = 0;
  if (variant == 2) ip.scale_jacobian = 0;
  if (variant == 3) ip.lag_opac = 1;
  if (variant == 4) ip.allow_rad_ceiling = 0, ip.allow_entr_in_4dprim = 0;
  if (variant == 5) ip.opdamp_maxlevels = 1, ip.maxiter = 9;
  if (variant == 6) op.ch.synchrotron_bridge = 1;
  if (variant == 7) op.ch.comptonization = 0, op.ch.kleinnishina = 0;
  if (variant == 8) op.ch.synchrotron = 0, op.kappaes_mode = KAPPAES_NONE;
  if (variant == 10) op.ch.bremsstrahlung = 0, ip.maxiter = 20;
  if (variant >= 12) ip.opdamp_maxlevels = 11 - variant;  // a ladder without rungs
  if (variant == 11) ip.convrelerr = 1.0e-12, ip.convrel = 1.0e-13;  // many iterations
  long bad = 0, bad_w = 0, ok = 0, rungs[7] = {0};
  FILE* results = argc > 4 ? fopen(argv[4], "wb") : nullptr;
  for (long c = 0; c < n; ++c) {
    Geom g;
    geom_from_record(&in[c * 37], g);
    const double dt = in[c * 37 + 23];
    double pp[NV], uu[NV], pl[NV], ul[NV];
    memcpy(pp, &in[c * 37 + 24], sizeof pp);
    memcpy(pl, pp, sizeof pl);
    memset(uu, 0, sizeof uu);
    memset(ul, 0, sizeof ul);
    const double* pp00 = &in[c * 37 + 24];
    const ImplicitResult a = solve_implicit_lab(uu, pp, g, dt, gam, rp, op, ip);
    if (results) {
      const double r[6] = {(double)a.ok, (double)a.rung, (double)a.iters, (double)a.whichprim, (double)a.whicheq, (double)a.whichframe};
      fwrite(pp, 8, NV, results);
      fwrite(r, 8, 6, results);
    }
    const kc::lean::Warm w = kc::lean::warm_start(pl, g, dt, gam, op, ip);
    double uu0[kc::lean::NU0];
    kc::lean::RefScalars rs;
    kc::lean::reference(pl, w.ehat, g, gam, op, ip, uu0, rs, true);
    kc::lean::LocalCell cell;
    cell.init(g, dt, uu0, rs);
    struct Src {
      const double* pp00;
      const kc::lean::Warm* w;
      double* out;
      ImplicitResult res;
      bool given;
      void start(const kc::lean::LocalCell&, double q[NV]) {
        memcpy(q, pp00, sizeof(double) * NV);
        q[UU] = w->uu;
        q[EE] = w->ee;
      }
      bool take(kc::lean::LocalCell& cell, double q[NV], int& startwith) {
        if (given) return false;
        given = true;
        start(cell, q);
        startwith = w->startwith;
        return true;
      }
      void done(kc::lean::LocalCell&, double q[NV], const ImplicitResult& r) {
        res = r;
        memcpy(out, q, sizeof(double) * NV);
      }
    } src = {pp00, &w, pl, {}, false};
    kc::lean::solve_cells(src, cell, gam, rp, op, ip);
    const ImplicitResult b = src.res;
    if (b.ok) p2u(pl, ul, g, gam);
    else memcpy(pl, pp00, sizeof pl);
    if (memcmp(&a, &b, sizeof a) != 0 || !same(pp, pl, NV) || !same(uu, ul, NV)) {
      if (bad < 3) fprintf(stderr, "cell %ld: ok %d/%d rung %d/%d iters %d/%d\n", c, a.ok, b.ok, a.rung, b.rung, a.iters, b.iters);
      ++bad;
    }
    ok += a.ok;
    rungs[a.rung + 1] += 1;
    for (double y : {1.5, 1.0 / (gam - 1.0), 1.0 + 1.0 / (gam - 1.0), 0.3, 0.7, 1.0, 2.7, 3.2, 0.5, 2.0}) {
      const double x = k_pow_arg(c, pp00), r0 = kmath::pow(x, y), r1 = kc::lean::pow_pos(x, y);
      bad_w += !same(&r0, &r1, 1);
    }
    // the W inversion from a displaced guess, hot and entropy, and of broken conserveds
    p2u(pp00, uu, g, gam);
    for (int k = 0; k < 4; ++k) {
      double u2[NV], p1[NV], p2[NV];
      memcpy(u2, uu, sizeof u2);
      memcpy(p1, pp00, sizeof p1);
      const double h = 1.0 + 0.3 * ((double)((c * 7 + k * 13) % 17) / 17.0 - 0.5);
      p1[RHO] *= h;
      p1[UU] /= h * h;
      p1[VX] *= h;
      if (k == 2) u2[UU] = u2[RHO] * 0.3;
      if (k == 3) u2[RHO] = -u2[RHO];
      memcpy(p2, p1, sizeof p2);
      const int et = k == 1 ? ETYPE_ENTROPY : ETYPE_HOT;
      const int ra = u2p_solver_w(u2, p1, g, et, gam), rb = kc::lean::u2p_w(u2, p2, g, et, gam, true);
      if (ra != rb || !same(p1, p2, NV)) ++bad_w;
    }
  }
  if (results) fclose(results);
  printf("%ld %ld %ld", bad, bad_w, ok);
  for (long x : rungs) printf(" %ld", x);
  printf("\n");
  return 0;
}
