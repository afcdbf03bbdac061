// Device conservative-to-primitive recovery (FP64), following
// src/physics/eos/c2p.cpp:40-455, include/grace/physics/eos/c2p.hh:124-316,
// include/grace/physics/eos/kastaun_c2p.hh:44-402 and
// include/grace/physics/eos/ent_based_c2p.hh:44-260.  Root solves are
// Brent's method (Brent 1973, "zero") and the safeguarded Newton of
// include/grace/utils/rootfinding.hh:73-306.  Every loop is bounded: Brent
// by an iteration cap far above its convergence bound for the 1e-15
// abscissa tolerance, Newton by its 30-step limit.
#pragma once
#include "physics.cuh"

namespace grb {

// fatal conditions (the reference calls Kokkos::abort there) -> status bits
enum : uint32_t {
  FAT_C2P_RHO_HIGH = GRB_FLAG_C2P_RHO_TOO_HIGH, FAT_EOS_RHO_HIGH = GRB_FLAG_EOS_RHO_TOO_HIGH,
  FAT_EOS_EPS_HIGH = GRB_FLAG_EOS_EPS_TOO_HIGH, FAT_EOS_TEMP_HIGH = GRB_FLAG_EOS_TEMP_TOO_HIGH,
  FAT_EOS_PRESS_HIGH = GRB_FLAG_EOS_PRESS_TOO_HIGH
};
constexpr int kBrentMaxIter = 200;

// Brent's zero finder on [a,b] with tol = 2 eps |b| + t, given f(a) and
// f(b) already evaluated (fa0, fb0).  F: double(double).
template <class F>
GRB_HD double brent_f(F& f, double a, double b, double fa0, double fb0, double t, int& iters) {
  double sa = a, sb = b;
  double fa = fa0, fb = fb0;
  double c = sa, fc = fa, e = sb - sa, d = e;
  const double macheps = 2.220446049250313e-16;
  for (int it = 0; it < kBrentMaxIter; ++it) {
    if (fabs(fc) < fabs(fb)) {
      sa = sb; sb = c; c = sa;
      fa = fb; fb = fc; fc = fa;
    }
    const double tol = 2.0 * macheps * fabs(sb) + t;
    const double m = 0.5 * (c - sb);
    if (fabs(m) <= tol || fb == 0.0) break;
    if (fabs(e) < tol || fabs(fa) <= fabs(fb)) {
      e = m; d = e;
    } else {
      double s = fb / fa, p, q;
      if (sa == c) {
        p = 2.0 * m * s;
        q = 1.0 - s;
      } else {
        q = fa / fc;
        const double r = fb / fc;
        p = s * (2.0 * m * q * (q - r) - (sb - sa) * (r - 1.0));
        q = (q - 1.0) * (r - 1.0) * (s - 1.0);
      }
      if (0.0 < p) q = -q; else p = -p;
      s = e; e = d;
      if (2.0 * p < 3.0 * m * q - fabs(tol * q) && p < fabs(0.5 * s * q)) d = p / q;
      else { e = m; d = e; }
    }
    sa = sb; fa = fb;
    if (tol < fabs(d)) sb = sb + d;
    else if (0.0 < m) sb = sb + tol;
    else sb = sb - tol;
    fb = f(sb);
    ++iters;
    if ((0.0 < fb && 0.0 < fc) || (fb <= 0.0 && fc <= 0.0)) {
      c = sa; fc = fa; e = sb - sa; d = e;
    }
  }
  return sb;
}
template <class F>
GRB_HD double brent(F& f, double a, double b, double t, int& iters) {
  const double fa = f(a);
  const double fb = f(b);
  return brent_f(f, a, b, fa, fb, t, iters);
}

// Kastaun auxiliary function mu sqrt(h0^2 + rbar^2(mu)) - 1 (kastaun_c2p.hh:44-117)
struct KBr {
  double rsqr, bsqr, rbsqr, h0sqr;
  GRB_HD double xmu(double mu) const { return 1. / (1. + mu * bsqr); }
  GRB_HD double rb2(double mu, double x) const { return x * (rsqr * x + mu * (x + 1.0) * rbsqr); }
  GRB_HD double operator()(double mu) const {
    const double x = xmu(mu);
    return mu * sqrt(h0sqr + rb2(mu, x)) - 1.;
  }
  GRB_HD void fdf(double mu, double& f, double& df) const {
    const double x = xmu(mu), x2 = x * x;
    const double hw = sqrt(h0sqr + rb2(mu, x));
    const double b = x * (x2 * rsqr + mu * (1 + x + x2) * rbsqr);
    f = mu * hw - 1.;
    df = (h0sqr + b) / hw;
  }
};
GRB_HD double newton_br(double sa, double sb, const KBr& g, int maxiter, double tol, int& err) {
  const double macheps = 2.220446049250313e-16;
  double a = sa, b = sb, fa, fb, dum;
  g.fdf(a, fa, dum);
  g.fdf(b, fb, dum);
  if (fa == 0) { err = 0; return a; }
  if (fb == 0) { err = 0; return b; }
  if (fa * fb > 0) { err = 1; return 0; }
  double x = (fb * a - fa * b) / (fb - fa);
  for (int it = 0; it < maxiter; ++it) {
    const double xold = x;
    double fx, dfx;
    g.fdf(x, fx, dfx);
    if (fx * fb > 0) { fb = fx; b = x; }
    else if (fx * fa > 0) { fa = fx; a = x; }
    x -= fx / dfx;
    const double tt = 2. * macheps * fabs(x) + tol;
    if (fabs(x - xold) < tt || fx == 0) { err = 0; return x; }
    if (x > b || x < a) x = 0.5 * (b + a);
  }
  err = 1;
  return 0;
}

// Kastaun scalars (kastaun_c2p.hh:306-337)
struct KSc {
  double D, iD, q, s, ye, r2, Bt2, rBt, rBt2, h0, ih0;
  double rup[3], Bt[3], B[3];
};
GRB_HD KSc kscalars(const DevEos& e, const Met& m, double c[10]) {
  KSc k;
  k.h0 = e.h_min;
  k.ih0 = e.ih0;  // 1/h_min, correctly rounded on the host as 1 / k.h0 is here
  c[0] = fmax(0., c[0]);
  k.D = c[0];
  const double iD = 1.0 / k.D;
  k.iD = iD;
  k.q = c[4] * iD;
  k.s = c[6] * iD;
  const double r[3] = {c[1] * iD, c[2] * iD, c[3] * iD};
  const double isD = 1.0 / sqrt(k.D);
#pragma unroll
  for (int i = 0; i < 3; ++i) { k.B[i] = c[7 + i]; k.Bt[i] = c[7 + i] * isD; }
  k.r2 = sqs(m.gi, r);
  k.Bt2 = sqs(m.g, k.Bt);
  k.rBt = r[0] * k.Bt[0] + r[1] * k.Bt[1] + r[2] * k.Bt[2];
  k.rBt2 = k.rBt * k.rBt;
  mvs(m.gi, r, k.rup);
  k.ye = c[5] * iD;
  return k;
}

// Kastaun master function (kastaun_c2p.hh:122-295).  FAST (tuned mode): the
// same function up to rounding with three divisions per evaluation instead
// of five: rho = D sqrt(1 - v^2) and h/W = h sqrt(1 - v^2); W and
// W/(1+W) = 1/(1 + 1/W) from one reciprocal of (1/W)(1 + 1/W);
// h = (1+eps)(1+a) with a = P/(rho(1+eps)) formed as 1 + eps + P/rho, with
// 1/rho = W/D; and nu = max(nu_A, nu_B), nu_A = (1+a)(1+q-mu r^2) =
// h (1+q-mu r^2)/(1+eps), nu_B = h/W, decided by comparing
// 1+q-mu r^2 with (1+eps)/W (h, 1+eps > 0), so that 1/(nu + mu r^2) takes
// one division either way.
template <bool FAST = false>
struct KRt {
  const DevEos* e;
  double d, qtot, rsqr, bsqr, rbsqr, brosqr, vsqrmax, wmax;
  double id, iwmax, w1max;  // FAST: 1/D, 1/wmax, wmax/(1+wmax)
  GRB_HD KRt(const DevEos& eos, const KSc& k) : e(&eos) {
    d = k.D; qtot = k.q; rsqr = k.r2; bsqr = k.Bt2; rbsqr = k.rBt2;
    brosqr = rsqr * bsqr - rbsqr;
    id = iwmax = w1max = 0.0;
    if (FAST) {
      // 1/ws, 1/wmax and 1/(1 + wmax) from one reciprocal (all >= 1)
      const double zs = rsqr * (k.ih0 * k.ih0);
      const double ws = 1 + zs;
      wmax = sqrt(ws);
      const double r = 1.0 / (ws * wmax * (1 + wmax));
      vsqrmax = zs * (wmax * (1 + wmax)) * r;
      iwmax = ws * (1 + wmax) * r;
      w1max = wmax * (ws * wmax) * r;
      id = k.iD;
    } else {
      const double zs = rsqr / (k.h0 * k.h0);
      const double ws = 1 + zs;
      wmax = sqrt(ws);
      vsqrmax = zs / ws;
    }
  }
  // FAST form of eval (same arguments and results).
  GRB_HD double eval_f(double mu, bool full, uint32_t& sig, double& x, double& w, double& rho,
                       double& press, double& eps, double& temp, double& ent) const {
    x = 1. / (1. + mu * bsqr);
    const double rf = x * (rsqr * x + mu * (x + 1.0) * rbsqr);
    const double mx = mu * x;
    const double qf = qtot - 0.5 * (bsqr + mx * mx * brosqr);
    const double vsqr = rf * mu * mu;
    double iw, w1;  // 1/W and W/(1+W)
    if (vsqr > vsqrmax) {
      w = wmax;
      iw = iwmax;
      w1 = w1max;
      if (full) sig |= SIG_VEL_HIGH;
    } else {
      iw = sqrt(1 - vsqr);
      const double r = 1.0 / (iw * (1.0 + iw));
      w = (1.0 + iw) * r;
      w1 = iw * r;
    }
    rho = d * iw;
    const double rho0 = rho;
    if (full) {
      if (rho >= e->rhomax) { sig |= SIG_RHO_HIGH; rho = e->rhomax; }
      else if (rho <= e->rhomin) { sig |= SIG_RHO_LOW; rho = e->rhomin; }
    } else {
      rho = fmin(e->rhomax, fmax(e->rhomin, rho));
    }
    const double irho = rho == rho0 ? w * id : 1.0 / rho;
    eps = w * (qf - mu * rf * (1.0 - mu * w1));
    double lo, hi;
    eos_eps_range(*e, lo, hi, rho);
    uint32_t qe = 0;
    if (full) {
      hi = fmin(hi, e->eps_max);
      if (eps >= hi) { sig |= SIG_EPS_HIGH; eps = hi * 0.999; }
      else if (eps < lo) { sig |= SIG_EPS_LOW; eps = lo; }
      press = eos_Peps_full(*e, temp, ent, eps, rho, qe);
    } else {
      eps = fmin(hi, fmax(lo, eps));
      press = eos_Peps(*e, eps, rho, qe);
    }
    const double h = 1 + eps + press * irho;
    const double qa = 1 + qf - mu * rf;
    const double rmu = rf * mu;
    if (qa >= iw * (1 + eps)) return mu - (1 + eps) / (h * qa + rmu * (1 + eps));
    return mu - 1. / (h * iw + rmu);
  }
  GRB_HD double eval(double mu, bool full, uint32_t& sig, double& x, double& w, double& rho,
                     double& press, double& eps, double& temp, double& ent) const {
    if (FAST) return eval_f(mu, full, sig, x, w, rho, press, eps, temp, ent);
    x = 1. / (1. + mu * bsqr);
    const double rf = x * (rsqr * x + mu * (x + 1.0) * rbsqr);
    const double mx = mu * x;
    const double qf = qtot - 0.5 * (bsqr + mx * mx * brosqr);
    const double vsqr = rf * mu * mu;
    if (vsqr > vsqrmax) {
      w = wmax;
      if (full) sig |= SIG_VEL_HIGH;
    } else {
      w = 1 / sqrt(1 - vsqr);
    }
    rho = d / w;
    if (full) {
      if (rho >= e->rhomax) { sig |= SIG_RHO_HIGH; rho = e->rhomax; }
      else if (rho <= e->rhomin) { sig |= SIG_RHO_LOW; rho = e->rhomin; }
    } else {
      rho = fmin(e->rhomax, fmax(e->rhomin, rho));
    }
    eps = w * (qf - mu * rf * (1.0 - mu * w / (1 + w)));
    double lo, hi;
    eos_eps_range(*e, lo, hi, rho);
    uint32_t qe = 0;
    if (full) {
      hi = fmin(hi, e->eps_max);
      if (eps >= hi) { sig |= SIG_EPS_HIGH; eps = hi * 0.999; }
      else if (eps < lo) { sig |= SIG_EPS_LOW; eps = lo; }
      press = eos_Peps_full(*e, temp, ent, eps, rho, qe);
    } else {
      eps = fmin(hi, fmax(lo, eps));
      press = eos_Peps(*e, eps, rho, qe);
    }
    const double a = press / (rho * (1 + eps));
    const double h = (1 + eps) * (1 + a);
    const double hbw = fmax((1 + a) * (1 + qf - mu * rf), h / w);
    return mu - 1. / (hbw + rf * mu);
  }
  GRB_HD double operator()(double mu) const {
    uint32_t s = 0;
    double x, w, rho, p, eps, t, en;
    return eval(mu, false, s, x, w, rho, p, eps, t, en);
  }
};

// Entropy master function (ent_based_c2p.hh:44-170); s persists clamped.
struct ERt {
  const DevEos* e;
  double d, s, rsqr, bsqr, rbsqr, vsqrmax, wmax;
  GRB_HD ERt(const DevEos& eos, const KSc& k) : e(&eos) {
    d = k.D; s = k.s; rsqr = k.r2; bsqr = k.Bt2; rbsqr = k.rBt2;
    const double zs = rsqr / (k.h0 * k.h0);
    const double ws = 1 + zs;
    wmax = sqrt(ws);
    vsqrmax = zs / ws;
  }
  GRB_HD double eval(double mu, double& ent, bool full, uint32_t& sig, double& x, double& w,
                     double& rho, double& press, double& eps, double& temp) {
    x = 1. / (1. + mu * bsqr);
    const double rf = x * (rsqr * x + mu * (x + 1.0) * rbsqr);
    const double vsqr = rf * mu * mu;
    w = 1 / sqrt(1 - vsqr);
    if (vsqr > vsqrmax) { w = wmax; if (full) sig |= SIG_VEL_HIGH; }
    rho = d / w;
    if (full) {
      if (rho >= e->rhomax) { sig |= SIG_RHO_HIGH; rho = e->rhomax; }
      else if (rho <= e->rhomin) { sig |= SIG_RHO_LOW; rho = e->rhomin; }
    } else {
      rho = fmin(e->rhomax, fmax(e->rhomin, rho));
    }
    uint32_t qe = 0;
    press = eos_Pent(*e, temp, eps, ent, rho, qe);
    if (full) {
      if (qe & EOS_ENT_LOW) sig |= SIG_ENT_LOW;
      if (qe & EOS_ENT_HIGH) sig |= SIG_ENT_HIGH;
    }
    const double a = press / (rho * (1 + eps));
    const double h = (1 + eps) * (1 + a);
    return mu - 1. / (h / w + rf * mu);
  }
  GRB_HD double operator()(double mu) {
    uint32_t sg = 0;
    double x, w, rho, p, eps, t;
    return eval(mu, s, false, sg, x, w, rho, p, eps, t);
  }
};

GRB_HD double kastaun_mu0(const KSc& k) {
  double mu0 = k.ih0;  // = 1 / k.h0
  if (k.r2 >= k.h0 * k.h0) {
    KBr g{k.r2, k.Bt2, k.rBt2, k.h0 * k.h0};
    double lo = 1. / (g.h0sqr + g.rsqr);
    const double m0 = 1. / sqrt(g.h0sqr);
    double hi = 1.0 / sqrt(g.h0sqr + g.rb2(m0, g.xmu(m0)));
    lo *= (1 - 1e-10);
    hi *= (1 + 1e-10);
    if (hi <= lo) { lo = 0; hi = m0 * (1.0 + 1e-10); }
    int err;
    mu0 = newton_br(lo, hi, g, 30, 1e-10, err);
    if (err == 0) mu0 *= 1 + 1e-10;
    else mu0 = k.ih0;
  }
  return mu0;
}

// Optional learned bracket for the Kastaun solve.  mu0 (has_mu0): the plain
// bracket top already computed from the unchanged state.
struct Guess {
  bool valid;
  double lo, hi;
  double mu0;
  bool has_mu0;
};
GRB_HD Guess no_guess() { return Guess{false, 0., 0., 0., false}; }

// kastaun_c2p_t::invert (kastaun_c2p.hh:352-395).  With a learned bracket
// the unchanged Brent iteration starts from [gs.lo, gs.hi] when f changes
// sign there (the two end values are the iteration's own first two
// evaluations), and from the plain [0, mu0] otherwise.
template <bool FAST = false>
GRB_HD double kastaun_invert(const DevEos& e, const Met& m, double c[10], double pr[13],
                             uint32_t& sig, int& iters, const Guess& gs, bool& guess_used,
                             double& mu_out) {
  const KSc k = kscalars(e, m, c);
  const KRt<FAST> f(e, k);
  double mu;
  guess_used = false;
  const double mu0 = gs.has_mu0 ? gs.mu0 : kastaun_mu0(k);
  if (gs.valid) {
    const double lo = gs.lo, hi = fmin(gs.hi, mu0);
    if (hi > lo) {
      const double flo = f(lo), fhi = f(hi);
      if (flo * fhi < 0) {
        mu = brent_f(f, lo, hi, flo, fhi, 1e-15, iters);
        guess_used = true;
      }
    }
  }
  if (!guess_used) mu = brent(f, 0, mu0, 1e-15, iters);
  double x, w, rho, press, eps, temp, ent;
  const double res = f.eval(mu, true, sig, x, w, rho, press, eps, temp, ent);
  mu_out = mu;
  pr[GRB_P_EPS] = eps; pr[GRB_P_RHO] = rho; pr[GRB_P_PRESS] = press;
  pr[GRB_P_TEMP] = temp; pr[GRB_P_ENT] = ent;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    pr[GRB_P_BX + i] = k.B[i];
    pr[GRB_P_ZX + i] = w * mu * x * (k.rup[i] + mu * k.rBt * k.Bt[i]);
  }
  return fabs(res);
}

GRB_HD double entropy_invert(const DevEos& e, const Met& m, double c[10], double pr[13],
                             uint32_t& sig) {
  const KSc k = kscalars(e, m, c);
  double mu0 = 1 / k.h0;
  int it = 0;
  if (k.r2 >= k.h0 * k.h0) {
    KBr g{k.r2, k.Bt2, k.rBt2, k.h0 * k.h0};
    int rerr;
    mu0 = newton_br(0, 1. / k.h0, g, 30, 1e-10, rerr);
    if (rerr == 0) mu0 *= 1 + 1e-10;
    else mu0 = brent(g, 0, 1. / k.h0, 1e-10, it) * (1 + 1e-10);
  }
  ERt f(e, k);
  const double mu = brent(f, 0, mu0, 1e-15, it);
  double x, w, rho, press, eps, temp;
  double ent = f.s;
  const double res = f.eval(mu, ent, true, sig, x, w, rho, press, eps, temp);
  pr[GRB_P_EPS] = eps; pr[GRB_P_RHO] = rho; pr[GRB_P_PRESS] = press;
  pr[GRB_P_TEMP] = temp; pr[GRB_P_ENT] = ent;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    pr[GRB_P_BX + i] = k.B[i];
    pr[GRB_P_ZX + i] = w * mu * x * (k.rup[i] + mu * k.rBt * k.Bt[i]);
  }
  return fabs(res);
}

// prims -> densitized cons (c2p.cpp:416-455)
GRB_HD void prims_to_cons(const double pr[13], double c[10], const Met& m) {
  const double W = lorentz(m.g, pr + GRB_P_ZX);
  double b[4], b2;
  comoving_b(m.alp, m.beta, m.g, pr + GRB_P_BX, pr + GRB_P_ZX, W, b, b2);
  const double rhoh = pr[GRB_P_RHO] * (1. + pr[GRB_P_EPS]) + pr[GRB_P_PRESS] + b2;
  const double pstar = pr[GRB_P_PRESS] + 0.5 * b2;
  double bl[3], betal[3], zl[3];
  mvs(m.g, b + 1, bl);
  mvs(m.g, m.beta, betal);
  mvs(m.g, pr + GRB_P_ZX, zl);
  const double D = pr[GRB_P_RHO] * W;
  const double tau = rhoh * W * W - pstar - m.alp * m.alp * b[0] * b[0] - D;
  c[0] = m.sqrtg * D;
#pragma unroll
  for (int i = 0; i < 3; ++i) c[1 + i] = m.sqrtg * (rhoh * W * zl[i] - m.alp * b[0] * (bl[i] + betal[i] * b[0]));
  c[4] = m.sqrtg * tau;
  c[6] = m.sqrtg * (pr[GRB_P_ENT] * D);
  c[5] = c[0] * pr[GRB_P_YE];
}

// Lorentz factor and comoving-field scalars of one set of primitives (tuned
// mode), kept while z and B stay unchanged: z2 = z_i z^i, W = sqrt(1 + z2),
// Bz = B^i z_i, b^2 = (B_i B^i + Bz^2) / W^2 (comoving_b's b^2).
struct WB {
  double z2, W, iW, Bz, b2;
};
GRB_HD WB wb_of(const Met& m, const double pr[13]) {
  WB o;
  double zl[3];
  mvs(m.g, pr + GRB_P_ZX, zl);
  const double* z = pr + GRB_P_ZX;
  const double* B = pr + GRB_P_BX;
  o.z2 = z[0] * zl[0] + z[1] * zl[1] + z[2] * zl[2];
  o.iW = rsqrt(1. + o.z2);  // 1/W; W = (1 + z^2) / W without a square root
  o.W = (1. + o.z2) * o.iW;
  o.Bz = B[0] * zl[0] + B[1] * zl[1] + B[2] * zl[2];
  o.b2 = (sqs(m.g, B) + o.Bz * o.Bz) * o.iW * o.iW;
  return o;
}
GRB_HD void handle_sig(uint32_t sig, bool lenient, uint32_t& err, uint32_t& fatal) {
  if (sig & SIG_RHO_HIGH) {
    err |= ERR_SIG_RHO_HIGH | ERR_ALL_RESETS;
    if (!lenient) fatal |= FAT_C2P_RHO_HIGH;
  }
  if (sig & SIG_RHO_LOW)
    err |= ERR_RESET_DENS | ERR_RESET_TAU | ERR_RESET_STILDE | ERR_RESET_ENTROPY | ERR_SIG_RHO_LOW;
  if (sig & SIG_ENT_LOW) err |= ERR_RESET_ENTROPY | ERR_SIG_ENT_LOW;
  if (sig & SIG_ENT_HIGH) err |= ERR_RESET_ENTROPY | ERR_SIG_ENT_HIGH;
  if (sig & SIG_EPS_HIGH) err |= ERR_RESET_STILDE | ERR_RESET_TAU | ERR_SIG_EPS_HIGH;
  if (sig & SIG_EPS_LOW) err |= ERR_RESET_STILDE | ERR_RESET_TAU | ERR_SIG_EPS_LOW;
  if (sig & SIG_VEL_HIGH)
    err |= ERR_RESET_DENS | ERR_RESET_TAU | ERR_RESET_STILDE | ERR_RESET_ENTROPY | ERR_SIG_VEL_HIGH;
  if (sig & SIG_SIGMA_HIGH)
    err |= ERR_RESET_DENS | ERR_RESET_TAU | ERR_RESET_STILDE | ERR_RESET_ENTROPY | ERR_SIG_SIGMA_HIGH;
}
GRB_HD void handle_eos_sig(uint32_t q, bool lenient, uint32_t& err, uint32_t& fatal) {
  if (q & EOS_RHO_HIGH) { err |= ERR_SIG_RHO_HIGH; fatal |= FAT_EOS_RHO_HIGH; }
  if (q & EOS_RHO_LOW)
    err |= ERR_RESET_DENS | ERR_RESET_TAU | ERR_RESET_STILDE | ERR_RESET_ENTROPY | ERR_SIG_RHO_LOW;
  if (q & EOS_ENT_HIGH) err |= ERR_RESET_ENTROPY | ERR_SIG_ENT_HIGH;
  if (q & EOS_ENT_LOW) err |= ERR_RESET_ENTROPY | ERR_SIG_ENT_LOW;
  if (q & EOS_EPS_HIGH) { err |= ERR_SIG_EPS_HIGH | ERR_RESET_STILDE | ERR_RESET_TAU; if (!lenient) fatal |= FAT_EOS_EPS_HIGH; }
  if (q & EOS_EPS_LOW) err |= ERR_RESET_STILDE | ERR_RESET_TAU | ERR_SIG_EPS_LOW;
  if (q & EOS_TEMP_HIGH) { err |= ERR_SIG_TEMP_HIGH | ERR_RESET_STILDE | ERR_RESET_TAU; if (!lenient) fatal |= FAT_EOS_TEMP_HIGH; }
  if (q & EOS_TEMP_LOW) err |= ERR_RESET_STILDE | ERR_RESET_TAU | ERR_SIG_TEMP_LOW;
  if (q & EOS_PRESS_HIGH) { err |= ERR_SIG_PRESS_HIGH | ERR_RESET_STILDE | ERR_RESET_TAU; if (!lenient) fatal |= FAT_EOS_PRESS_HIGH; }
  if (q & EOS_PRESS_LOW) err |= ERR_RESET_STILDE | ERR_RESET_TAU | ERR_SIG_PRESS_LOW;
}

GRB_HD void reset_atmo(double c[10], double pr[13], const Met& m, const DevParams& P,
                       uint32_t& err) {
  pr[GRB_P_RHO] = P.rho_fl;
  pr[GRB_P_YE] = P.ye_fl;
  pr[GRB_P_TEMP] = P.temp_fl;
  pr[GRB_P_ZX] = pr[GRB_P_ZY] = pr[GRB_P_ZZ] = 0.;
  double cs2;
  uint32_t q = 0;
  pr[GRB_P_PRESS] = eos_PT(P.eos, pr[GRB_P_EPS], cs2, &pr[GRB_P_ENT], pr[GRB_P_TEMP], pr[GRB_P_RHO], q);
  prims_to_cons(pr, c, m);
  err |= ERR_ALL_RESETS | ERR_ATMO;
}

struct C2POut {
  uint32_t err;
  uint32_t fatal;
  int iters;
  bool floored;
  bool guess_used;
  double mu;  // Kastaun root, 0 where the Kastaun solve did not run
  double W, iW;  // Lorentz factor of the final primitives (tuned mode)
};

// conservs_to_prims (c2p.cpp:188-414), in three parts (c2p_front: up to the
// decision to distrust the Kastaun result; c2p_backup: the entropy-based
// solve; c2p_back: signals, atmosphere, temperature floor, limit_primitives,
// prims_to_cons).  c2p() runs the three in sequence: the reference's order of
// operations.  c: densitized cons with densitized cell-centred B (in),
// re-densitized consistent cons (out).  FAST (the tuned mode's learned
// bracket; its plain bracket takes c2p_front_f below): multiplications by
// 1/sqrt(gamma) and 1/D where the reference divides repeatedly by the same
// value, the FAST master function, and W, b^mu, b^2 formed once per set of
// primitives (WB) instead of in each of the beta test, limit_primitives and
// prims_to_cons; equal to the reference's operations up to rounding.
struct C2PState {
  C2POut o;
  uint32_t ret;
  bool failed, lenient, ran, backup, done;
  WB wb;
  bool wb_ok;  // wb belongs to the current z and B
  // c2p_front_f: the top of the Kastaun bracket (0: not formed), and whether
  // prims' entropy is set (otherwise that slot holds the thermal energy, from
  // which c2p_back_f forms it)
  double mu0;
  bool ent_ok;
};

template <bool FAST = false>
GRB_HD C2PState c2p_front(double c[10], double pr[13], const Met& m, const DevParams& P, bool dry_run,
                          double alp_bh_thresh, const Guess& gs) {
  C2PState F{};
  F.o = C2POut{0u, 0u, 0, false, false, 0.0, 0.0, 0.0};
  F.wb_ok = false;
  F.ent_ok = true;
  F.failed = false;
  F.ret = 0;
  const DevEos& e = P.eos;
  C2POut& o = F.o;
  o.err = ERR_RESET_ENTROPY;
  const double isg = FAST ? 1.0 / m.sqrtg : 0.0;
#pragma unroll
  for (int v = 0; v < 10; ++v) c[v] = FAST ? c[v] * isg : c[v] / m.sqrtg;
  pr[GRB_P_BX] = c[7]; pr[GRB_P_BY] = c[8]; pr[GRB_P_BZ] = c[9];
  if (c[0] < 0) {
    reset_atmo(c, pr, m, P, o.err);
    o.floored = true;
    F.done = true;
    return F;
  }
  const double iD0 = FAST ? 1.0 / c[0] : 0.0;
  pr[GRB_P_YE] = FAST ? c[5] * iD0 : c[5] / c[0];
  if (pr[GRB_P_YE] > e.yemax) { pr[GRB_P_YE] = e.yemax; o.err |= ERR_RESET_YE; }
  if (pr[GRB_P_YE] < 0.0) { pr[GRB_P_YE] = 0.0; o.err |= ERR_RESET_YE; }
  F.lenient = m.alp < alp_bh_thresh;
  {  // limit_conservatives (c2p.cpp:117-157)
    double lo, hi;
    eos_eps_range(e, lo, hi, c[0]);
    const double B2 = sqs(m.g, c + 7);
    if ((FAST ? c[4] * iD0 - 0.5 * B2 * iD0 : c[4] / c[0] - 0.5 * B2 / c[0]) < fmin(0.0, lo)) {
      c[4] = lo * c[0] + 0.5 * B2;
      o.err |= ERR_RESET_TAU;
      o.floored = true;
    }
    const double qd = (FAST ? c[4] * iD0 : c[4] / c[0]) + 1;
    const double st2 = FAST ? sqs(m.gi, c + 1) * (iD0 * iD0) : sqs(m.gi, c + 1) / (c[0] * c[0]);
    if (st2 > qd * qd) {
      const double f = sqrt(qd * qd / st2);
      c[1] *= f; c[2] *= f; c[3] *= f;
      o.err |= ERR_RESET_STILDE;
      o.floored = true;
    }
  }
  if (o.floored && dry_run) {
    F.done = true;
    return F;
  }
  if (c[0] >= P.rho_fl * (1 + P.atmo_tol)) {
    F.ran = true;
    Guess g2 = gs;
    if (o.floored) g2.has_mu0 = false;  // limit_conservatives changed the state
    const double res = kastaun_invert<FAST>(e, m, c, pr, F.ret, o.iters, g2, o.guess_used, o.mu);
    F.failed = (fabs(res) > P.tol) || (F.ret & SIG_RHO_HIGH) || (F.ret & SIG_EPS_HIGH) || !isfinite(res);
    if (dry_run) return F;  // no backup in a dry run: beta is not needed
    double beta;
    if (FAST) {
      F.wb = wb_of(m, pr);
      F.wb_ok = true;
      beta = 2.0 * pr[GRB_P_PRESS] / fmax(F.wb.b2, 1e-50);
    } else {
      const double W = lorentz(m.g, pr + GRB_P_ZX);
      double b[4], b2;
      comoving_b(m.alp, m.beta, m.g, pr + GRB_P_BX, pr + GRB_P_ZX, W, b, b2);
      beta = 2.0 * pr[GRB_P_PRESS] / fmax(b2, 1e-50);
    }
    const bool distrust = F.failed || (F.ret & SIG_EPS_LOW) || (beta <= P.beta_fallback);
    F.backup = distrust && P.use_ent_backup && !dry_run;
  } else {
    F.failed = true;
  }
  return F;
}

// The entropy-based backup of a distrusted Kastaun result (c2p.cpp:262-290).
GRB_HD void c2p_backup(C2PState& F, double c[10], double pr[13], const Met& m, const DevParams& P) {
  double save[13];
#pragma unroll
  for (int v = 0; v < 13; ++v) save[v] = pr[v];
  uint32_t bret = 0;
  const double rb = entropy_invert(P.eos, m, c, pr, bret);
  const bool ok = (fabs(rb) <= P.tol) && isfinite(rb) && (pr[GRB_P_EPS] < P.eos.eps_max);
  if (ok) {
    F.ret = bret;
    F.failed = false;
    F.o.err |= ERR_ENT_BACKUP;
    F.wb_ok = false;
  } else if (!F.failed) {
#pragma unroll
    for (int v = 0; v < 13; ++v) pr[v] = save[v];
  } else {
    F.wb_ok = false;
  }
}

// kDry: a dry run (the FOFC flag's), which needs only o.floored: the final
// prims_to_cons is skipped.
template <bool kDry = false>
GRB_HD void c2p_back(C2PState& F, double c[10], double pr[13], const Met& m, const DevParams& P, double r_sph) {
  const DevEos& e = P.eos;
  C2POut& o = F.o;
  if (F.ran) {
    const uint32_t ret = F.ret;
    if (ret & (SIG_EPS_HIGH | SIG_RHO_LOW | SIG_RHO_HIGH | SIG_VEL_HIGH)) o.floored = true;
    if (e.kind == GRB_EOS_IDEAL_GAS && (ret & SIG_EPS_LOW)) o.floored = true;
    handle_sig(ret, F.lenient, o.err, o.fatal);
  }
  const bool excise = P.excise_by_radius ? (r_sph <= P.r_ex) : (m.alp <= P.alp_ex);
  if (F.failed || excise || pr[GRB_P_RHO] < (1. + P.atmo_tol) * P.rho_fl) {
    reset_atmo(c, pr, m, P, o.err);
    o.floored = true;
  } else if (pr[GRB_P_TEMP] < P.temp_fl) {
    pr[GRB_P_TEMP] = P.temp_fl;
    double cs2;
    uint32_t q = 0;
    pr[GRB_P_PRESS] = eos_PT(e, pr[GRB_P_EPS], cs2, &pr[GRB_P_ENT], pr[GRB_P_TEMP], pr[GRB_P_RHO], q);
    handle_eos_sig(q, F.lenient, o.err, o.fatal);
    o.err |= ERR_RESET_TAU | ERR_RESET_STILDE | ERR_RESET_ENTROPY | ERR_T_FLOORED;
    if (e.kind == GRB_EOS_IDEAL_GAS) o.floored = true;
  } else {  // limit_primitives (c2p.cpp:63-115)
    uint32_t s2 = 0;
    const double z2max = P.max_w * P.max_w - 1.;
    const double z2 = sqs(m.g, pr + GRB_P_ZX);
    if (z2 >= z2max) {
      const double zn = 0.99 * sqrt(z2max / z2);
      pr[GRB_P_ZX] *= zn; pr[GRB_P_ZY] *= zn; pr[GRB_P_ZZ] *= zn;
      s2 |= SIG_VEL_HIGH;
    }
    const double W = lorentz(m.g, pr + GRB_P_ZX);
    double b[4], b2;
    comoving_b(m.alp, m.beta, m.g, pr + GRB_P_BX, pr + GRB_P_ZX, W, b, b2);
    const double sigma = b2 / pr[GRB_P_RHO];
    if (sigma >= P.max_sigma) {
      pr[GRB_P_RHO] *= 1.001 * sigma / P.max_sigma;
      double cs2;
      uint32_t q = 0;
      pr[GRB_P_PRESS] = eos_PT(e, pr[GRB_P_EPS], cs2, &pr[GRB_P_ENT], pr[GRB_P_TEMP], pr[GRB_P_RHO], q);
      s2 |= SIG_SIGMA_HIGH;
    }
    handle_sig(s2, F.lenient, o.err, o.fatal);
    if (s2 & (SIG_VEL_HIGH | SIG_SIGMA_HIGH)) o.floored = true;
  }
  if (!kDry) prims_to_cons(pr, c, m);
}

GRB_HD C2POut c2p(double c[10], double pr[13], const Met& m, const DevParams& P, double r_sph,
                  bool dry_run, double alp_bh_thresh, const Guess& gs) {
  C2PState F = c2p_front(c, pr, m, P, dry_run, alp_bh_thresh, gs);
  if (F.done) return F.o;
  if (F.backup) c2p_backup(F, c, pr, m, P);
  c2p_back(F, c, pr, m, P, r_sph);
  return F.o;
}
// The FOFC flag's dry run (c2p.cpp:188-414 with the dry-run flag): whether
// the state would be floored; no entropy backup, no final prims_to_cons.
GRB_HD bool c2p_floored(double c[10], double pr[13], const Met& m, const DevParams& P, double r_sph) {
  C2PState F = c2p_front(c, pr, m, P, true, 1e30, no_guess());
  if (F.done) return F.o.floored;
  c2p_back<true>(F, c, pr, m, P, r_sph);
  return F.o.floored;
}

// ---- the c2p of the tuned mode ----------------------------------------------
// The same functions and decisions as c2p_front, c2p_backup and c2p_back
// above, equal up to rounding, arranged for the GPU.  What bound the direct
// form was not FP64 throughput (27 % of the pipe) but instruction count and
// fetch: the master function inlined at each of its call sites, every
// division and root with its slow-path branch, min/max sequences, the
// transcendental calls of three equation-of-state branches.  Here
//  - each root solve evaluates its function at one place;
//  - the function's quotients and roots are rcp_f, rsqrt_f: W = rsqrt(1 - v^2),
//    W/(1+W) = 1/(1 + 1/W), P/rho without rho for the ideal gas;
//  - the Kastaun scalars are formed once, limit_conservatives' among them, and
//    B.z = W mu (r.B), so W, B.z and b^2 of the solution need no contraction;
//  - the primitives' replacements (atmosphere, temperature floor,
//    magnetisation limit) share one equation-of-state evaluation, and the
//    entropy is formed once, at the end.

// Scalars of one state (kastaun_c2p.hh:306-337): D, 1/D, D^(-1/2), q = tau/D,
// r^2, b^2 = B^2/D, (r.b)^2 and r^2 b^2 minus it, r.b.
struct KScF {
  double D, iD, isD, q, r2, b2, rb2, bro, rBt;
  double ow, vmax;  // 1 - v_max^2 = 1 / (1 + r^2 / h0^2), v_max^2
};
// Quotients and root are correctly rounded, in the reference's order, for the
// plain mode's iterates (W^2 / f', 10^5 in fast magnetised flows, amplifies
// their rounding in the primitives).
GRB_HD void kscf(const DevEos& e, const Met& m, const double c[10], KScF& k) {
  k.D = c[0];
  k.iD = 1.0 / k.D;
  k.q = c[4] * k.iD;
  const double isD = 1.0 / sqrt(k.D);
  double r[3], Bt[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) { r[i] = c[1 + i] * k.iD; Bt[i] = c[7 + i] * isD; }
  k.r2 = sqs(m.gi, r);
  k.b2 = sqs(m.g, Bt);
  k.rBt = r[0] * Bt[0] + r[1] * Bt[1] + r[2] * Bt[2];
  k.rb2 = k.rBt * k.rBt;
  k.bro = k.r2 * k.b2 - k.rb2;
  k.isD = isD;
  // v^2 is compared with v_max^2 itself: cold flows lie within rounding of it,
  // which 1 - v^2 would lose
  const double zs = k.r2 * (e.ih0 * e.ih0);
  k.vmax = zs / (1.0 + zs);
  k.ow = rcp_f(1.0 + zs);
}

// What a root solve and the primitives from it need of a state: the scalars,
// r^i and the entropy D s / D.  The conservatives and the metric are dead
// across the solve (the few states that need the metric again get it from a
// functor that reloads it), which is what keeps the solve's registers few.
struct C2PLive {
  KScF k;
  double rup[3], s;
};
GRB_HD void c2p_live(const DevEos& e, const Met& m, const double c[10], C2PLive& L) {
  kscf(e, m, c, L.k);
  mvs(m.gi, c + 1, L.rup);
#pragma unroll
  for (int i = 0; i < 3; ++i) L.rup[i] *= L.k.iD;
  L.s = c[6] * L.k.iD;
}

// Cold part of the hybrid EOS at rho: P_cold / rho and eps_cold.
GRB_HD void pw_cold_f(const DevEos& e, double& rho, double irho, double& pr, double& ec) {
  const int i = pw_idx(e, rho);
  pr = e.G[i] == 2.0 ? e.K[i] * rho : e.K[i] * pw_pow(rho, e.G[i]) * irho;
  ec = e.E[i] + pr * e.iGm1[i];
}
GRB_HD double clamp_f(double x, double lo, double hi) {
  // as fmin(hi, fmax(lo, x)): the bound for a NaN
  x = x > lo ? x : lo;
  return x < hi ? x : hi;
}

// Kastaun's master function at mu (kastaun_c2p.hh:122-295); the members
// keep what the solution needs.  raw: eps before its clamps; eth: eps -
// eps_cold (hybrid) or eps (ideal gas); prho: P / rho.
struct KFn {
  const DevEos* e;
  const KScF* k;
  double x, w, iw, rho, eps, raw, lo, eth, prho;
  bool vhigh;
  GRB_HD double operator()(double mu) {
    x = rcp_f(1. + mu * k->b2);
    const double rf = x * (k->r2 * x + mu * (x + 1.0) * k->rb2);
    const double mx = mu * x;
    const double qf = k->q - 0.5 * (k->b2 + mx * mx * k->bro);
    const double rmu = rf * mu;
    const double vsqr = rmu * mu;
    vhigh = vsqr > k->vmax;
    const double om = vhigh ? k->ow : 1. - vsqr;
    w = rsqrt_f(om);
    iw = om * w;
    raw = w * (qf - rmu * (1.0 - mu * rcp_f(1.0 + iw)));
    rho = k->D * iw;
    if (e->kind == GRB_EOS_IDEAL_GAS) {
      lo = 0.0;
      eps = clamp_f(raw, 0.0, e->eps_max);
      eth = eps;
      prho = e->gm1 * eps;
    } else {
      double irho = w * k->iD, pr, ec;
      if (rho > e->rhomax || rho < e->rhomin) irho = rcp_f(clamp_f(rho, e->rhomin, e->rhomax));
      double r = clamp_f(rho, e->rhomin, e->rhomax);
      pw_cold_f(*e, r, irho, pr, ec);
      lo = ec < e->eps_max ? ec : e->eps_max;
      eps = clamp_f(raw, lo, e->eps_max);
      eth = eps - ec;
      prho = pr + eth * e->gthm1;
    }
    const double h = 1. + eps + prho, e1 = 1. + eps;
    const double qa = 1. + qf - rmu;
    // nu = max(h qa / (1 + eps), h / W)
    const bool a = qa >= iw * e1;
    const double num = a ? e1 : 1.0;
    return mu - num * rcp_f(h * (a ? qa : iw) + rmu * num);
  }
  GRB_HD void clamp() {}
};

// The entropy-based master function at mu (ent_based_c2p.hh:44-170) with
// the thermal energy eth = exp(Gamma' (s + log rho)), Gamma' = Gamma - 1 or
// Gamma_th - 1: with s + log D in sl and log(rho/D) = log(1 - v^2)/2, one
// logarithm and one exponential an evaluation.
struct EFn {
  const DevEos* e;
  const KScF* k;
  double sl, g, elo;  // elo: the least thermal energy
  double x, w, iw, rho, eps, eth, raw, hi, prho;
  bool vhigh;
  GRB_HD double operator()(double mu) {
    x = rcp_f(1. + mu * k->b2);
    const double rf = x * (k->r2 * x + mu * (x + 1.0) * k->rb2);
    const double rmu = rf * mu;
    const double vsqr = rmu * mu;
    vhigh = vsqr > k->vmax;
    const double om = vhigh ? k->ow : 1. - vsqr;
    w = rsqrt_f(om);
    iw = om * w;
    rho = k->D * iw;
    double lr = 0.5 * log(om), pr = 0.0, ec = 0.0, r = rho, irho = w * k->iD;
    if (rho > e->rhomax || rho < e->rhomin) {
      r = clamp_f(rho, e->rhomin, e->rhomax);
      irho = rcp_f(r);
      lr = log(r * k->iD);
    }
    if (e->kind != GRB_EOS_IDEAL_GAS) pw_cold_f(*e, r, irho, pr, ec);
    raw = exp(g * (sl + lr));
    hi = e->eps_max - ec;
    eth = raw > elo ? raw : elo;
    eth = eth < hi ? eth : hi;
    eps = ec + eth;
    prho = pr + eth * g;
    return mu - rcp_f((1. + eps + prho) * iw + rmu);
  }
  // keeps s in its range at the density last visited
  GRB_HD void clamp() {
    if (eth != raw) sl = log(eth) / g + log(k->D) - log(clamp_f(rho, e->rhomin, e->rhomax));
  }
};

// brent() from [0, top] with f evaluated at one place, and once more at the
// root where that was not the last point, so that f's members belong to it.
// The iterates are the plain mode's, so the root is the plain solve's own, to
// the last place in most states, where two converged solvers differ by
// Brent's 1e-15.  It ends only with f's two signs within the tolerance of each
// other: in fast flows f at the bracket's top lies below its own rounding,
// which W^2 amplifies, although the root is a factor away, so neither a small
// |f| nor a small step tells a root.  (A secant iteration that stopped on
// those took 3.1 evaluations instead of 6 on the blast wave's states and 4 to
// 8 % less time a step, and returned the bracket's top for 7 in 1000 states of
// an ideal gas of Gamma = 2 with eps to 1e4.)
template <class Fn>
GRB_HD double brent_root(Fn& f, double top, bool clamp, int& iters, double& res) {
  const double macheps = 2.220446049250313e-16;
  double sa = 0.0, sb = 0.0, fa = 0.0, fb = 0.0, c = 0.0, fc = 0.0, e = 0.0, d = 0.0;
  bool last = false;
  for (int it = -2;; ++it) {
    const double x = sb, fx = f(x);
    res = fx;
    if (last) break;
    if (it < 0 && clamp) f.clamp();
    if (it == -2) {
      fa = fx;
      sb = top;
      continue;
    }
    fb = fx;
    if (it == -1) {
      c = sa; fc = fa; e = sb - sa; d = e;
    } else {
      ++iters;
      if ((0.0 < fb && 0.0 < fc) || (fb <= 0.0 && fc <= 0.0)) {
        c = sa; fc = fa; e = sb - sa; d = e;
      }
    }
    if (fabs(fc) < fabs(fb)) {
      sa = sb; sb = c; c = sa;
      fa = fb; fb = fc; fc = fa;
    }
    const double tol = 2.0 * macheps * fabs(sb) + 1e-15;
    const double m = 0.5 * (c - sb);
    if (fabs(m) <= tol || fb == 0.0 || it >= kBrentMaxIter) {
      if (it >= 0 && sb == x) break;  // (at the ends f.clamp() followed)
      last = true;
      continue;
    }
    if (fabs(e) < tol || fabs(fa) <= fabs(fb)) {
      e = m; d = e;
    } else {
      const double ifa = rcp_f(fa);
      double s = fb * ifa, p, q;
      if (sa == c) {
        p = 2.0 * m * s;
        q = 1.0 - s;
      } else {
        const double ifc = rcp_f(fc);
        q = fa * ifc;
        const double r = fb * ifc;
        p = s * (2.0 * m * q * (q - r) - (sb - sa) * (r - 1.0));
        q = (q - 1.0) * (r - 1.0) * (s - 1.0);
      }
      if (0.0 < p) q = -q; else p = -p;
      s = e; e = d;
      if (2.0 * p < 3.0 * m * q - fabs(tol * q) && p < fabs(0.5 * s * q)) d = p * rcp_f(q);
      else { e = m; d = e; }
    }
    sa = sb; fa = fb;
    if (tol < fabs(d)) sb = sb + d;
    else if (0.0 < m) sb = sb + tol;
    else sb = sb - tol;
  }
  return sb;
}

// kastaun_mu0 (kastaun_c2p.hh:355-369): 1/h0, or for r >= h0 the root of
// mu sqrt(h0^2 + rbar^2(mu)) = 1 by newton_br's iteration from the same
// bracket, the auxiliary function evaluated at one place.
GRB_HD double mu0_f(const DevEos& e, const KScF& k) {
  const double h02 = e.h_min * e.h_min;
  if (!(k.r2 >= h02)) return e.ih0;
  double a = 0.0, b = 0.0, fa = 0.0, fb = 0.0, x = e.ih0, xold = 0.0, mu0 = e.ih0;
  for (int it = -3; it < 30; ++it) {
    const double xx = rcp_f(1. + x * k.b2), x2 = xx * xx;
    const double u = h02 + xx * (k.r2 * xx + x * (xx + 1.0) * k.rb2);
    const double ihw = rsqrt_f(u);
    if (it == -3) {  // the bracket
      a = rcp_f(h02 + k.r2) * (1 - 1e-10);
      b = ihw * (1 + 1e-10);
      if (b <= a) { a = 0.0; b = e.ih0 * (1.0 + 1e-10); }
      x = a;
      continue;
    }
    const double f = x * (u * ihw) - 1.;
    if (it == -2) {
      fa = f;
      x = b;
      continue;
    }
    if (it == -1) {
      fb = f;
      if (fa * fb > 0) break;
      x = (fb * a - fa * b) * rcp_f(fb - fa);
      continue;
    }
    const double df = (h02 + xx * (x2 * k.r2 + x * (1 + xx + x2) * k.rb2)) * ihw;
    xold = x;
    if (f * fb > 0) { fb = f; b = x; }
    else if (f * fa > 0) { fa = f; a = x; }
    x -= f * rcp_f(df);
    if (fabs(x - xold) < 2. * 2.220446049250313e-16 * fabs(x) + 1e-10 || f == 0) {
      mu0 = x * (1 + 1e-10);
      break;
    }
    if (x > b || x < a) x = 0.5 * (b + a);
  }
  return mu0;
}

// Writes the primitives of a solution (Kastaun's or the entropy's; prims'
// B set) and its W, B.z and b^2; met(): the state's metric, for the velocity
// limit, where they come from the primitives.
template <class Fn, class MetF>
GRB_HD void take_solution(const DevEos& e, const C2PLive& L, const Fn& f, double mu, double pr[13], WB& wb,
                          MetF&& met) {
  const KScF& k = L.k;
  const double rho = clamp_f(f.rho, e.rhomin, e.rhomax);
  pr[GRB_P_RHO] = rho;
  pr[GRB_P_EPS] = f.eps;
  pr[GRB_P_PRESS] = f.prho * rho;
  pr[GRB_P_TEMP] = e.kind == GRB_EOS_IDEAL_GAS ? f.eth * e.gm1 : fmax(0.0, f.eth * e.gthm1);
  const double kz = f.w * mu * f.x, kb = mu * k.rBt * k.isD;
#pragma unroll
  for (int i = 0; i < 3; ++i) pr[GRB_P_ZX + i] = kz * (L.rup[i] + kb * pr[GRB_P_BX + i]);
  wb.W = f.w;
  wb.iW = f.iw;
  wb.z2 = f.w * f.w - 1.0;
  wb.Bz = f.w * mu * (k.rBt * (k.isD * k.D));
  wb.b2 = (k.b2 * k.D + wb.Bz * wb.Bz) * (f.iw * f.iw);
  if (f.vhigh) wb = wb_of(met(), pr);
}

// c2p_front in the tuned mode (plain bracket).
template <bool kDry = false, class MetF>
GRB_HD C2PState c2p_front_f(double c[10], double pr[13], const Met& m, const DevParams& P, double alp_bh_thresh,
                            C2PLive& L, MetF&& met) {
  C2PState F{};
  const DevEos& e = P.eos;
  C2POut& o = F.o;
  KScF& k = L.k;
  o.err = ERR_RESET_ENTROPY;
  F.failed = true;
#pragma unroll
  for (int v = 0; v < 10; ++v) c[v] *= m.isqrtg;
  pr[GRB_P_BX] = c[7]; pr[GRB_P_BY] = c[8]; pr[GRB_P_BZ] = c[9];
  F.lenient = m.alp < alp_bh_thresh;
  if (c[0] < 0) return F;  // c2p_back_f resets it to the atmosphere
  kscf(e, m, c, k);
  double ye = c[5] * k.iD;
  if (ye > e.yemax) { ye = e.yemax; o.err |= ERR_RESET_YE; }
  if (ye < 0.0) { ye = 0.0; o.err |= ERR_RESET_YE; }
  pr[GRB_P_YE] = ye;
  // limit_conservatives (c2p.cpp:117-157): tau below min(0, least eps).  The
  // least eps, negative only where the cold table's offsets are, is formed for
  // the states below 0 alone, and compared through the tau it gives (a value
  // less live: this kernel's registers are full).
  const double B2 = sqs(m.g, c + 7);
  if (k.q - 0.5 * B2 * k.iD < 0.0) {
    double lo, hi;
    eos_eps_range(e, lo, hi, c[0]);
    const double tau = lo * c[0] + 0.5 * B2;
    if (lo >= 0.0 || c[4] < tau) {
      c[4] = tau;
      k.q = c[4] * k.iD;
      o.err |= ERR_RESET_TAU;
      o.floored = true;
    }
  }
  const double qd = k.q + 1;
  if (!(k.r2 <= qd * qd)) {
    // S^2 / D^2 itself: r^i = S^i / D overflows before it, and infinite r^i
    // leave r^2 undefined
    const double st2 = sqs(m.gi, c + 1) * (k.iD * k.iD);
    if (st2 > qd * qd) {
      const double f = sqrt(qd * qd / st2);
      c[1] *= f; c[2] *= f; c[3] *= f;
      kscf(e, m, c, k);
      o.err |= ERR_RESET_STILDE;
      o.floored = true;
    }
  }
  if (o.floored && kDry) {
    F.done = true;
    return F;
  }
  if (!(c[0] >= P.rho_fl * (1 + P.atmo_tol))) return F;
  F.ran = true;
  if (!kDry) {
    mvs(m.gi, c + 1, L.rup);
#pragma unroll
    for (int i = 0; i < 3; ++i) L.rup[i] *= k.iD;
    L.s = c[6] * k.iD;
  }
  KFn f;
  f.e = &e;
  f.k = &k;
  F.mu0 = mu0_f(e, k);
  double res;
  const double mu = brent_root(f, F.mu0, false, o.iters, res);
  o.mu = mu;
  // the signals of the full evaluation (kastaun_c2p.hh:245-290)
  if (f.vhigh) F.ret |= SIG_VEL_HIGH;
  if (f.rho >= e.rhomax) F.ret |= SIG_RHO_HIGH;
  else if (f.rho <= e.rhomin) F.ret |= SIG_RHO_LOW;
  if (f.raw >= e.eps_max) F.ret |= SIG_EPS_HIGH;
  else if (f.raw < f.lo) F.ret |= SIG_EPS_LOW;
  // (a NaN tau reaches f through the clamped eps alone, which hides it)
  F.failed = !(fabs(res) <= P.tol) || !(f.raw == f.raw) || (F.ret & (SIG_RHO_HIGH | SIG_EPS_HIGH));
  F.wb_ok = true;
  if (kDry) {
    // only rho, T, z^2 and b^2 decide whether the state is floored
    pr[GRB_P_RHO] = clamp_f(f.rho, e.rhomin, e.rhomax);
    pr[GRB_P_TEMP] = e.kind == GRB_EOS_IDEAL_GAS ? f.eth * e.gm1 : f.eth * e.gthm1;
    F.wb.z2 = f.w * f.w - 1.0;
    F.wb.Bz = f.w * mu * (k.rBt * (k.isD * k.D));
    F.wb.b2 = (k.b2 * k.D + F.wb.Bz * F.wb.Bz) * (f.iw * f.iw);
    return F;
  }
  take_solution(e, L, f, mu, pr, F.wb, met);
  pr[GRB_P_ENT] = f.eth;
  const bool distrust =
      F.failed || (F.ret & SIG_EPS_LOW) || 2.0 * pr[GRB_P_PRESS] <= P.beta_fallback * fmax(F.wb.b2, 1e-50);
  F.backup = distrust && P.use_ent_backup;
  return F;
}

// c2p_backup in the tuned mode.  The reference's solve clamps the entropy to
// its range at every density it visits and keeps it clamped: the range at
// the bracket's two ends, its largest and smallest density, covers all.
template <class MetF>
GRB_HD void c2p_backup_f(C2PState& F, const C2PLive& L, double pr[13], const DevParams& P, MetF&& met) {
  const DevEos& e = P.eos;
  const bool ideal = e.kind == GRB_EOS_IDEAL_GAS;
  const KScF& k = L.k;
  const double mu0 = F.mu0 > 0.0 ? F.mu0 : mu0_f(e, k);
  EFn f;
  f.e = &e;
  f.k = &k;
  f.g = ideal ? e.gm1 : e.gthm1;
  f.elo = ideal ? e.ent_min : e.entropy_min;
  const double lD = log(k.D), s0 = L.s;
  f.sl = s0 + lD;
  // whether any density of the bracket may leave the entropy's range: the
  // thermal energy at rho = D, and a lower bound of it at D/W
  const double E0 = exp(f.g * f.sl);
  double pr0 = 0.0, ec0 = 0.0, r0 = k.D;
  if (!ideal) pw_cold_f(e, r0, k.iD, pr0, ec0);
  const bool clamp = !(E0 * k.ow >= f.elo && E0 <= e.eps_max - ec0 && f.g <= 2.0);
  int it = 0;
  double res;
  const double mu = brent_root(f, mu0, clamp, it, res);
  // (the clamps of eth would let a NaN entropy pass)
  if (s0 == s0 && fabs(res) <= P.tol && f.eps < e.eps_max) {
    uint32_t sig = 0;
    if (f.vhigh) sig |= SIG_VEL_HIGH;
    if (f.rho >= e.rhomax) sig |= SIG_RHO_HIGH;
    else if (f.rho <= e.rhomin) sig |= SIG_RHO_LOW;
    if (f.raw < f.elo * (1 - 1e-12)) sig |= SIG_ENT_LOW;
    if (f.raw > f.hi * (1 + 1e-12)) sig |= SIG_ENT_HIGH;
    F.ret = sig;
    F.failed = false;
    F.o.err |= ERR_ENT_BACKUP;
    take_solution(e, L, f, mu, pr, F.wb, met);
    F.wb_ok = true;
    pr[GRB_P_ENT] = clamp ? f.sl - lD : s0;
    F.ent_ok = true;
  }
  // otherwise the Kastaun primitives stand, or the state is reset if that failed
}

// c2p_back in the tuned mode.  excise: the state lies in the excised region.
// kAllCons false: the returned cons hold only what the reset flags in o.err
// ask for.
template <bool kAllCons = true, bool kDry = false, class MetF>
GRB_HD void c2p_back_f(C2PState& F, double c[10], double pr[13], double sqrtg, const DevParams& P, bool excise,
                       MetF&& met) {
  const DevEos& e = P.eos;
  const bool ideal = e.kind == GRB_EOS_IDEAL_GAS;
  C2POut& o = F.o;
  WB& wb = F.wb;
  if (F.ran) {
    const uint32_t ret = F.ret;
    if (ret & (SIG_EPS_HIGH | SIG_RHO_LOW | SIG_RHO_HIGH | SIG_VEL_HIGH)) o.floored = true;
    if (ideal && (ret & SIG_EPS_LOW)) o.floored = true;
    handle_sig(ret, F.lenient, o.err, o.fatal);
  }
  // which replacement of the primitives: 1 atmosphere, 2 temperature floor, 3 magnetisation
  int rep = 0;
  if (F.failed || excise || pr[GRB_P_RHO] < (1. + P.atmo_tol) * P.rho_fl) {
    rep = 1;
    o.floored = true;
    o.err |= ERR_ALL_RESETS | ERR_ATMO;
    pr[GRB_P_RHO] = P.rho_fl;
    pr[GRB_P_YE] = P.ye_fl;
    pr[GRB_P_TEMP] = P.temp_fl;
    pr[GRB_P_ZX] = pr[GRB_P_ZY] = pr[GRB_P_ZZ] = 0.;
    F.wb_ok = false;
  } else if (pr[GRB_P_TEMP] < P.temp_fl) {
    rep = 2;
    pr[GRB_P_TEMP] = P.temp_fl;
    o.err |= ERR_RESET_TAU | ERR_RESET_STILDE | ERR_RESET_ENTROPY | ERR_T_FLOORED;
    if (ideal) o.floored = true;
  } else {  // limit_primitives (c2p.cpp:63-115)
    uint32_t s2 = 0;
    const double z2max = P.max_w * P.max_w - 1.;
    if (!F.wb_ok) { wb = wb_of(met(), pr); F.wb_ok = true; }
    if (wb.z2 >= z2max) {
      s2 |= SIG_VEL_HIGH;
      if (!kDry) {
        const double zn = 0.99 * sqrt(z2max / wb.z2);
        pr[GRB_P_ZX] *= zn; pr[GRB_P_ZY] *= zn; pr[GRB_P_ZZ] *= zn;
        wb = wb_of(met(), pr);
      }
    }
    if (wb.b2 >= P.max_sigma * pr[GRB_P_RHO]) {
      s2 |= SIG_SIGMA_HIGH;
      rep = 3;
      if (!kDry) pr[GRB_P_RHO] = 1.001 * wb.b2 / P.max_sigma;
    }
    handle_sig(s2, F.lenient, o.err, o.fatal);
    if (s2) o.floored = true;
  }
  if (kDry) return;
  if (rep) {
    double cs2;
    uint32_t q = 0;
    pr[GRB_P_PRESS] = eos_PT(e, pr[GRB_P_EPS], cs2, nullptr, pr[GRB_P_TEMP], pr[GRB_P_RHO], q);
    if (rep == 2) handle_eos_sig(q, F.lenient, o.err, o.fatal);
    F.ent_ok = false;
    pr[GRB_P_ENT] = ideal ? pr[GRB_P_EPS] : fmax(0.0, pr[GRB_P_TEMP] * e.igthm1);
  }
  if (!F.ent_ok) {
    const double eth = pr[GRB_P_ENT];
    pr[GRB_P_ENT] = ideal ? log(eth) * e.igm1 - log(pr[GRB_P_RHO])
                          : log(fmax(eth, e.entropy_min)) * e.igthm1 - log(pr[GRB_P_RHO]);
  }
  const uint32_t need = kAllCons ? ~0u : o.err;
  if (!F.wb_ok || (need & (ERR_RESET_STILDE | ERR_RESET_TAU))) {
    const Met m = met();
    if (!F.wb_ok) wb = wb_of(m, pr);
    double zl[3], Bl[3];
    mvs(m.g, pr + GRB_P_ZX, zl);
    mvs(m.g, pr + GRB_P_BX, Bl);
    const double rhoh = pr[GRB_P_RHO] * (1. + pr[GRB_P_EPS]) + pr[GRB_P_PRESS] + wb.b2;
    const double pstar = pr[GRB_P_PRESS] + 0.5 * wb.b2;
    const double hW = rhoh * wb.W;
#pragma unroll
    for (int i = 0; i < 3; ++i)
      c[1 + i] = sqrtg * (hW * zl[i] - wb.Bz * ((Bl[i] + wb.Bz * zl[i]) * wb.iW));
    c[4] = sqrtg * (hW * wb.W - pstar - wb.Bz * wb.Bz - pr[GRB_P_RHO] * wb.W);
  }
  o.W = wb.W;
  o.iW = wb.iW;
  const double D = pr[GRB_P_RHO] * wb.W;
  c[0] = sqrtg * D;
  c[6] = sqrtg * (pr[GRB_P_ENT] * D);
  c[5] = c[0] * pr[GRB_P_YE];
}

// Whether conservs_to_prims excises the state.
GRB_HD bool excised(const DevParams& P, double alp, double r_sph) {
  return P.excise_by_radius ? (r_sph <= P.r_ex) : (alp <= P.alp_ex);
}

// The whole c2p in the tuned mode, and the FOFC flag's dry run.
template <bool kAllCons, class MetF>
GRB_HD C2POut c2p_f(double c[10], double pr[13], const Met& m, const DevParams& P, double r_sph, double alp_bh_thresh,
                    MetF&& met) {
  C2PLive L;
  const bool ex = excised(P, m.alp, r_sph);
  const double sqrtg = m.sqrtg;
  C2PState F = c2p_front_f(c, pr, m, P, alp_bh_thresh, L, met);
  if (F.backup) c2p_backup_f(F, L, pr, P, met);
  c2p_back_f<kAllCons>(F, c, pr, sqrtg, P, ex, met);
  return F.o;
}
template <class MetF>
GRB_HD bool c2p_floored_f(double c[10], double pr[13], const Met& m, const DevParams& P, double r_sph, MetF&& met) {
  C2PLive L;
  const bool ex = excised(P, m.alp, r_sph);
  C2PState F = c2p_front_f<true>(c, pr, m, P, 1e30, L, met);
  if (!F.done) c2p_back_f<true, true>(F, c, pr, 0.0, P, ex, met);
  return F.o.floored;
}

}  // namespace grb
