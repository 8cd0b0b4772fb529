// gp_lm_fast.cuh -- one Levenberg-Marquardt step of the contact solve as straight-line
// code, with the same rounded operations as lm_step (gp_lm.cuh).
//
// What bounds a solve is its chain of dependent FP64 operations.  On the B200 an FP64
// add, multiply or multiply-add takes 8 cycles, a division 112 and a square root 80, and
// the compiler's division and square root each end in a branch to their rare cases, so
// that independent ones do not overlap either (eight independent divisions: 8 x 113
// cycles).  A step has about 45 of them.  Here they are branch-free: a quotient is a
// hardware seed, a cubic Newton step and one correction with an exact remainder, so that
// independent ones fill each other's latency, several quotients by one divisor share its
// reciprocal, and a root brings the reciprocal of itself along.  The step holds its state in registers (nothing is passed by address),
// takes the pivot column's norm once and leaves out what lm_step forms and never reads.
// Operands outside the range in which the short forms are sound raise a flag, and a
// flagged step is run by lm_step: 49 of 2.87 M steps of 150,000 pairs shaped like those
// of the 512^3 workload.
//
// Measured (B200, such pairs; kernel time, results identical bit for bit):
//   one solve         6.2 us a step -> 1.9
//   2,000 solves      0.81 ms -> 0.22 (the longest takes 128 steps)
//   150,000 solves    2.45 ms -> 0.90
#pragma once
#include "gp_lm.cuh"

namespace gp {

#define GP_LF static __device__ __forceinline__

// Collected exponent checks: the largest distance of a checked high word from the lower
// end of the safe range [2^-300, 2^300).
struct LfGuard {
  unsigned far = 0u;
  static constexpr int kLo = (1023 - 300) << 20;
  static constexpr unsigned kSpan = 600u << 20;
  __device__ __forceinline__ void in(double v) {
    far = max(far, (unsigned)((__double2hiint(v) & 0x7fffffff) - kLo));
  }
  // A sum of squares s2 whose root is MINPACK's norm (lm_enorm).  From 2^-73 = 1.06e-22
  // on, components below rdwarf (squares below 1.5e-39) change neither the sum nor the
  // norm; below that every component has to lie above rdwarf (least: the smallest of
  // their high words).  Below 2^119 no component reaches rgiant / 3.
  __device__ __forceinline__ void norm(double s2, int least) {
    constexpr int lo = (1023 - 73) << 20;
    constexpr unsigned span = (73u + 119u) << 20;
    const int h = __double2hiint(s2);
    const bool fine = (unsigned)(h - lo) < span || (h < lo && least > 0x3be6a1c6);   // the high word of rdwarf
    far = max(far, fine ? 0u : 0xffffffffu);
  }
  // v is below 2^1023 in magnitude, neither infinite nor NaN
  __device__ __forceinline__ void finite(double v) { far = max(far, high(v) < 0x7fe00000 ? 0u : 0xffffffffu); }
  static __device__ __forceinline__ int high(double v) { return __double2hiint(v) & 0x7fffffff; }
  __device__ __forceinline__ bool ok() const { return far < kSpan; }
};

// Reciprocal of b to within an ulp: hardware seed (relative error e0 <= 2^-19), then
// y0 (1 + e + e^2) with e = 1 - b y0, whose truncation error is e0^3.
struct LfRcp {
  double b, y;
};
GP_LF LfRcp lf_rcp(double b, LfGuard& g) {
  g.in(b);
  double y0;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y0) : "d"(b));
  const double e = __fma_rn(-b, y0, 1.0);
  return {b, __fma_rn(y0, __fma_rn(e, e, e), y0)};
}

// a / b: q0 = a y is within 1.5 ulp, its remainder a - b q0 is exact in one fused
// operation, and q0 + r y rounds to the correctly rounded quotient (the correction step
// of P. Markstein, IBM J. Res. Dev. 34 (1990) 111) unless the quotient lies within 2^-52
// ulp of the midpoint between two doubles.
GP_LF double lf_quot(double a, const LfRcp& r) {
  const double q = __dmul_rn(a, r.y);
  return __fma_rn(__fma_rn(-r.b, q, a), r.y, q);
}
GP_LF double lf_div(double a, const LfRcp& r, LfGuard& g) {
  g.in(a);
  return lf_quot(a, r);
}
GP_LF double lf_div(double a, double b, LfGuard& g) {
  const LfRcp r = lf_rcp(b, g);
  g.in(a);
  return lf_quot(a, r);
}
// sqrt(a) and the reciprocal of that root: hardware seed of 1/sqrt, a cubic Newton step for
// both, one correction of the root with the exact remainder a - s^2 (as above; same
// condition).  1/sqrt(a) is within 1.5 ulp of 1/s, so a quotient by the root needs no
// reciprocal of its own.  The caller checks a.
GP_LF LfRcp lf_root(double a) {
  double y0;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y0) : "d"(a));
  const double t = __dmul_rn(a, y0);
  const double e = __fma_rn(-t, y0, 1.0);
  const double pe = __dmul_rn(e, __fma_rn(0.375, e, 0.5));
  const double s = __fma_rn(t, pe, t), y = __fma_rn(y0, pe, y0);
  return {__fma_rn(__fma_rn(-s, s, a), __dmul_rn(0.5, y), s), y};
}
GP_LF double lf_sqrt(double a, LfGuard& g) {
  g.in(a);
  return lf_root(a).b;
}

// MINPACK's norm (lm_enorm) where it is sqrt of the sum of squares, with its reciprocal.
GP_LF LfRcp lf_norm2(double x, double y, LfGuard& g) {
  const double s = x * x + y * y;
  g.norm(s, min(g.high(x), g.high(y)));
  return lf_root(s);
}
GP_LF LfRcp lf_norm3(double x, double y, double z, LfGuard& g) {
  const double s = x * x + y * y + z * z;
  g.norm(s, min(g.high(x), min(g.high(y), g.high(z))));
  return lf_root(s);
}

// ct_sincos without its range branch (the caller's guard covers it) and its switch.
GP_LF void lf_sincos(double x, double& s, double& c, LfGuard& g) {
  g.far = max(g.far, (__double2hiint(x) & 0x7fffffff) < (1023 + 20) << 20 ? 0u : 0xffffffffu);   // |x| < 2^20
  // rint by adding 1.5 2^52, whose sum's low word is the integer itself
  const double m = x * 0.6366197723675814 + 6755399441055744.0, k = m - 6755399441055744.0;
  const double r = ((x - k * 1.5707963267341256) - k * 6.077100506303966e-11) - k * 2.0222662487959506e-21;
  const double z = r * r;
  const double sn = r + r * z * ct_poly_sin(z);
  const double cs = 1.0 + z * (-0.5 + z * ct_poly_cos(z));
  const int q = __double2loint(m);
  const double a = (q & 1) ? cs : sn, b = (q & 1) ? sn : cs;
  s = (q & 2) ? -a : a;
  c = ((q + 1) & 2) ? -b : b;
}

// support_eval
template <class Prob>
GP_LF void lf_support(const Prob& P, double x0, double x1, SupportEval& E, LfGuard& g) {
  lf_sincos(x0, E.s0, E.k0, g);
  lf_sincos(x1, E.s1, E.k1, g);
  const double c1[3] = {E.k0 * E.k1, E.s0 * E.k1, E.s1};
  const double c2[3] = {-c1[0], -c1[1], -c1[2]};
  double t1[3], t2[3];
  prob_matvec<0>(P, c1, t1);
  prob_matvec<1>(P, c2, t2);
  const double q1 = 0.25 * (c1[0] * t1[0] + c1[1] * t1[1] + c1[2] * t1[2]);
  const double q2 = 0.25 * (c2[0] * t2[0] + c2[1] * t2[1] + c2[2] * t2[2]);
  g.in(q1);
  g.in(q2);
  const LfRcp l1 = lf_root(q1), l2 = lf_root(q2);
  E.l1 = l1.b;
  E.l2 = l2.b;
  E.f1 = lf_quot(1.0, {2.0 * l1.b, 0.5 * l1.y});
  E.f2 = lf_quot(1.0, {2.0 * l2.b, 0.5 * l2.y});
#pragma unroll
  for (int i = 0; i < 3; ++i)
    E.depth[i] = (E.f1 * t1[i] + P.template b<0>(i)) - (E.f2 * t2[i] + P.template b<1>(i));
}

// grad_coeff applied to the two columns of dc/dx (lm_jac's matvec)
template <int W, class Prob>
GP_LF void lf_grad(const Prob& P, const double c[3], double l, double s, const double ga[3], const double gb[3],
                   double oa[3], double ob[3], LfGuard& g) {
  double row[3];
#pragma unroll
  for (int j = 0; j < 3; ++j)
    row[j] = c[0] * P.template e<W>(3 * j) + c[1] * P.template e<W>(1 + 3 * j) + c[2] * P.template e<W>(2 + 3 * j);
  // 1 / (8 l^3) from s = 1 / (2 l): s^3 is within 3 ulp of it
  const double l3 = 8.0 * (l * l * l);
  g.in(l3);
  const double t = lf_quot(1.0, {l3, s * s * s});
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    double co[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const double eo = P.template e<W>(i) * (c[0] * row[j]) + P.template e<W>(i + 3) * (c[1] * row[j]) +
                        P.template e<W>(i + 6) * (c[2] * row[j]);
      co[j] = s * P.template e<W>(i + 3 * j) - t * eo;
    }
    oa[i] = co[0] * ga[0] + co[1] * ga[1] + co[2] * ga[2];
    ob[i] = co[0] * gb[0] + co[1] * gb[1] + co[2] * gb[2];
  }
}

// One Givens rotation of lm_qrsolv: cos and sin that rotate sdiag into r.
GP_LF void lf_givens(double r, double sd, double& cs, double& sn, LfGuard& g) {
  const bool big = fabs(r) >= fabs(sd);
  const double t = lf_div(big ? sd : r, big ? r : sd, g);
  const double u = lf_quot(0.5, lf_root(0.25 + 0.25 * (t * t)));
  const double v = u * t;
  cs = big ? u : v;
  sn = big ? v : u;
}

// lm_step's result codes; *ok false where the step must be run by lm_step instead (S is
// then as before the step, apart from values that lm_step forms again).
template <class Prob>
GP_LF int lm_step_fast(const Prob& P, LmState& S, double tol, bool& ok) {
  constexpr int maxfev = 300;
  LfGuard g;
  const LfRcp rf = lf_rcp(S.fnorm, g);
  double d0 = S.diag[0], d1 = S.diag[1];
  if (S.need_jac) {
    // lm_jac
    double a[6];
    {
      const SupportEval& E = S.E;
      const double ga[3] = {-E.s0 * E.k1, E.k0 * E.k1, 0.0}, gb[3] = {-E.k0 * E.s1, -E.s0 * E.s1, E.k1};
      const double na[3] = {-ga[0], -ga[1], -ga[2]}, nb[3] = {-gb[0], -gb[1], -gb[2]};
      const double c1[3] = {E.k0 * E.k1, E.s0 * E.k1, E.s1}, c2[3] = {-c1[0], -c1[1], -c1[2]};
      double pa[3], pb[3], qa[3], qb[3];
      lf_grad<0>(P, c1, E.l1, E.f1, ga, gb, pa, pb, g);
      lf_grad<1>(P, c2, E.l2, E.f2, na, nb, qa, qb, g);
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        a[i] = 2.0 * (E.depth[i] * (pa[i] - qa[i]));
        a[i + 3] = 2.0 * (E.depth[i] * (pb[i] - qb[i]));
      }
    }
    // lm_qrfac: the pivot column's norm is the one already taken
    const LfRcp c0 = lf_norm3(a[0], a[1], a[2], g), c1 = lf_norm3(a[3], a[4], a[5], g);
    const double ac0 = c0.b, ac1 = c1.b;
    const bool sw = ac1 > ac0;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const double t = a[i];
      a[i] = sw ? a[i + 3] : t;
      a[i + 3] = sw ? t : a[i + 3];
    }
    LfRcp r0 = sw ? c1 : c0;
    if (a[0] < 0.0) r0 = {-r0.b, -r0.y};
    const double n0 = r0.b;
#pragma unroll
    for (int i = 0; i < 3; ++i) a[i] = lf_div(a[i], r0, g);
    a[0] = a[0] + 1.0;
    const LfRcp ra0 = lf_rcp(a[0], g);
    {
      const double temp = lf_div((a[0] * a[3] + a[1] * a[4]) + a[2] * a[5], ra0, g);
#pragma unroll
      for (int i = 0; i < 3; ++i) a[i + 3] = a[i + 3] - temp * a[i];
    }
    LfRcp r1 = lf_norm2(a[4], a[5], g);
    if (a[4] < 0.0) r1 = {-r1.b, -r1.y};
    const double n1 = r1.b;
    a[4] = lf_div(a[4], r1, g);
    a[5] = lf_div(a[5], r1, g);
    a[4] = a[4] + 1.0;
    // Q^T fvec
    double w[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) w[i] = S.E.depth[i] * S.E.depth[i];
    {
      const double t = lf_div(-((a[0] * w[0] + a[1] * w[1]) + a[2] * w[2]), ra0, g);
#pragma unroll
      for (int i = 0; i < 3; ++i) w[i] = w[i] + a[i] * t;
      const double t1 = lf_div(-(a[4] * w[1] + a[5] * w[2]), a[4], g);
      w[1] = w[1] + a[4] * t1;
    }
    S.swapped = sw;
    S.fjac[0] = -n0;
    S.fjac[3] = a[3];
    S.fjac[4] = -n1;
    S.qtf[0] = w[0];
    S.qtf[1] = w[1];
    if (S.iter == 1) {
      d0 = ac0;
      d1 = ac1;
      S.xnorm = lf_norm2(ac0 * S.x[0], ac1 * S.x[1], g).b;
      S.delta = 100.0 * S.xnorm;
    }
    {
      const double s0 = lf_div(w[0], rf, g), s1 = lf_div(w[1], rf, g);
      const double g0 = fabs(lf_div(S.fjac[0] * s0, sel(sw, ac0, ac1), g));
      const double g1 = fabs(lf_div(S.fjac[3] * s0 + S.fjac[4] * s1, sel(!sw, ac0, ac1), g));
      double gnorm = (0.0 > g0) ? 0.0 : g0;
      gnorm = (gnorm > g1) ? gnorm : g1;
      S.gnorm = gnorm;
    }
    d0 = (d0 > ac0) ? d0 : ac0;
    d1 = (d1 > ac1) ? d1 : ac1;
  }
  const bool sw = S.swapped;
  const double R0 = S.fjac[0], R3 = S.fjac[3], R4 = S.fjac[4], q0 = S.qtf[0], q1 = S.qtf[1];
  double delta = S.delta, par = S.par;
  // lm_lmpar
  double x0, x1, w0, w1;
  {
    const LfRcp rr0 = lf_rcp(R0, g), rr4 = lf_rcp(R4, g);
    const double z1 = lf_div(q1, rr4, g);
    const double z0 = lf_div(q0 - R3 * z1, rr0, g);
    x0 = sel(sw, z0, z1);
    x1 = sel(sw, z1, z0);
    w0 = d0 * x0;
    w1 = d1 * x1;
    const LfRcp gauss = lf_norm2(w0, w1, g);
    double fp = gauss.b - delta;
    if (fp <= 0.1 * delta) {
      par = 0.0;
    } else {
      const double dp0 = sel(sw, d0, d1), dp1 = sel(!sw, d0, d1);
      const LfRcp rdel = lf_rcp(delta, g);
      double parl, paru, gn;
      {
        double v0 = dp0 * lf_div(sel(sw, w0, w1), gauss, g);
        double v1 = dp1 * lf_div(sel(!sw, w0, w1), gauss, g);
        v0 = lf_div(v0 - 0.0, rr0, g);
        v1 = lf_div(v1 - (0.0 + R3 * v0), rr4, g);
        const LfRcp rt = lf_norm2(v0, v1, g);
        parl = lf_div(lf_div(lf_div(fp, rdel, g), rt, g), rt, g);
        const double s0 = 0.0 + R0 * q0, s1 = (0.0 + R3 * q0) + R4 * q1;
        gn = lf_norm2(lf_div(s0, dp0, g), lf_div(s1, dp1, g), g).b;
        paru = lf_div(gn, rdel, g);
      }
      double p = par;
      p = (p > parl) ? p : parl;
      p = (p < paru) ? p : paru;
      if (p == 0.0) p = lf_div(gn, gauss, g);
#pragma unroll 1
      for (int iter = 1;; ++iter) {
        const double sp = lf_sqrt(p, g);
        // lm_qrsolv with diag = sp * diag
        const double e0 = sp * dp0, e1 = sp * dp1;
        double cs, sn, sd0, sd1, r1, y0, y1, b;
        lf_givens(R0, e0, cs, sn, g);
        sd0 = cs * R0 + sn * e0;
        y0 = cs * q0 + sn * 0.0;
        b = -sn * q0 + cs * 0.0;
        r1 = cs * R3 + sn * 0.0;
        const double t1 = -sn * R3 + cs * 0.0;
        // the element the first rotation left in sdiag[1]
        double r4 = R4, q = q1;
        if (t1 != 0.0) {
          lf_givens(r4, t1, cs, sn, g);
          r4 = cs * r4 + sn * t1;
          const double temp = cs * q + sn * b;
          b = -sn * q + cs * b;
          q = temp;
        }
        lf_givens(r4, e1, cs, sn, g);
        sd1 = cs * r4 + sn * e1;
        y1 = cs * q + sn * 0.0;
        const LfRcp rs0 = lf_rcp(sd0, g), rs1 = lf_rcp(sd1, g);
        y1 = lf_div(y1, rs1, g);
        y0 = lf_div(y0 - (0.0 + r1 * y1), rs0, g);
        x0 = sel(sw, y0, y1);
        x1 = sel(sw, y1, y0);
        w0 = d0 * x0;
        w1 = d1 * x1;
        const LfRcp rn = lf_norm2(w0, w1, g);
        const double told = fp;
        fp = rn.b - delta;
        if (fabs(fp) <= 0.1 * delta || (parl == 0.0 && fp <= told && told < 0.0) || iter == 10 || !g.ok()) break;
        double v0 = dp0 * lf_div(sel(sw, w0, w1), rn, g);
        double v1 = dp1 * lf_div(sel(!sw, w0, w1), rn, g);
        v0 = lf_div(v0, rs0, g);
        v1 = v1 - r1 * v0;
        v1 = lf_div(v1, rs1, g);
        const LfRcp rt = lf_norm2(v0, v1, g);
        const double parc = lf_div(lf_div(lf_div(fp, rdel, g), rt, g), rt, g);
        if (fp > 0.0) parl = (parl > p) ? parl : p;
        if (fp < 0.0) paru = (paru < p) ? paru : p;
        const double t2 = p + parc;
        p = (parl > t2) ? parl : t2;
      }
      par = p;
    }
  }
  // the trial point
  const double s0 = -x0, s1 = -x1;
  const double xt0 = S.x[0] + s0, xt1 = S.x[1] + s1;
  const double pnorm = lf_norm2(d0 * s0, d1 * s1, g).b;
  if (S.iter == 1) delta = (delta < pnorm) ? delta : pnorm;
  SupportEval E2;
  lf_support(P, xt0, xt1, E2, g);
  const double fnorm1 = lf_norm3(E2.depth[0] * E2.depth[0], E2.depth[1] * E2.depth[1], E2.depth[2] * E2.depth[2], g).b;
  double actred = -1.0;
  if (0.1 * fnorm1 < S.fnorm) { const double r = lf_quot(fnorm1, rf); actred = 1.0 - r * r; }
  const double p0 = sel(sw, s0, s1), p1 = sel(!sw, s0, s1);
  const double v0 = (0.0 + R0 * p0) + R3 * p1, v1 = 0.0 + R4 * p1;
  const double temp1 = lf_div(lf_norm2(v0, v1, g).b, rf, g);
  double temp2 = 0.0;
  if (par != 0.0) temp2 = lf_div(lf_sqrt(par, g) * pnorm, rf, g);
  const double prered = temp1 * temp1 + (temp2 * temp2) * 2.0;
  const double dirder = -(temp1 * temp1 + temp2 * temp2);
  // |actred| is 0 or from 1e-16 to 100
  const double ratio = lf_quot(actred, lf_rcp(prered, g));
  double temp = S.temp;
  if (ratio <= 0.25) {
    if (actred >= 0.0) temp = 0.5;
    if (actred < 0.0) temp = lf_div(0.5 * dirder, dirder + 0.5 * actred, g);
    if (0.1 * fnorm1 >= S.fnorm || temp < 0.1) temp = 0.1;
    const double pt = lf_quot(pnorm, {0.1, 10.0});
    const double m = (delta < pt) ? delta : pt;
    delta = temp * m;
    if (par != 0.0) par = lf_div(par, temp, g);
  } else if (par == 0.0 || ratio >= 0.75) {
    delta = pnorm * 2.0;
    par = 0.5 * par;
  }
  const bool accept = ratio >= 1.0e-4;
  double xnorm = S.xnorm;
  if (accept) xnorm = lf_norm2(d0 * xt0, d1 * xt1, g).b;
  ok = g.ok();
  if (!ok) return 0;
  ++S.nfev;
  S.need_jac = false;
  S.diag[0] = d0;
  S.diag[1] = d1;
  S.delta = delta;
  S.par = par;
  S.temp = temp;
  S.xnorm = xnorm;
  if (accept) {
    S.x[0] = xt0;
    S.x[1] = xt1;
    S.E = E2;
    S.fnorm = fnorm1;
    ++S.iter;
  }
  int info = 0;
  if (fabs(actred) <= tol && prered <= tol && 0.5 * ratio <= 1.0) info = 1;
  if (delta <= tol * xnorm) info = info != 0 ? 3 : 2;
  if (info != 0) return info;
  if (S.nfev >= maxfev) info = 5;
  if (fabs(actred) <= DBL_EPSILON && prered <= DBL_EPSILON && 0.5 * ratio <= 1.0) info = 6;
  if (delta <= DBL_EPSILON * xnorm) info = 7;
  if (S.gnorm <= DBL_EPSILON) info = 8;
  if (info != 0) return info == 8 ? 4 : info;
  if (accept) S.need_jac = true;
  return 0;
}

// lm_step where the straight-line step gave up.  Out of line, on copies, so that the
// caller's problem and state stay in registers.
static __device__ __noinline__ int lm_step_general(const ContactProb* P, LmState* S) {
  return lm_step(*P, *S, kContactTol);
}

// One step of the solve; 0 to continue, otherwise lmder's info code.
GP_LF int lm_advance(const ContactProb& P, LmState& S) {
  bool ok;
  int info = lm_step_fast(P, S, kContactTol, ok);
  if (!ok) {
    const ContactProb p = P;
    LmState s = S;
    info = lm_step_general(&p, &s);
    S = s;
  }
  return info;
}

// The solve's start: the problem, the starting angles and the residual there.  Returns
// false when there is nothing to solve (contact_setup).  Out of line, once per solve.
static __device__ __noinline__ bool solve_start(double a1, double bb1, double a2, double bb2, const double c1[3],
                                                const Quat& q1, const double c2[3], const Quat& q2, ContactProb& P,
                                                LmState& S) {
  if (!contact_setup(a1, bb1, a2, bb2, c1, q1, c2, q2, P, S.x)) return false;
  lm_begin(P, S);
  return true;
}

// ellipsoid_contact_detection.f90:1-187 for one pair, start to finish.
GP_LF bool contact_detection(double a1, double bb1, double a2, double bb2, const double c1[3], const Quat& q1,
                             const double c2[3], const Quat& q2, double ept1[3], double ept2[3], double cn[3]) {
  ContactProb p;
  LmState s;
  if (!solve_start(a1, bb1, a2, bb2, c1, q1, c2, q2, p, s)) {
#pragma unroll
    for (int i = 0; i < 3; ++i) { ept1[i] = CUDART_NAN; ept2[i] = CUDART_NAN; cn[i] = CUDART_NAN; }
    return false;
  }
  double x[2];
  {
    const ContactProb P = p;
    LmState S = s;
    while (lm_advance(P, S) == 0) {
    }
    x[0] = S.x[0];
    x[1] = S.x[1];
  }
  return contact_finish(a1, bb1, a2, bb2, q1, q2, p, x, ept1, ept2, cn);
}

}  // namespace gp
