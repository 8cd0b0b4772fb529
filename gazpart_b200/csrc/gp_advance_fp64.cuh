// gp_advance_fp64.cuh -- the FP64 form's RK2 step of one particle as straight-line code.
//
// The step evaluates the force and torque correlations twice: about 45 powers, 40
// divisions and 25 square roots.  Called one by one each power is some hundred
// instructions that end in range branches, and the compiler's division (112 cycles) and
// square root (80) do not overlap either, so the warps waited on FP64 latency with the
// pipe mostly idle.  Here
//  - a base's logarithm is taken once, in two doubles, and each of its powers is one
//    product and one exponential (x^y = 2^(y log2 x)); quotients by powers are products
//    with the negative power;
//  - divisions and roots are gp_lm_fast.cuh's branch-free ones, correctly rounded like the
//    ones they replace, several quotients by one divisor sharing its reciprocal;
//  - sine and cosine are taken on the ranges that occur.
// Operands outside the ranges in which this is sound, an intersected wall and every error
// raise a flag, and integrate_slot then advances the particle by advance_particle, which
// is written for any operands.
//
// Accuracy, on 2 M arguments over these ranges against 64-bit-mantissa results (largest
// and mean error in ulps): the powers 0.95 and 0.26 (CUDA's pow 1.35 and 0.31), sine and
// cosine 0.78 and 0.16 (CUDA's sincos 1.35 and 0.17); quotients and roots were equal to
// CUDA's in every case.
//
// Exact zeros are inside the ranges: particles that settle in still fluid have them in the
// spin and the torque at every step, bodies along or across the flow in the slip.
//
// Measured (B200, integrate of one step): 1 M particles 0.58 -> 0.30 ms, 10,000 38 -> 21 us;
// 1 M settling in still fluid 0.61 -> 0.33 (1.17 where a zero raises the flag).
#pragma once
#include "gp_lm_fast.cuh"

namespace gp {

// log2 x = hi + lo for x in the guard's range.  x = 2^k m with m in [1, 2); the table holds
// a 10-bit reciprocal of the middle of each 64th of [1, 2) and its -log2 as the sum of a
// multiple of 2^-40 (so that k is added exactly) and a rest, and r = m inv - 1 is formed in
// one rounding; log2(1 + r) is its series with the first term in two doubles (table-driven
// reduction after P.T.P. Tang, ACM Trans. Math. Softw. 16 (1990) 378).
struct Log2 {
  double hi, lo;
};
struct alignas(32) Log2Row {
  double inv, hi, lo, pad;
};
static __device__ const Log2Row g_log2_rows[64] = {
    {0x1.fc00000000000p-1, 0x1.72c7ba2100000p-7, -0x1.19b14945cf6bap-44, 0.0},
    {0x1.f480000000000p-1, 0x1.0c7b844f00000p-5, -0x1.d0d656726e19bp-42, 0.0},
    {0x1.ed00000000000p-1, 0x1.beec9151a0000p-5, 0x1.585ca360898fbp-42, 0.0},
    {0x1.e580000000000p-1, 0x1.3a0cf56a00000p-4, 0x1.b12a90d3a7915p-42, 0.0},
    {0x1.de80000000000p-1, 0x1.8fdf1ca8f0000p-4, -0x1.595f2f68d91fdp-44, 0.0},
    {0x1.d780000000000p-1, 0x1.e6f50c2da0000p-4, -0x1.15844900583dep-45, 0.0},
    {0x1.d100000000000p-1, 0x1.1c7e77dde0000p-3, 0x1.9edc58b89b49ep-42, 0.0},
    {0x1.ca80000000000p-1, 0x1.46163957b0000p-3, -0x1.fa4a9eb6b8621p-44, 0.0},
    {0x1.c400000000000p-1, 0x1.7046031c78000p-3, 0x1.f84be19cb9578p-43, 0.0},
    {0x1.be00000000000p-1, 0x1.97c1cb13c8000p-3, -0x1.3f7a55cd2af4cp-47, 0.0},
    {0x1.b800000000000p-1, 0x1.bfc67a8000000p-3, -0x1.667f21fa8423fp-44, 0.0},
    {0x1.b200000000000p-1, 0x1.e857d3d360000p-3, 0x1.367bde40c5e6dp-43, 0.0},
    {0x1.ac80000000000p-1, 0x1.070352293c000p-2, 0x1.72468f6eed407p-42, 0.0},
    {0x1.a700000000000p-1, 0x1.1a190a5d68000p-2, -0x1.6bf2e7459b97dp-43, 0.0},
    {0x1.a180000000000p-1, 0x1.2d6eb41524000p-2, -0x1.b6145ff213790p-43, 0.0},
    {0x1.9c00000000000p-1, 0x1.4106017c40000p-2, -0x1.35d71963580bap-42, 0.0},
    {0x1.9700000000000p-1, 0x1.530fd08f28000p-2, 0x1.fa709d0b28090p-42, 0.0},
    {0x1.9200000000000p-1, 0x1.6552b49988000p-2, -0x1.d8894dbdff331p-42, 0.0},
    {0x1.8d00000000000p-1, 0x1.77d01b66fc000p-2, -0x1.64adb1adca9a8p-45, 0.0},
    {0x1.8880000000000p-1, 0x1.88a76b7e54000p-2, 0x1.38b2546b396e9p-43, 0.0},
    {0x1.8400000000000p-1, 0x1.99b072a96c000p-2, 0x1.ac9bca36fd02ep-44, 0.0},
    {0x1.7f80000000000p-1, 0x1.aaec59dadc000p-2, -0x1.2420130cd23b5p-42, 0.0},
    {0x1.7b00000000000p-1, 0x1.bc5c548924000p-2, 0x1.4cb9d5e17a5ebp-42, 0.0},
    {0x1.7680000000000p-1, 0x1.ce01a12f5c000p-2, 0x1.8d11f5fdec0d4p-42, 0.0},
    {0x1.7280000000000p-1, 0x1.dddecf870c000p-2, 0x1.305af9767a020p-44, 0.0},
    {0x1.6e00000000000p-1, 0x1.efec61b010000p-2, 0x1.f855b4987c5d5p-42, 0.0},
    {0x1.6a00000000000p-1, 0x1.0014332be0000p-1, 0x1.9518ce032f41dp-48, 0.0},
    {0x1.6600000000000p-1, 0x1.08494c66b8000p-1, 0x1.ddf82e1fe57c7p-42, 0.0},
    {0x1.6200000000000p-1, 0x1.1096015dee000p-1, 0x1.3676289cd3dd4p-43, 0.0},
    {0x1.5e80000000000p-1, 0x1.17ece95560000p-1, -0x1.46fab3fa1a144p-44, 0.0},
    {0x1.5b00000000000p-1, 0x1.1f56ac9eda000p-1, -0x1.5cb804b949696p-43, 0.0},
    {0x1.5700000000000p-1, 0x1.27e72080fc000p-1, 0x1.bcb999fe93d45p-42, 0.0},
    {0x1.5380000000000p-1, 0x1.2f7a997fb6000p-1, -0x1.ab45da1d64cdep-42, 0.0},
    {0x1.5000000000000p-1, 0x1.37222bb708000p-1, -0x1.708b4b2b5056cp-42, 0.0},
    {0x1.4c80000000000p-1, 0x1.3ede42e88c000p-1, 0x1.e12462f69f788p-43, 0.0},
    {0x1.4980000000000p-1, 0x1.4590247acc000p-1, 0x1.c783c39e591e3p-42, 0.0},
    {0x1.4600000000000p-1, 0x1.4d7380dcc4000p-1, 0x1.1646b761c48dep-44, 0.0},
    {0x1.4300000000000p-1, 0x1.5447b72664000p-1, 0x1.cd53be1f94c50p-44, 0.0},
    {0x1.3f80000000000p-1, 0x1.5c53ef8e2e000p-1, -0x1.286fbc7f749ffp-45, 0.0},
    {0x1.3c80000000000p-1, 0x1.634be1dab2000p-1, -0x1.d33642a048025p-43, 0.0},
    {0x1.3980000000000p-1, 0x1.6a54d1a668000p-1, -0x1.3b5f7fb2daa67p-42, 0.0},
    {0x1.3680000000000p-1, 0x1.716f1296b6000p-1, -0x1.63268bcb6f2bep-42, 0.0},
    {0x1.3380000000000p-1, 0x1.789afac0b8000p-1, -0x1.e0b3dbe80c6c7p-42, 0.0},
    {0x1.3100000000000p-1, 0x1.7ea2a2ed98000p-1, -0x1.98eec5e85b29fp-44, 0.0},
    {0x1.2e00000000000p-1, 0x1.85efd062c6000p-1, 0x1.5b338360c2ae2p-43, 0.0},
    {0x1.2b80000000000p-1, 0x1.8c13b3791c000p-1, 0x1.dffed11e2bd73p-42, 0.0},
    {0x1.2880000000000p-1, 0x1.938360a10a000p-1, 0x1.601ccfac2b557p-45, 0.0},
    {0x1.2600000000000p-1, 0x1.99c48be206000p-1, 0x1.e41fa0a62e6aep-44, 0.0},
    {0x1.2380000000000p-1, 0x1.a013639988000p-1, 0x1.d25cfd9459b34p-44, 0.0},
    {0x1.2080000000000p-1, 0x1.a7b794e2e0000p-1, -0x1.3cf0ff16ff990p-43, 0.0},
    {0x1.1e00000000000p-1, 0x1.ae255819f0000p-1, 0x1.1659d8e2d7d38p-44, 0.0},
    {0x1.1b80000000000p-1, 0x1.b4a18e5b20000p-1, 0x1.023272a855a1ap-43, 0.0},
    {0x1.1980000000000p-1, 0x1.b9dc4d0b8c000p-1, -0x1.6be4a29c44115p-43, 0.0},
    {0x1.1700000000000p-1, 0x1.c0732be1ea000p-1, -0x1.49209a68c72a1p-49, 0.0},
    {0x1.1480000000000p-1, 0x1.c71939b5d8000p-1, 0x1.0ac59a41a5281p-42, 0.0},
    {0x1.1200000000000p-1, 0x1.cdcebd2374000p-1, -0x1.9ad57391924a7p-43, 0.0},
    {0x1.1000000000000p-1, 0x1.d338120a6e000p-1, -0x1.3167ccc538261p-44, 0.0},
    {0x1.0d80000000000p-1, 0x1.da0a215466000p-1, 0x1.323682bdd649ep-42, 0.0},
    {0x1.0b80000000000p-1, 0x1.df8aae0e46000p-1, 0x1.eacede1650abdp-42, 0.0},
    {0x1.0980000000000p-1, 0x1.e515cce9f6000p-1, 0x1.411c95ce3da68p-42, 0.0},
    {0x1.0700000000000p-1, 0x1.ec12cf6b98000p-1, -0x1.6898809d2dc10p-43, 0.0},
    {0x1.0500000000000p-1, 0x1.f1b64e22be000p-1, -0x1.0f86666e80f71p-42, 0.0},
    {0x1.0300000000000p-1, 0x1.f764e7742c000p-1, -0x1.7b0c4bb41a6c9p-42, 0.0},
    {0x1.0100000000000p-1, 0x1.fd1ec77250000p-1, 0x1.54e22d4990b6ep-42, 0.0}};

GP_LF Log2 fw_log2(double x, LfGuard& g, int least_exp, int most_exp) {
  const int h = __double2hiint(x);
  // 2^least <= x < 2^most (also false for negative numbers, zero, infinity and NaN)
  g.far = max(g.far, (unsigned)(h - ((1023 + least_exp) << 20)) < (unsigned)((most_exp - least_exp) << 20) ? 0u
                                                                                                            : 0xffffffffu);
  const int k = (h >> 20) - 1023;
  const double m = __hiloint2double((h & 0xfffff) | 0x3ff00000, __double2loint(x));
  const Log2Row& row = g_log2_rows[(h >> 14) & 63];
  const double2 a = __ldg(reinterpret_cast<const double2*>(&row));
  const double tlo = __ldg(&row.lo);
  const double r = __fma_rn(m, a.x, -1.0);
  constexpr double c = 0x1.71547652b82fep+0, cl = 0x1.777d0ffda0d24p-56;   // 1 / ln 2
  const double p = __dmul_rn(r, c);
  const double pl = __fma_rn(r, cl, __fma_rn(r, c, -p));
  // the series from r^2 on: (-1)^(n+1) / (n ln 2)
  double q = 0x1.484b13d7c02a9p-3;
  q = __fma_rn(q, r, -0x1.71547652b82fep-3);
  q = __fma_rn(q, r, 0x1.a61762a7aded9p-3);
  q = __fma_rn(q, r, -0x1.ec709dc3a03fdp-3);
  q = __fma_rn(q, r, 0x1.2776c50ef9bfep-2);
  q = __fma_rn(q, r, -0x1.71547652b82fep-2);
  q = __fma_rn(q, r, 0x1.ec709dc3a03fdp-2);
  q = __fma_rn(q, r, -0x1.71547652b82fep-1);
  const double rest = __fma_rn(__dmul_rn(r, r), q, __dadd_rn(pl, tlo));
  const double s = __dadd_rn((double)k, a.y);   // exact
  const double t = __dadd_rn(s, p);             // two-sum
  const double v = __dsub_rn(t, s);
  const double e = __dadd_rn(__dsub_rn(s, __dsub_rn(t, v)), __dsub_rn(p, v));
  const double lo = __dadd_rn(e, rest);
  const double hi = __dadd_rn(t, lo);
  return {hi, __dsub_rn(lo, __dsub_rn(hi, t))};
}

// 2^(y (hi + lo)), results below 2^-1020 as 2^-1020 (they stand for a factor that vanishes
// beside the others).  2^f on |f| <= 1/2 by its Taylor series to f^13 (rest below 2^-57).
GP_LF double fw_pow(const Log2& l, double y) {
  const double th = fmax(__dmul_rn(y, l.hi), -1020.0);
  const double tl = __fma_rn(y, l.lo, __fma_rn(y, l.hi, -th));
  const double m = __dadd_rn(th, 6755399441055744.0);   // 1.5 2^52: rounds to an integer
  const double f = __dadd_rn(__dsub_rn(th, __dsub_rn(m, 6755399441055744.0)), th > -1020.0 ? tl : 0.0);
  double q = 0x1.816193166d0f9p-40;
  q = __fma_rn(q, f, 0x1.c3bd650fc2986p-36);
  q = __fma_rn(q, f, 0x1.e8cac7351bb25p-32);
  q = __fma_rn(q, f, 0x1.e4cf5158b8ecap-28);
  q = __fma_rn(q, f, 0x1.b5253d395e7c4p-24);
  q = __fma_rn(q, f, 0x1.62c0223a5c824p-20);
  q = __fma_rn(q, f, 0x1.ffcbfc588b0c7p-17);
  q = __fma_rn(q, f, 0x1.430912f86c787p-13);
  q = __fma_rn(q, f, 0x1.5d87fe78a6731p-10);
  q = __fma_rn(q, f, 0x1.3b2ab6fba4e77p-7);
  q = __fma_rn(q, f, 0x1.c6b08d704a0c0p-5);
  q = __fma_rn(q, f, 0x1.ebfbdff82c58fp-3);
  q = __fma_rn(q, f, 0x1.62e42fefa39efp-1);
  const double r = __fma_rn(q, f, 1.0);
  return __hiloint2double(__double2hiint(r) + (__double2loint(m) << 20), __double2loint(r));
}

// Sine and cosine for 0 <= x < 2^20: lf_sincos's reduction and series with fused
// operations, the reduced argument and 1 - z/2 each with the rest that rounding left.
GP_LF void fw_sincos(double x, double& s, double& c, LfGuard& g) {
  g.far = max(g.far, (unsigned)__double2hiint(x) < (unsigned)((1023 + 20) << 20) ? 0u : 0xffffffffu);
  const double m = __fma_rn(x, 0.6366197723675814, 6755399441055744.0), k = __dsub_rn(m, 6755399441055744.0);
  const double r1 = __fma_rn(-k, 1.5707963267341256, x), r = __fma_rn(-k, 6.077100506303966e-11, r1);
  const double rl = __fma_rn(-k, 2.0222662487959506e-21, __fma_rn(-k, 6.077100506303966e-11, __dsub_rn(r1, r)));
  const double z = __dmul_rn(r, r);
  double a = -7.647163731819816e-13, b = -1.1470745597729725e-11;   // Taylor: 1/15!, 1/14!, ...
  a = __fma_rn(2.8114572543455206e-15, z, a);
  b = __fma_rn(4.779477332387385e-14, z, b);
  a = __fma_rn(a, z, 1.6059043836821613e-10);
  b = __fma_rn(b, z, 2.08767569878681e-09);
  a = __fma_rn(a, z, -2.505210838544172e-08);
  b = __fma_rn(b, z, -2.755731922398589e-07);
  a = __fma_rn(a, z, 2.7557319223985893e-06);
  b = __fma_rn(b, z, 2.48015873015873e-05);
  a = __fma_rn(a, z, -0.0001984126984126984);
  b = __fma_rn(b, z, -0.001388888888888889);
  a = __fma_rn(a, z, 0.008333333333333333);
  b = __fma_rn(b, z, 0.041666666666666664);
  a = __fma_rn(a, z, -0.16666666666666666);
  const double sn = __dadd_rn(r, __fma_rn(__dmul_rn(r, z), a, rl));
  const double hz = __dmul_rn(0.5, z), w1 = __dsub_rn(1.0, hz);
  const double cs = __dadd_rn(w1, __fma_rn(__dmul_rn(z, z), b, __fma_rn(-r, rl, __dsub_rn(__dsub_rn(1.0, w1), hz))));
  const int q = __double2loint(m);
  const double u = (q & 1) ? cs : sn, w = (q & 1) ? sn : cs;
  s = (q & 2) ? -u : u;
  c = ((q + 1) & 2) ? -w : w;
}

// Quotients and roots that take an exact zero: in still fluid, or with a body along or across
// the flow, components of the slip, the spin and the torque are zero at every step.
// a / r.b for r.b > 0, the zero with a's sign (lf_quot's remainder would lose a negative one).
// No guard: the caller knows that a is finite, or looks at what comes of it.
GP_LF double fw_quot(double a, const LfRcp& r) {
  const double q = __dmul_rn(a, r.y);
  return __fma_rn(-__fma_rn(r.b, q, -a), r.y, q);
}
GP_LF bool is_zero(double a) { return (LfGuard::high(a) | __double2loint(a)) == 0; }
GP_LF double fw_sqrt(double a, LfGuard& g) {
  const bool zero = is_zero(a);
  const double v = zero ? 1.0 : a;
  g.in(v);
  const double s = lf_root(v).b;
  return zero ? 0.0 : s;
}

// slip64 with what the correlations take of it.
struct SlipFast {
  bool moving;   // the slip is not zero (a particle set off with the fluid's velocity)
  bool along;    // the slip is along the axis, its transverse parts are zero
  double p[3], umag, rep, phi, sphi, cphi;
  LfRcp syz;     // the transverse slip as a divisor (1 along the axis)
  Log2 lrep, lsin, lcos;
};
GP_LF void fw_slip(const PartConst& pc, const LfRcp& rv, const double u[3], const double uf[3], const double r[9],
                   SlipFast& s, LfGuard& g) {
  const double p[3] = {uf[0] - u[0], uf[1] - u[1], uf[2] - u[2]};
  const double pp = p[0] * p[0] + p[1] * p[1] + p[2] * p[2];
  s.moving = pp != 0.0;
  if (!s.moving) return;
  s.rep = lf_quot(lf_sqrt(pp, g) * pc.deq, rv);
  matvec_t(r, p, s.p);
  const double yz = s.p[1] * s.p[1] + s.p[2] * s.p[2];
  s.along = is_zero(yz);
  s.syz = lf_root(s.along ? 1.0 : yz);
  g.in(s.along ? 1.0 : yz);
  s.umag = lf_sqrt(s.p[0] * s.p[0] + s.p[1] * s.p[1] + s.p[2] * s.p[2], g);
  // across the axis the quotient is infinite, along it the sine is zero, and so is each of
  // its powers (their exponents are above 1/2 from Re = 2^-100 on)
  const bool across = is_zero(s.p[0]);
  const double tphi = lf_quot(s.along ? 0.0 : s.syz.b, lf_rcp(across ? 1.0 : s.p[0], g));
  s.phi = fabs(atan(across ? CUDART_INF : tphi));
  fw_sincos(s.phi, s.sphi, s.cphi, g);
  s.lrep = fw_log2(s.rep, g, s.along ? -100 : -200, 20);
  s.lsin = fw_log2(s.along ? 1.0 : s.sphi, g, -160, 1);
  if (s.along) s.lsin.hi = -4096.0;
  s.lcos = fw_log2(s.cphi, g, -60, 1);
}

// fluid_force: drag plus lift in the lab frame
GP_LF void fw_force(const PartConst& pc, const SlipFast& s, const double r[9], double f[3], LfGuard& g) {
  f[0] = f[1] = f[2] = 0.0;
  if (!s.moving) return;
  const double cd0 = 18.12 * fw_pow(s.lrep, -1.023) + 4.26 * fw_pow(s.lrep, -0.384);
  const double cd90 = 21.52 * fw_pow(s.lrep, -0.990) + 2.86 * fw_pow(s.lrep, -0.260);
  const double cdrag = cd0 + (cd90 - cd0) * fw_pow(s.lsin, 1.95);
  const double clift = (0.083 * fw_pow(s.lrep, 0.21) + 1.582 * fw_pow(s.lrep, -0.851)) *
                       fw_pow(s.lsin, 1.842 + -0.802 * fw_pow(s.lrep, -0.006)) *
                       fw_pow(s.lcos, 0.874 + 0.009 * fw_pow(s.lrep, 0.570));
  const double kd = pc.cdrag * cdrag * s.umag;
  double fd[3] = {kd * s.p[0], kd * s.p[1], kd * s.p[2]};
  const double kl = pc.cdrag * clift * (s.umag * s.umag);
  double fl[3] = {kl * s.sphi * copysign(1.0, -s.p[0]), kl * s.cphi * fw_quot(s.p[1], s.syz),
                  kl * s.cphi * fw_quot(s.p[2], s.syz)};
  matvec(r, fd, fd);
  matvec(r, fl, fl);
#pragma unroll
  for (int i = 0; i < 3; ++i) f[i] = fd[i] + fl[i];
}

// fluid_torque: pitching plus rotation torque in the body frame
GP_LF void fw_torque(const PartConst& pc, const LfRcp& rv, const SlipFast& s, const double wv[3], const double o[3],
                     const double r[9], double t[3], LfGuard& g) {
  double curl[3];
  matvec_t(r, wv, curl);
  const double o0 = 0.5 * curl[0] - o[0], o1 = 0.5 * curl[1] - o[1], o2 = 0.5 * curl[2] - o[2];
  double tp1 = 0.0, tp2 = 0.0, tr0 = 0.0, tr1 = 0.0, tr2 = 0.0;
  if (s.moving) {
    const double ctp = (0.935 * fw_pow(s.lrep, -0.146) + -0.469 * fw_pow(s.lrep, -0.145)) *
                       fw_pow(s.lsin, 0.116 + 0.748 * fw_pow(s.lrep, 0.041)) *
                       fw_pow(s.lcos, 0.221 + 0.657 * fw_pow(s.lrep, 0.044));
    const double cp = pc.cpitch * ctp * (s.umag * s.umag);
    tp1 = cp * fw_quot(fabs(s.p[2]), s.syz) * copysign(1.0, s.p[0] * s.p[2]);
    tp2 = cp * fw_quot(fabs(s.p[1]), s.syz) * copysign(1.0, s.p[0] * s.p[1]);
  }
  const double ww = o0 * o0 + o1 * o1 + o2 * o2;
  if (ww != 0.0) {
    const double rer = lf_quot(lf_sqrt(ww, g) * (pc.deq * pc.deq), rv);
    const double oyz = fw_sqrt(o2 * o2 + o1 * o1, g);
    const Log2 l = fw_log2(rer, g, -300, 40);
    const double ctr = 0.573 * fw_pow(l, -0.154) + lf_quot(116.61, lf_rcp(rer, g));
    const double ctr2 = 1.244 * fw_pow(l, 0.239) + 378.12 * fw_pow(l, -0.789);
    tr0 = ctr * pc.crot * pc.h5 * fabs(o0) * o0;
    tr1 = ctr2 * pc.crot * pc.h5 * oyz * o1;
    tr2 = ctr2 * pc.crot * pc.h5 * oyz * o2;
  }
  t[0] = 0.0 + tr0;
  t[1] = tp1 + tr1;
  t[2] = tp2 + tr2;
}

// quaternion_integration
GP_LF void fw_quaternion(Quat& q, const double r[9], const double o[3], double dt, LfGuard& g) {
  double w[3];
  matvec(r, o, w);
  const double ww = w[0] * w[0] + w[1] * w[1] + w[2] * w[2];
  if (ww == 0.0) return;
  g.in(ww);
  const LfRcp rn = lf_root(ww);
  double s, c;
  fw_sincos((rn.b * dt) / 2.0, s, c, g);
  const Quat map = {c, s * fw_quot(w[0], rn), s * fw_quot(w[1], rn), s * fw_quot(w[2], rn)};
  q = mult_quat(map, q);
}

// A particle on the way through the integrate: its columns in shared memory, one entry a
// thread (nobody else's business, so no barriers), read again where they are needed instead
// of kept in registers.  The step's own register file is too small for its state, and what
// it spilled went through an L1 that the streamed columns kept flushing: 73 local loads a
// particle, more than 100 cycles each.
constexpr int kIntegrateThreads = 128;
enum { kSlotX = 0, kSlotU = 3, kSlotQ = 6, kSlotO = 10, kSlotConst = 13, kSlotFluid = 23, kSlotWork = 29 };
constexpr int kSlotIn = 29;      // columns read: 13 state, 10 constants, 6 fluid
struct Slot {
  unsigned at;                   // shared-memory address of column 0's entry
  __device__ __forceinline__ double get(int k) const {
    double v;
    asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(at + k * (kIntegrateThreads * 8)));
    return v;
  }
  __device__ __forceinline__ void put(int k, double v) const {
    asm volatile("st.shared.f64 [%0], %1;" ::"r"(at + k * (kIntegrateThreads * 8)), "d"(v) : "memory");
  }
  __device__ __forceinline__ void get3(int k, double v[3]) const {
    v[0] = get(k); v[1] = get(k + 1); v[2] = get(k + 2);
  }
  __device__ __forceinline__ void put3(int k, const double v[3]) const {
    put(k, v[0]); put(k + 1, v[1]); put(k + 2, v[2]);
  }
  __device__ __forceinline__ Quat quat() const { return {get(kSlotQ), get(kSlotQ + 1), get(kSlotQ + 2), get(kSlotQ + 3)}; }
  __device__ __forceinline__ void put_quat(const Quat& q) const {
    put(kSlotQ, q.a); put(kSlotQ + 1, q.b); put(kSlotQ + 2, q.c); put(kSlotQ + 3, q.d);
  }
  __device__ __forceinline__ void get_const(PartConst& c) const {
    c.a = get(13); c.b = get(14); c.deq = get(15); c.cdrag = get(16); c.cpitch = get(17);
    c.crot = get(18); c.h5 = get(19); c.ipxx = get(20); c.ipyy = get(21); c.ipzz = get(22);
  }
};

// Whether the body intersects its wall (or the test fails), for a centre within 1.5 radii
// of it.  Out of line: few particles come here.
static __device__ __noinline__ bool wall_hit(double lx, const PartConst* pc, double x, double y, double z,
                                             const Quat* q) {
  double wn[3], arm[3], dx;
  bool isect;
  return wall_test(lx, *pc, fmax(pc->a, pc->b), x, y, z, *q, wn, arm, dx, isect) != 0 || isect;
}
// wall_test's own early exit first.
GP_LF bool off_wall(double lx, double rmax, double x) { return fabs(x - ((x < lx / 2.0) ? 0.0 : lx)) > 1.5 * rmax; }

// advance_particle<false> away from the walls.  False: not done (the general step starts
// from the pool again).  The slot's quaternion and work columns (six) are overwritten.
GP_LF bool advance_particle_fast(const InstDev& I, const Slot& a, double xn[3], double un[3], double on[3], Quat& qn) {
  LfGuard g;
  const double dt = I.dtime;
  PartConst pc;
  a.get_const(pc);
  const LfRcp rv = lf_rcp(I.visc, g);
  auto spin_rate = [&](const double t[3], const double o[3], double k[3]) {
    k[0] = fw_quot(t[0] + o[1] * o[2] * (pc.ipyy - pc.ipzz), lf_rcp(pc.ipxx, g));
    k[1] = fw_quot(t[1] + o[2] * o[0] * (pc.ipzz - pc.ipxx), lf_rcp(pc.ipyy, g));
    k[2] = fw_quot(t[2] + o[0] * o[1] * (pc.ipxx - pc.ipyy), lf_rcp(pc.ipzz, g));
  };
  auto at_wall = [&](double x, double y, double z, const Quat& q) {
    if (off_wall(I.lx, fmax(pc.a, pc.b), x)) return false;
    PartConst c;
    a.get_const(c);
    const Quat qq = q;
    return wall_hit(I.lx, &c, x, y, z, &qq);
  };
  double f[3], t[3], r[9], k1[3];
  Quat q1 = a.quat();
  rotmat(q1, r);
  {
    SlipFast s;
    double u[3], uf[3];
    a.get3(kSlotU, u);
    a.get3(kSlotFluid, uf);
    fw_slip(pc, rv, u, uf, r, s, g);
    fw_force(pc, s, r, f, g);
    f[2] = f[2] + I.gravity;
    a.put3(kSlotWork, f);
    double wv[3], o[3];
    a.get3(kSlotFluid + 3, wv);
    a.get3(kSlotO, o);
    fw_torque(pc, rv, s, wv, o, r, t, g);
    spin_rate(t, o, k1);
    a.put3(kSlotWork + 3, k1);
  }
  // the predictor's velocity and spin, formed again where they are needed
  auto predicted = [&](int col, int rate, double v[3]) {
#pragma unroll
    for (int i = 0; i < 3; ++i) v[i] = a.get(col + i) + dt * a.get(rate + i);
  };
  double o1[3];
  predicted(kSlotO, kSlotWork + 3, o1);
  fw_quaternion(q1, r, o1, dt, g);
  if (at_wall(a.get(0) + dt * a.get(3), a.get(1) + dt * a.get(4), a.get(2) + dt * a.get(5), q1)) return false;
  a.put_quat(q1);
  rotmat(q1, r);
  {
    SlipFast s;
    double u[3], uf[3];
    predicted(kSlotU, kSlotWork, u);
    a.get3(kSlotFluid, uf);
    fw_slip(pc, rv, u, uf, r, s, g);
    fw_force(pc, s, r, f, g);
  }
  {
    SlipFast s;
    double u[3], uf[3], wv[3];
    a.get3(kSlotU, u);
    a.get3(kSlotFluid, uf);
    fw_slip(pc, rv, u, uf, r, s, g);
    a.get3(kSlotFluid + 3, wv);
    predicted(kSlotO, kSlotWork + 3, o1);
    fw_torque(pc, rv, s, wv, o1, r, t, g);
  }
  double k2o[3];
  spin_rate(t, o1, k2o);
  const double k2u[3] = {f[0], f[1], f[2] + I.gravity};
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const double u = a.get(kSlotU + i), k1u = a.get(kSlotWork + i);
    xn[i] = a.get(i) + 0.5 * dt * (u + (u + dt * k1u));
    un[i] = u + 0.5 * dt * (k1u + k2u[i]);
    on[i] = a.get(kSlotO + i) + 0.5 * dt * (a.get(kSlotWork + 3 + i) + k2o[i]);
  }
  // the spin's quotients are unguarded: both stages' end up here
  g.finite(on[0]); g.finite(on[1]); g.finite(on[2]);
  qn = a.quat();
  if (at_wall(xn[0], xn[1], xn[2], qn)) return false;
  fw_quaternion(qn, r, on, dt, g);
  return g.ok();
}

}  // namespace gp
