// Two-float arithmetic for the FP64 particle path.
//
// GB300 issues FP64 at 1/64 of the FP32 rate, so a value held as an unevaluated
// sum of two floats (h + l, 48 bits) and combined by error-free
// transformations (Dekker 1971, Knuth TAOCP 2, 4.2.2) costs 7 to 11 FP32
// instructions per operation where one FP64 instruction takes as many issue
// slots as 64 of them.  Used where a relative error of some 2^-46 of an
// intermediate cannot reach the result's last bits: increments and corrections
// that are added to FP64 values they are small against.  Sums and products that
// must round like FP64 stay FP64 (newton_ff below names them).
// The intrinsics keep the compiler from contracting or reordering.
#pragma once
#include "lacmo_physics.cuh"

namespace lacmo {

struct ff {
  float h, l;
};
// a double constant as two floats (folded by the compiler)
#define FFC(x) (ff{(float)(x), (float)((x) - (double)(float)(x))})
LACMO_DEV float fm(float a, float b) { return __fmul_rn(a, b); }
LACMO_DEV float fa(float a, float b) { return __fadd_rn(a, b); }
LACMO_DEV float fs(float a, float b) { return __fsub_rn(a, b); }
LACMO_DEV float fma_(float a, float b, float c) { return __fmaf_rn(a, b, c); }
// s + e = a + b exactly; ff_quick for |a| >= |b|
LACMO_DEV ff ff_quick(float a, float b) {
  const float s = fa(a, b);
  return ff{s, fs(b, fs(s, a))};
}
LACMO_DEV ff ff_sum(float a, float b) {
  const float s = fa(a, b), bb = fs(s, a);
  return ff{s, fa(fs(a, fs(s, bb)), fs(b, bb))};
}
LACMO_DEV ff ff_neg(ff a) { return ff{-a.h, -a.l}; }
LACMO_DEV ff ff_mul(ff a, ff b) {   // relative error below 2^-45
  const float p = fm(a.h, b.h);
  float e = fma_(a.h, b.h, -p);
  e = fma_(a.h, b.l, e);
  e = fma_(a.l, b.h, e);
  return ff_quick(p, e);
}
LACMO_DEV ff ff_mul(ff a, float b) {
  const float p = fm(a.h, b);
  return ff_quick(p, fma_(a.l, b, fma_(a.h, b, -p)));
}
// a + b within 2^-46 (|a| + |b|)
LACMO_DEV ff ff_add(ff a, ff b) {
  const ff s = ff_sum(a.h, b.h);
  return ff_quick(s.h, fa(s.l, fa(a.l, b.l)));
}
LACMO_DEV ff ff_add(ff a, float b) {
  const ff s = ff_sum(a.h, b);
  return ff_quick(s.h, fa(s.l, a.l));
}
LACMO_DEV ff ff_sub(ff a, ff b) { return ff_add(a, ff_neg(b)); }
// c + a b for a constant c with |c| >= |a b|
LACMO_DEV ff ff_horner(ff c, ff a, ff b) {
  const ff p = ff_mul(a, b);
  const ff s = ff_quick(c.h, p.h);
  return ff_quick(s.h, fa(s.l, fa(c.l, p.l)));
}
LACMO_DEV ff ff_one_plus(ff a) {   // |a| <= 1
  const ff s = ff_quick(1.0f, a.h);
  return ff_quick(s.h, fa(s.l, a.l));
}
// 1 / b: the approximate reciprocal and its residual to second order
LACMO_DEV ff ff_rcp(ff b) {
  const float y = f_rcp(b.h);
  float e = fma_(-b.h, y, 1.0f);
  e = fma_(-b.l, y, e);
  e = fma_(e, e, e);
  return ff_quick(y, fm(y, e));
}
// x^(-1/3), x > 0: 2^(-log2(x) / 3), one FP32 Newton step, then the residual
// 1 - x z^3 in two floats to second order
LACMO_DEV ff ff_icbrt(ff x) {
  float z = f_ex2(f_lg2(x.h) * (-1.0f / 3.0f));
  z = fma_(fm(z, 1.0f / 3.0f), fma_(-fm(x.h, z), fm(z, z), 1.0f), z);
  const float q = fm(z, z);
  const ff t = ff_mul(ff_mul(ff{q, fma_(z, z, -q)}, z), x);
  const float e = fs(fs(1.0f, t.h), t.l);
  return ff_quick(z, fm(fm(z, e), fma_(e, 2.0f / 9.0f, 1.0f / 3.0f)));
}
// expm1(e) for |e| < 0.25 by its Taylor series, the tail from e^8 on in FP32
LACMO_DEV ff ff_expm1(ff e) {
  float t = 2.5052108e-08f;                      // 1/11!
  t = t * e.h + 2.7557319e-07f;                  // 1/10!
  t = t * e.h + 2.7557319e-06f;                  // 1/9!
  t = t * e.h + 2.4801587e-05f;                  // 1/8!
  ff s = ff_horner(FFC(1.0 / 5040.0), e, ff{t, 0.0f});
  s = ff_horner(FFC(1.0 / 720.0), e, s);
  s = ff_horner(FFC(1.0 / 120.0), e, s);
  s = ff_horner(FFC(1.0 / 24.0), e, s);
  s = ff_horner(FFC(1.0 / 6.0), e, s);
  s = ff_horner(ff{0.5f, 0.0f}, e, s);
  return ff_mul(e, ff_one_plus(ff_mul(e, s)));
}
// x split after its 24th bit with integer operations; the low part keeps 24
// more of the 29 bits left (0 below 2^-75; NaN beyond the FP32 range)
LACMO_DEV ff d2ff(double x) {
  const uint32_t hi = (uint32_t)__double2hiint(x), lo = (uint32_t)__double2loint(x);
  const uint32_t ax = hi & 0x7fffffffu, sign = hi & 0x80000000u;
  const uint32_t f = __funnelshift_l(lo, ax, 3) - (384u << 23);
  const uint32_t ef = f >> 23;
  const float sc = __uint_as_float(((ef > 53u ? ef - 52u : 0u) << 23) | sign);
  ff r;
  r.h = __uint_as_float(ax < (897u << 20) ? sign
                                          : (ax < (1151u << 20) ? f | sign : 0x7fffffffu));
  r.l = ax < (897u << 20) || ax >= (1151u << 20) ? 0.0f
                                                 : fm((float)(lo & 0x1fffffffu), sc);
  return r;
}
LACMO_DEV double ff2d(ff a) { return f2d_int(a.h) + f2d_int(a.l); }
// The same bits without an FP64 instruction, |l| <= ulp(h) / 2: l in units of h's 53-bit ulp (half
// of it below a power of two), rounded by the conversion to integer, added to h's
// bits.  Some 18 integer instructions where one FP64 addition takes the SM's FP64
// pipe for as long as 64 of them; for kernels that fill that pipe (its chain is some
// tens of cycles longer than the addition's).
LACMO_DEV double ff2d_int(ff a) {
  const uint32_t hb = __float_as_uint(a.h), eh = (hb >> 23) & 0xffu;
  if (eh - 55u >= 200u) return ff2d(a);   // 0, below 2^-72 (l may be subnormal), not finite
  const uint32_t lb = __float_as_uint(a.l) ^ (hb & 0x80000000u);   // l away from zero
  const uint32_t below = (hb & 0x007fffffu) == 0u ? lb >> 31 : 0u;
  const int k = __float2int_rn(fm(__uint_as_float(lb), __uint_as_float((306u + below - eh) << 23)));
  return __longlong_as_double(__double_as_longlong(f2d_int(a.h)) + (long long)k);
}

// ---------------------------------------------------------------------------
// A cell's terms for the FP64 particle sub-step: one record of 128 bytes
// (write_aux), and its wind as base values and differences (write_wind), another
// 128 bytes.
struct CellFF {
  double S_m1;      // S - 1
  ff cx;            // 3 / (4 pi rho_w)
  ff ce;            // 2e6 sigma_w / (R_v T rho_w)
  ff la, lb, c1, c2;
  ff n0, n1, n3;    // NaCl solution density over rho_w: n0 + n1 w + n3 w^2
  ff mr;            // mu / rho_w
  float rm, pad0;   // rho_f / mu
  double L_v;       // heat of vaporisation
  double pad[3];
};
struct WindFF {
  double U0[2];     // u at (i, j - 1), (i, j)
  double dxU[3];    // u(i + 1, j - 1 + b) - u(i, j - 1 + b)
  double dyU[2];    // u(i, j + b) - u(i, j - 1 + b)
  double V0[2];     // w at (i - 1, j), (i, j)
  double dyV[3];    // w(i - 1 + a, j + 1) - w(i - 1 + a, j)
  double dxV[2];    // w(i + a, j) - w(i - 1 + a, j)
  int32_t i, j, edge, pad;   // edge: bit 0 bottom row, bit 1 top row
};
static_assert(sizeof(CellFF) == 128 && sizeof(WindFF) == 128, "one line each");

// Mass rate and derivative of microphysics.py:1359-1469 (AS) and :1239-1353
// (NaCl) at mass m, as dt gamma and dt dgamma/dm.  FP64: the total mass, the
// solute fraction w, the water activity and S_eq - 1 = (a_w - 1) + a_w
// expm1(eps), and the residual f2 = (S - 1) - (S_eq - 1), whose cancellation
// they decide (S and S_eq themselves are never formed, so f2 loses less than a
// difference of numbers near 1).  Two floats: everything that scales f2 or its
// derivative, with the common factor 1 / m_p taken out:
//   q = m_s / m, u = w rho'(w) / rho, v = R (1 + u) / 3, A = R + l_alpha, ...
//   D = m_p dS_eq/dm = -w a_w'(w) e^eps + S_eq eps (-s1 q (1 + q) / (1 + s2 q)
//       + (2u - 1) / 3)
//   dt gamma = G f2, G = 4 pi 1e12 dt R^2 / den, den = A S_eq c1 + B c2
//   dt gamma' = G / m_p (f2 (2 (1 + u) / 3 - ((D A + S_eq v) c1 + v c2) / den) - D)
// nacl_rho: density and surface tension of the NaCl solution (the first
// evaluation; the reference's iterations use those of ammonium sulfate).
// ks scales a_w - 1 (KS; the adjoint's hygroscopicity).
// Returns false when eps leaves the series' range (0.25; R below some 5 nm).
// FULL: for a full FP64 pipe (ff2d_int).
template <bool FULL>
LACMO_DEV double ff2d_of(ff a) { return FULL ? ff2d_int(a) : ff2d(a); }
template <bool KS, bool FULL>
LACMO_DEV bool mass_rate_ff(int sol, bool nacl_rho, double m, double ms, ff msf, const CellFF& c,
                            ff gdt, double ks, ff& gd, ff& x) {
  const double mp = m + ms;
  const ff imp = ff_rcp(d2ff(mp));
  const ff wf = ff_mul(msf, imp);
  double w = ff2d_of<FULL>(wf);
  w = fma(fma(-w, mp, ms), f2d_int(imp.h), w);   // m_s / m_p, one correction
  const ff q = ff_mul(msf, ff_rcp(d2ff(m)));
  ff pr, pd, da;
  double aw_m1;
  if (sol == SOL_AS) {
    aw_m1 = w * (((LC_PAR_WAT_ACT_AS_0 * w + LC_PAR_WAT_ACT_AS_1) * w + LC_PAR_WAT_ACT_AS_2) * w +
                 LC_PAR_WAT_ACT_AS_3);
    da = ff_add(FFC(LC_PAR_WAT_ACT_DERIV_AS_1), ff_mul(FFC(LC_PAR_WAT_ACT_DERIV_AS_0), wf));
    da = ff_add(FFC(LC_PAR_WAT_ACT_DERIV_AS_2), ff_mul(da, wf));
    da = ff_add(FFC(LC_PAR_WAT_ACT_DERIV_AS_3), ff_mul(da, wf));
    pd = ff_horner(FFC(LC_PAR_RHO_DERIV_AS_1), FFC(LC_PAR_RHO_DERIV_AS_0), wf);
    pd = ff_horner(FFC(LC_PAR_RHO_DERIV_AS_2), pd, wf);
  } else {
    aw_m1 = w * (((LC_PAR_WAT_ACT_NACL_0 * w + LC_PAR_WAT_ACT_NACL_1) * w +
                  LC_PAR_WAT_ACT_NACL_2) * w + LC_PAR_WAT_ACT_NACL_3);
    da = ff_add(FFC(LC_PAR_WAT_ACT_DERIV_NACL_1), ff_mul(FFC(LC_PAR_WAT_ACT_DERIV_NACL_0), wf));
    da = ff_add(FFC(LC_PAR_WAT_ACT_DERIV_NACL_2), ff_mul(da, wf));
    da = ff_add(FFC(LC_PAR_WAT_ACT_DERIV_NACL_3), ff_mul(da, wf));
    pd = ff_add(c.n1, ff_mul(ff{2.0f * c.n3.h, 2.0f * c.n3.l}, wf));
  }
  if (nacl_rho) {
    pr = ff_add(c.n0, ff_mul(ff_add(c.n1, ff_mul(c.n3, wf)), wf));
  } else {
    pr = ff_horner(FFC(LC_PAR_RHO_AS_1), FFC(LC_PAR_RHO_AS_0), wf);
    pr = ff_horner(FFC(LC_PAR_RHO_AS_2), pr, wf);
    pr = ff_one_plus(ff_mul(pr, wf));
  }
  if (KS) {
    aw_m1 *= ks;
    da = ff_mul(da, d2ff(ks));
  }
  const float s1h = sol == SOL_AS ? FFC(LC_PAR_SIGMA_AS).h : FFC(LC_PAR_SIGMA_NACL).h;
  const float s1l = sol == SOL_AS ? FFC(LC_PAR_SIGMA_AS).l : FFC(LC_PAR_SIGMA_NACL).l;
  const ff s1 = {s1h, s1l};
  const ff s1q = ff_mul(s1, q);
  // sigma / sigma_w = 1 + s2 q; s2 is that of ammonium sulfate in the iterations
  const ff sg = ff_add((nacl_rho || sol == SOL_AS) ? s1q : ff_mul(FFC(LC_PAR_SIGMA_AS), q), 1.0f);
  const ff ipr = ff_rcp(pr);
  const ff xr = ff_mul(ff_mul(c.cx, d2ff(mp)), ipr);
  const ff z = ff_icbrt(xr);                       // 1 / R
  const ff R = ff_mul(ff_mul(xr, z), z);
  const ff eps = ff_mul(ff_mul(c.ce, sg), ff_mul(ipr, z));
  const ff em1 = ff_expm1(eps);
  const double sm1 = fma(1.0 + aw_m1, ff2d_of<FULL>(em1), aw_m1);   // S_eq - 1
  const double f2d_ = c.S_m1 - sm1;
  const ff f2 = d2ff(f2d_);
  const ff Seq = ff_add(d2ff(sm1), 1.0f);
  const ff u = ff_mul(ff_mul(wf, pd), ipr);
  const ff t13 = ff_mul(ff_add(u, 1.0f), FFC(1.0 / 3.0));
  const ff v = ff_mul(R, t13);
  const ff A = ff_add(c.la, R), B = ff_add(c.lb, R);
  const ff y = ff_mul(ff_mul(s1q, ff_add(q, 1.0f)), ff_rcp(sg));
  // (2u - 1) / 3 = 2 (1 + u) / 3 - 1
  const ff z3 = ff_sub(ff_add(ff{2.0f * t13.h, 2.0f * t13.l}, -1.0f), y);
  const ff D = ff_sub(ff_mul(ff_mul(Seq, eps), z3),
                      ff_mul(ff_mul(wf, da), ff_one_plus(em1)));
  const ff iden = ff_rcp(ff_add(ff_mul(ff_mul(A, Seq), c.c1), ff_mul(B, c.c2)));
  const ff num = ff_add(ff_mul(ff_add(ff_mul(D, A), ff_mul(Seq, v)), c.c1), ff_mul(v, c.c2));
  const ff G = ff_mul(ff_mul(gdt, ff_mul(R, R)), iden);
  const ff k1 = ff_sub(ff{2.0f * t13.h, 2.0f * t13.l}, ff_mul(num, iden));
  const ff k2 = ff_sub(ff_mul(f2, k1), D);
  gd = ff_mul(G, f2);
  x = ff_mul(ff_mul(G, imp), k2);
  return eps.h < 0.25f;
}
LACMO_DEV ff damp_ff(ff x) {   // 1 / (1 - x) for x < 0.9, else 10
  const ff r = ff_rcp(ff_add(ff_neg(x), 1.0f));
  return x.h < 0.9f ? r : ff{10.0f, 0.0f};
}
// masses the two-float arithmetic takes: 2^-60 <= m < 2^97, not NaN
LACMO_DEV bool ff_mass_ok(double m) {
  return (uint32_t)__double2hiint(m) - 0x3c300000u < 0x09d00000u;
}
// The damped Newton of integration.py:728-836 (newton_full) in this arithmetic:
// the new mass.  ok is false when a step left the arithmetic's range, or moved
// the mass by more than an eighth of it: the scale of the step, good to some
// 2^-44, then shows in the mass (the caller repeats in FP64).  Against the same
// map in 64-bit mantissas (80,000 SIPs of fresh and raining states, AS and NaCl)
// the masses are off by 0.3 to 0.9 of newton_full's error in every range of
// step sizes below an eighth, and by 1.3 to 10 of it above.
template <bool KS, bool FULL>
LACMO_DEV double newton_ff(int sol, int no_iter, double m_w, double m_s, const CellFF& c, ff gdt,
                           double ks, bool* ok) {
  const double floor_m = m_s * (LC_W_S_MAX_AS_INV - 1.0);
  const ff msf = d2ff(m_s);
  ff gd, x;
  bool good = mass_rate_ff<KS, FULL>(sol, sol != SOL_AS, m_w, m_s, msf, c, gdt, ks, gd, x);
  // np_max for a positive floor by the bits; NaN and infinity clear good
  auto floored = [&](double m) {
    good = good && (uint32_t)((__double2hiint(m) >> 20) & 0x7ff) != 0x7ffu;
    return __double_as_longlong(m) > __double_as_longlong(floor_m) ? m : floor_m;
  };
  double m = floored(m_w + ff2d_of<FULL>(ff_mul(gd, damp_ff(x))));
  for (int it = 0;;) {
    const ff d = d2ff(m - m_w);
    good = good && fabsf(d.h) <= 0.125f * d2f_int(m);
    if (++it >= no_iter) break;
    good = mass_rate_ff<KS, FULL>(sol, false, m, m_s, msf, c, gdt, ks, gd, x) && good;
    m = floored(m + ff2d_of<FULL>(ff_mul(ff_sub(gd, d), damp_ff(x))));
  }
  *ok = good && ff_mass_ok(m_w) && ff_mass_ok(m_s) && m < 1e29;
  return m;
}

// ---------------------------------------------------------------------------
// The same Newton in plain FP64 with few instructions, for SIPs whose step needs
// all 53 bits: reciprocals and the cube root from FP32 seeds (2^-22) and one
// Householder iteration (Householder, The Numerical Treatment of a Single Nonlinear
// Equation, 1970): with the residual e of the seed, the binomial series of
// (1 - e)^-1 and (1 - e)^(-1/3) to second and third order.  The differences from
// saturation and the factored derivative of mass_rate_ff; about 100 FP64
// instructions an evaluation where mass_rate_and_derivative takes some 220.
LACMO_DEV double rcp64(double b) {
  const double y = f2d_int(f_rcp(d2f_int(b)));
  double e = fma(-b, y, 1.0);
  e = fma(e, e, e);
  return fma(y, e, y);
}
LACMO_DEV double icbrt64(double x) {   // x^(-1/3), x > 0
  const float xf = d2f_int(x);
  float zf = f_ex2(f_lg2(xf) * (-1.0f / 3.0f));
  zf = fma_(fm(zf, 1.0f / 3.0f), fma_(-fm(xf, zf), fm(zf, zf), 1.0f), zf);
  const double z = f2d_int(zf);
  const double e = fma(-x, (z * z) * z, 1.0);
  return fma(z, e * fma(e, fma(e, 14.0 / 81.0, 2.0 / 9.0), 1.0 / 3.0), z);
}
struct CellFast {
  double S_m1, cx, ce, la, lb, c1, c2;
  double n0, n1, n3;   // NaCl: solution density over rho_w
};
LACMO_DEV CellFast cell_fast(int sol, const CellAmb& a) {
  CellFast c;
  const double ir = 1.0 / a.rhow;
  c.S_m1 = a.S - 1.0;
  c.cx = LC_FOUR_PI_OVER_THREE_INV * ir;
  c.ce = 2.0E6 * a.sigw / (LC_R_V * a.T * a.rhow);
  c.la = a.lap0; c.lb = a.lbp0; c.c1 = a.c1; c.c2 = a.c2;
  c.n0 = c.n1 = c.n3 = 0.0;
  if (sol != SOL_AS) {
    c.n0 = (LC_PAR_SOL_DENS_NACL_0 + LC_PAR_SOL_DENS_NACL_2 * a.T +
            LC_PAR_SOL_DENS_NACL_5 * a.T * a.T) * ir;
    c.n1 = (LC_PAR_SOL_DENS_NACL_1 + LC_PAR_SOL_DENS_NACL_4 * a.T) * ir;
    c.n3 = LC_PAR_SOL_DENS_NACL_3 * ir;
  }
  return c;
}
LACMO_DEV void mass_rate_fast(int sol, bool nacl_rho, double m, double ms, const CellFast& c,
                              double gdt, double ks, double& gd, double& x) {
  const double mp = m + ms;
  const double imp = rcp64(mp);
  const double w0 = ms * imp, w = fma(fma(-w0, mp, ms), imp, w0);
  const double q = ms * rcp64(m);
  double P, da, pd, pr;
  if (sol == SOL_AS) {
    P = w * (((LC_PAR_WAT_ACT_AS_0 * w + LC_PAR_WAT_ACT_AS_1) * w + LC_PAR_WAT_ACT_AS_2) * w +
             LC_PAR_WAT_ACT_AS_3);
    da = ((LC_PAR_WAT_ACT_DERIV_AS_0 * w + LC_PAR_WAT_ACT_DERIV_AS_1) * w +
          LC_PAR_WAT_ACT_DERIV_AS_2) * w + LC_PAR_WAT_ACT_DERIV_AS_3;
    pd = (LC_PAR_RHO_DERIV_AS_0 * w + LC_PAR_RHO_DERIV_AS_1) * w + LC_PAR_RHO_DERIV_AS_2;
  } else {
    P = w * (((LC_PAR_WAT_ACT_NACL_0 * w + LC_PAR_WAT_ACT_NACL_1) * w +
              LC_PAR_WAT_ACT_NACL_2) * w + LC_PAR_WAT_ACT_NACL_3);
    da = ((LC_PAR_WAT_ACT_DERIV_NACL_0 * w + LC_PAR_WAT_ACT_DERIV_NACL_1) * w +
          LC_PAR_WAT_ACT_DERIV_NACL_2) * w + LC_PAR_WAT_ACT_DERIV_NACL_3;
    pd = c.n1 + 2.0 * c.n3 * w;
  }
  pr = nacl_rho ? c.n0 + (c.n1 + c.n3 * w) * w
                : ((LC_PAR_RHO_AS_0 * w + LC_PAR_RHO_AS_1) * w + LC_PAR_RHO_AS_2) * w +
                      LC_PAR_RHO_AS_3;
  P *= ks;
  da *= ks;
  const double s1 = sol == SOL_AS ? LC_PAR_SIGMA_AS : LC_PAR_SIGMA_NACL;
  const double sg = fma(nacl_rho ? s1 : LC_PAR_SIGMA_AS, q, 1.0);
  const double ipr = rcp64(pr);
  const double xr = c.cx * mp * ipr;
  const double z = icbrt64(xr), R = xr * z * z;
  const double eps = c.ce * sg * (ipr * z);
  double em1;
  if (eps < 0.25) {
    // eps + eps^2 s(eps): the series in two floats
    const ff e = d2ff(eps);
    float t = 2.7557319e-07f;                      // 1/10!
    t = t * e.h + 2.7557319e-06f;                  // 1/9!
    t = t * e.h + 2.4801587e-05f;                  // 1/8!
    ff s = ff_horner(FFC(1.0 / 5040.0), e, ff{t, 0.0f});
    s = ff_horner(FFC(1.0 / 720.0), e, s);
    s = ff_horner(FFC(1.0 / 120.0), e, s);
    s = ff_horner(FFC(1.0 / 24.0), e, s);
    s = ff_horner(FFC(1.0 / 6.0), e, s);
    s = ff_horner(ff{0.5f, 0.0f}, e, s);
    em1 = fma(eps * eps, ff2d(s), eps);
  } else {
    em1 = expm1(eps);
  }
  const double sm1 = fma(1.0 + P, em1, P);
  const double f2 = c.S_m1 - sm1, Seq = 1.0 + sm1;
  const double u = w * pd * ipr, t = fma(u, LC_ONE_THIRD, LC_ONE_THIRD), v = R * t;
  const double A = c.la + R, B = c.lb + R;
  const double y = s1 * q * (1.0 + q) * rcp64(sg);
  const double D = Seq * eps * (2.0 * t - 1.0 - y) - w * da * (1.0 + em1);
  const double iden = rcp64(A * Seq * c.c1 + B * c.c2);
  const double N = (D * A + Seq * v) * c.c1 + v * c.c2;
  const double G = gdt * (R * R) * iden;
  gd = G * f2;
  x = G * imp * (f2 * (2.0 * t - N * iden) - D);
}
LACMO_DEV double damp64(double x) { return x < 0.9 ? rcp64(1.0 - x) : 10.0; }
// newton_full's new mass; masses outside the two-float range take newton_full
LACMO_DEV double newton_fast(int sol, double dt, int no_iter, double m_w, double m_s,
                             const CellFast& c, double ks) {
  const double floor_m = m_s * (LC_W_S_MAX_AS_INV - 1.0);
  const double gdt = LC_FOUR_PI * 1.0E12 * dt;
  double gd, x;
  mass_rate_fast(sol, sol != SOL_AS, m_w, m_s, c, gdt, ks, gd, x);
  double m = np_max(floor_m, m_w + gd * damp64(x));
#pragma unroll 1
  for (int it = 1; it < no_iter; ++it) {
    mass_rate_fast(sol, false, m, m_s, c, gdt, ks, gd, x);
    m = np_max(floor_m, m + (gd + m_w - m) * damp64(x));
  }
  return m;
}

}  // namespace lacmo
