// FP64 exp, log, square root, reciprocal and quotient with few FP64
// instructions, for the per-cell thermodynamics.
//
// Those kernels run one to four threads per cell and wait for one serial chain of
// FP64 operations (some 60 to 100 cycles each on GB300).  Here the leading terms stay FP64
// and the series' tails, small against them, are two-float (lacmo_ff.cuh): 11 FP64
// instructions for exp and for log.  Reductions and series are the textbook ones
// (Muller, Elementary Functions, 3rd ed.): exp(x) = 2^k exp(r), |r| <= ln 2 / 2,
// by Taylor's series; log(m) = f - s (f - R), f = m - 1, s = f / (2 + f), R the
// odd series of 2 atanh(s) beyond its first term, over s.  Arguments outside the
// stated range go to the library functions.  The fields they give stay within a
// few roundings of long double over 180 to 420 K (tests/test_gpu_cells64.py).
#pragma once
#include "lacmo_ff.cuh"

namespace lacmo {

// a / b, the quotient's last bits from its residual, and sqrt(x) by one Householder
// iteration from the FP32 reciprocal root (as rcp64), for |b| and x from 2^-125 to
// 2^125 and normal quotients; the library's outside (a state that blew up).
// Compared with the library's functions by tests/test_gpu_math64.py.
LACMO_DEV bool ff_range(double x) {   // 2^-125 <= |x| < 2^125
  return ((uint32_t)__double2hiint(x) & 0x7fffffffu) - (898u << 20) < (250u << 20);
}
static __device__ __noinline__ double div_any(double a, double b) { return a / b; }
static __device__ __noinline__ double sqrt_any(double x) { return sqrt(x); }
LACMO_DEV double rcp64_any(double b) { return ff_range(b) ? rcp64(b) : div_any(1.0, b); }
LACMO_DEV double div64(double a, double b) {
  const double r = rcp64(b), q = __dmul_rn(a, r);
  const double d = __fma_rn(__fma_rn(-q, b, a), r, q);
  const bool normal = ((uint32_t)__double2hiint(d) & 0x7fffffffu) - (1u << 20) < (2045u << 20);
  return ff_range(b) && normal ? d : div_any(a, b);
}
LACMO_DEV double sqrt64(double x) {
  if (!ff_range(x) || x < 0.0) return sqrt_any(x);
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(d2f_int(x)));
  const double z = f2d_int(y), s = __dmul_rn(x, z);
  const double e = __fma_rn(-s, z, 1.0);                 // 2^-21
  return __fma_rn(__dmul_rn(s, e), __fma_rn(e, 0.375, 0.5), s);
}
constexpr double LN2_HI = 0x1.62e42fefa38p-1;            // 41 bits of ln 2
constexpr double LN2_LO = 0x1.ef35793c7673p-45;
LACMO_DEV double exp64(double x) {
  if (!(fabs(x) < 700.0)) return exp(x);
  const double t = __fma_rn(x, 0x1.71547652b82fep+0, 6755399441055744.0);   // x / ln 2
  const int k = __double2loint(t);
  const double kd = __dsub_rn(t, 6755399441055744.0);
  const double r = __fma_rn(kd, -LN2_LO, __fma_rn(kd, -LN2_HI, x));
  const ff f = d2ff(r);
  float u = 1.6059044e-10f;                              // 1/13!
  u = u * f.h + 2.0876757e-09f;
  u = u * f.h + 2.5052108e-08f;
  u = u * f.h + 2.7557319e-07f;
  u = u * f.h + 2.7557319e-06f;                          // 1/9!
  ff s = ff_horner(FFC(1.0 / 40320.0), f, ff{u, 0.0f});
  s = ff_horner(FFC(1.0 / 5040.0), f, s);
  s = ff_horner(FFC(1.0 / 720.0), f, s);
  s = ff_horner(FFC(1.0 / 120.0), f, s);
  double p = __fma_rn(r, ff2d(s), 1.0 / 24.0);
  p = __fma_rn(r, p, 1.0 / 6.0);
  p = __fma_rn(r, p, 0.5);
  const double y = __dadd_rn(1.0, __fma_rn(__dmul_rn(r, r), p, r));
  return __hiloint2double(__double2hiint(y) + (k << 20), __double2loint(y));
}
LACMO_DEV double log64(double x) {
  const uint32_t hx = (uint32_t)__double2hiint(x);
  if (hx - 0x00100000u >= 0x7fe00000u) return log(x);    // not a positive normal number
  // x = 2^e m, sqrt(1/2) <= m < sqrt(2)
  const uint32_t h = hx + (0x3ff00000u - 0x3fe6a09eu);
  const int e = (int)(h >> 20) - 0x3ff;
  const double m = __hiloint2double((int)((h & 0x000fffffu) + 0x3fe6a09eu), __double2loint(x));
  const double f = __dsub_rn(m, 1.0);
  const double s = __dmul_rn(f, rcp64(__dadd_rn(m, 1.0)));
  const ff sf = d2ff(s), z = ff_mul(sf, sf);
  float u = 2.0f / 23.0f;
  u = u * z.h + 2.0f / 21.0f;
  u = u * z.h + 2.0f / 19.0f;
  u = u * z.h + 2.0f / 17.0f;
  u = u * z.h + 2.0f / 15.0f;
  u = u * z.h + 2.0f / 13.0f;
  ff t = ff_horner(FFC(2.0 / 11.0), z, ff{u, 0.0f});
  t = ff_horner(FFC(2.0 / 9.0), z, t);
  t = ff_horner(FFC(2.0 / 7.0), z, t);
  t = ff_horner(FFC(2.0 / 5.0), z, t);
  t = ff_horner(FFC(2.0 / 3.0), z, t);
  const double w = __fma_rn(s, f, -ff2d(ff_mul(ff_mul(sf, z), t)));   // s (f - R)
  const double ed = (double)e;
  return __fma_rn(ed, LN2_HI, __dadd_rn(f, __fma_rn(ed, LN2_LO, -w)));
}

// (the aarch64 compiler fails on these inlined into the four-lane update)
static __device__ __noinline__ double log64_call(double x) { return log64(x); }
static __device__ __noinline__ double exp64_call(double x) { return exp64(x); }

// ---- the cell update of integration.py:402-438 (Theta, r_v) and the fields that
// follow from it (atmosphere.py, update_material_properties :359).  The powers
// go through one logarithm each, pow(x, y) = exp(y log x), with |y log x| below
// 1 (the Exner powers share log x; T^1.94 = T^2 T^-0.06, T^1.5 = T sqrt(T)), so
// that exp's argument carries no more than half an ulp of 1.  Out of line, and
// with every rounding written out: the time step, its start and the adjoint's replay
// run the same code and get the same bits.
static __device__ __noinline__ void cell_step64(double* Th_io, double* rv_io, double rho_d,
                                                double mdi, double L_v0, double dTh, double drv,
                                                double dml, double V, double p_ref_inv) {
  const double Th = __dadd_rn(*Th_io, dTh);
  const double r_v = __dadd_rn(*rv_io, __dadd_rn(drv, -__dmul_rn(dml, mdi)));
  const double L = log64(__dmul_rn(__dmul_rn(__dmul_rn(p_ref_inv, LC_R_D), rho_d), Th));
  const double ToT = exp64(__dmul_rn(LC_KAPPA_FACTOR2, L));
  const double den = __dmul_rn(__dmul_rn(__dmul_rn(LC_C_PD, rho_d), V),
                               __fma_rn(r_v, LC_HEAT_FACTOR_R_V, 1.0));
  *Th_io = __dadd_rn(Th, div64(__dmul_rn(ToT, __dmul_rn(L_v0, dml)), den));
  *rv_io = r_v;
}
struct CellTerms {   // the terms of make_cell_amb (lacmo_physics.cuh)
  double sigw, rhow, lap0, lbp0, c1, c2;
};
LACMO_DEV CellTerms cell_terms64(double T, double p, double e_s, double L_v, double K, double D_v) {
  CellTerms t;
  const double tau = __dsub_rn(1.0, __dmul_rn(T, 1.0 / 647.096));
  t.sigw = __dmul_rn(__dmul_rn(0.2358, exp64(__dmul_rn(1.256, log64(tau)))),
                     __fma_rn(-0.625, tau, 1.0));
  const double d = __dsub_rn(T, LC_PAR_WATER_DENS_2);
  t.rhow = __fma_rn(LC_PAR_WATER_DENS_1, __dmul_rn(d, d), LC_PAR_WATER_DENS_0);
  const double dT = __dsub_rn(T, LC_T_ALPHA_0);
  t.lap0 = div64(__dmul_rn(__fma_rn(LC_C_ALPHA_2, dT, LC_C_ALPHA_1), K), p);
  t.lbp0 = __dmul_rn(__dmul_rn(LC_C_BETA_1, __fma_rn(LC_C_BETA_2, dT, 1.0)), D_v);
  t.c1 = div64(__dmul_rn(L_v, L_v), __dmul_rn(__dmul_rn(__dmul_rn(LC_R_V, K), T), T));
  t.c2 = div64(__dmul_rn(LC_R_V, T), __dmul_rn(D_v, e_s));
  return t;
}
struct CellState {
  double T, p, e_s, S, K, D_v, L_v, mu, rho_f;
  CellTerms t;
};
static __device__ __noinline__ CellState cell_state64(double Th, double r_v, double rho_d,
                                                      double p_ref, double p_ref_inv) {
  CellState a;
  const double L2 = log64(__dmul_rn(__dmul_rn(__dmul_rn(rho_d, Th), LC_R_D), p_ref_inv));
  const double pdr = exp64(__dmul_rn(LC_KAPPA_FACTOR, L2));
  a.T = __dmul_rn(Th, exp64(__dmul_rn(LC_KAPPA_FACTOR * LC_KAPPA_AIR_DRY, L2)));
  a.p = __dmul_rn(__dmul_rn(pdr, p_ref), __fma_rn(r_v, 1.0 / LC_EPSILON_GC, 1.0));
  a.e_s = __dmul_rn(2.53E11, exp64(div64(-5420.0, a.T)));
  a.S = div64(__dmul_rn(__dmul_rn(__dmul_rn(rho_d, r_v), a.T), LC_R_V), a.e_s);
  a.K = __dmul_rn(4.1868E-3, __fma_rn(0.017, __dsub_rn(a.T, 273.15), 5.69));
  const double T2 = __dmul_rn(a.T, a.T);
  a.D_v = div64(__dmul_rn(4.01218E-5, __dmul_rn(T2, exp64(__dmul_rn(-0.06, log64(a.T))))), a.p);
  a.L_v = __dmul_rn(1.0E3, __fma_rn(-2.358, __dsub_rn(a.T, 273.0), 2500.82));
  a.mu = div64(__dmul_rn(1.458E-6, __dmul_rn(a.T, sqrt64(a.T))), __dadd_rn(a.T, 110.4));
  a.rho_f = __dmul_rn(rho_d, __dadd_rn(1.0, r_v));
  a.t = cell_terms64(a.T, a.p, a.e_s, a.L_v, a.K, a.D_v);
  return a;
}
// cell_state64 by four lanes of a warp for each cell (threadIdx.x & 3: role 0 to 3;
// all 32 lanes take part), bit for bit: logarithms, exponentials and quotients that
// do not depend on each other run side by side, one in each lane, so the chain of
// FP64 operations a cell waits for is less than half of one thread's.  irho and
// kelvin: see write_rec64.
LACMO_DEV CellState cell_state64_x4(double Th, double r_v, double rho_d, double p_ref,
                                    double p_ref_inv, double* irho, double* kelvin) {
  const int lane = threadIdx.x & 31, role = lane & 3;
  auto from = [&](double v, int r) { return __shfl_sync(0xffffffffu, v, (lane & 28) | r); };
  auto pick = [&](double a0, double a1, double a2, double a3) {
    return role < 2 ? (role ? a1 : a0) : (role == 2 ? a2 : a3);
  };
  CellState a;
  const double L2 = log64_call(__dmul_rn(__dmul_rn(__dmul_rn(rho_d, Th), LC_R_D), p_ref_inv));
  const double e0 =
      exp64_call(__dmul_rn(role ? LC_KAPPA_FACTOR * LC_KAPPA_AIR_DRY : LC_KAPPA_FACTOR, L2));
  const double T = a.T = __dmul_rn(Th, from(e0, 1));
  a.p = __dmul_rn(__dmul_rn(from(e0, 0), p_ref), __fma_rn(r_v, 1.0 / LC_EPSILON_GC, 1.0));
  a.K = __dmul_rn(4.1868E-3, __fma_rn(0.017, __dsub_rn(T, 273.15), 5.69));
  a.L_v = __dmul_rn(1.0E3, __fma_rn(-2.358, __dsub_rn(T, 273.0), 2500.82));
  const double T2 = __dmul_rn(T, T), RvT = __dmul_rn(LC_R_V, T);
  const double tau = __dsub_rn(1.0, __dmul_rn(T, 1.0 / 647.096));
  const double d = __dsub_rn(T, LC_PAR_WATER_DENS_2);
  a.t.rhow = __fma_rn(LC_PAR_WATER_DENS_1, __dmul_rn(d, d), LC_PAR_WATER_DENS_0);
  *irho = rcp64_any(a.t.rhow);
  const double dT = __dsub_rn(T, LC_T_ALPHA_0);
  // -5420 / T, mu, lap0, c1
  const double q1 = div64(
      pick(-5420.0, __dmul_rn(1.458E-6, __dmul_rn(T, sqrt64(T))),
           __dmul_rn(__fma_rn(LC_C_ALPHA_2, dT, LC_C_ALPHA_1), a.K), __dmul_rn(a.L_v, a.L_v)),
      pick(T, __dadd_rn(T, 110.4), a.p, __dmul_rn(__dmul_rn(__dmul_rn(LC_R_V, a.K), T), T)));
  const double lg = log64_call(role == 2 ? tau : T);
  const double e1 = exp64_call(pick(q1, __dmul_rn(-0.06, lg), __dmul_rn(1.256, lg), 0.0));
  a.e_s = __dmul_rn(2.53E11, from(e1, 0));
  a.t.sigw = __dmul_rn(__dmul_rn(0.2358, from(e1, 2)), __fma_rn(-0.625, tau, 1.0));
  // S, D_v, the Kelvin term
  const double q2 = div64(
      pick(__dmul_rn(__dmul_rn(__dmul_rn(rho_d, r_v), T), LC_R_V),
           __dmul_rn(4.01218E-5, __dmul_rn(T2, e1)), __dmul_rn(__dmul_rn(2.0E6, a.t.sigw), *irho),
           1.0),
      pick(a.e_s, a.p, RvT, 1.0));
  a.S = from(q2, 0);
  a.D_v = from(q2, 1);
  *kelvin = from(q2, 2);
  a.t.c2 = div64(RvT, __dmul_rn(a.D_v, a.e_s));
  a.mu = from(q1, 1);
  a.t.lap0 = from(q1, 2);
  a.t.c1 = from(q1, 3);
  a.t.lbp0 = __dmul_rn(__dmul_rn(LC_C_BETA_1, __fma_rn(LC_C_BETA_2, dT, 1.0)), a.D_v);
  a.rho_f = __dmul_rn(rho_d, __dadd_rn(1.0, r_v));
  return a;
}
// the FP64 path's record of a cell; irho = rcp64_any(rho_w), kelvin: kelvin_term64
LACMO_DEV double kelvin_term64(double T, double sigw, double irho) {
  return div64(__dmul_rn(__dmul_rn(2.0E6, sigw), irho), __dmul_rn(LC_R_V, T));
}
static __device__ __noinline__ void write_rec64(CellFF* out, double T, double S, double L_v,
                                                double mu, double rho_f, CellTerms t, double irho,
                                                double kelvin) {
  CellFF r;
  r.S_m1 = __dsub_rn(S, 1.0);
  r.cx = d2ff(__dmul_rn(LC_FOUR_PI_OVER_THREE_INV, irho));
  r.ce = d2ff(kelvin);
  r.la = d2ff(t.lap0); r.lb = d2ff(t.lbp0); r.c1 = d2ff(t.c1); r.c2 = d2ff(t.c2);
  const double n0 = __fma_rn(__fma_rn(LC_PAR_SOL_DENS_NACL_5, T, LC_PAR_SOL_DENS_NACL_2), T,
                             LC_PAR_SOL_DENS_NACL_0);
  r.n0 = d2ff(__dmul_rn(n0, irho));
  r.n1 = d2ff(__dmul_rn(__fma_rn(LC_PAR_SOL_DENS_NACL_4, T, LC_PAR_SOL_DENS_NACL_1), irho));
  r.n3 = d2ff(__dmul_rn(LC_PAR_SOL_DENS_NACL_3, irho));
  r.mr = d2ff(__dmul_rn(mu, irho));
  r.rm = d2f_int(rho_f) * f_rcp(d2f_int(mu));
  r.pad0 = 0.0f;
  r.L_v = L_v;
  r.pad[0] = r.pad[1] = r.pad[2] = 0.0;
  *out = r;
}
static __device__ __noinline__ void write_rec64(CellFF* out, double T, double S, double L_v,
                                                double mu, double rho_f, CellTerms t) {
  const double irho = rcp64_any(t.rhow);
  write_rec64(out, T, S, L_v, mu, rho_f, t, irho, kelvin_term64(T, t.sigw, irho));
}

}  // namespace lacmo
