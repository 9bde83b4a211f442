// Hand-written adjoint of the condensation sub-steps with their cell heat and
// vapour feedback and the grid advection of Theta and r_v (integration.py:
// 840-940 with the Newton of :728-836, the grid update of :402-484 and the
// advective increments of :80-287, 1483-1508, 1536-1561), for gradients of
// liquid water and surface rain with respect to per-SIP solute mass,
// hygroscopicity and the strength of the prescribed mass flux.
//
// Differentiated model: the SIPs' cells per sub-step and their multiplicities
// are recorded events (positions, ground removal and collisions are held
// fixed; SIP motion reaches condensation only through the piecewise constant
// cell index); every sub-step runs the condensation step of each SIP, either
// the time step's own map of no_iter damped Newton evaluations (the product's
// map, differentiated exactly with forward-mode duals through every
// evaluation, second derivatives included) or the implicit Euler step solved
// to convergence (implicit-function theorem), and then updates Theta and r_v
// of each cell from the condensed mass and the half step's advective (+
// relaxation) increments, with all ambient terms (T, p, S, e_s, K, D_v, L_v,
// sigma_w, rho_w) functions of the cell's Theta and r_v.  The reference sets a
// SIP's temperature to its cell's at the start of every sub-step
// (integration.py:1059-1060), so T_p is the ambient T here.
// Hygroscopicity: the ammonium-sulfate water activity a_w(w_s) (material_
// properties.py:429-436) becomes 1 + (kappa / 0.6) (a_w(w_s) - 1), so kappa =
// 0.6 reproduces the reference.
//
// Reverse sweep per sub-step: the time step's map is differentiated backwards
// through its evaluations (mass_rate_rev below), in the two-float arithmetic the
// time step runs in (lacmo_ff.cuh); the converged step, and SIPs outside that
// arithmetic's range, take forward-mode dual numbers in FP64.  A cell's ambient
// terms and their derivatives by Theta and r_v are formed once per cell and
// sub-step; the cell update's Jacobian comes from duals, the increments' from
// duals through the limited face fluxes.  Sums over a cell's SIPs use atomics
// (FP64).
#include <cuda_runtime.h>

#include "lacmo_ff.cuh"
#include "lacmo_internal.cuh"
#include "lacmo_math64.cuh"
#include "lacmo_physics.cuh"

namespace lacmo {
namespace adj {

// ---- dual numbers: value and N partial derivatives ----
template <int N>
struct Dual {
  double v;
  double d[N];
};
template <int N>
__device__ __forceinline__ Dual<N> cst(double v) {
  Dual<N> r; r.v = v;
#pragma unroll
  for (int i = 0; i < N; ++i) r.d[i] = 0.0;
  return r;
}
template <int N>
__device__ __forceinline__ Dual<N> var(double v, int k) {
  Dual<N> r = cst<N>(v); r.d[k] = 1.0; return r;
}
template <int N>
__device__ __forceinline__ Dual<N> operator+(const Dual<N>& a, const Dual<N>& b) {
  Dual<N> r; r.v = a.v + b.v;
#pragma unroll
  for (int i = 0; i < N; ++i) r.d[i] = a.d[i] + b.d[i];
  return r;
}
template <int N>
__device__ __forceinline__ Dual<N> operator-(const Dual<N>& a, const Dual<N>& b) {
  Dual<N> r; r.v = a.v - b.v;
#pragma unroll
  for (int i = 0; i < N; ++i) r.d[i] = a.d[i] - b.d[i];
  return r;
}
template <int N>
__device__ __forceinline__ Dual<N> operator*(const Dual<N>& a, const Dual<N>& b) {
  Dual<N> r; r.v = a.v * b.v;
#pragma unroll
  for (int i = 0; i < N; ++i) r.d[i] = a.d[i] * b.v + a.v * b.d[i];
  return r;
}
template <int N>
__device__ __forceinline__ Dual<N> operator/(const Dual<N>& a, const Dual<N>& b) {
  Dual<N> r; r.v = a.v / b.v;
  const double ib = 1.0 / b.v;
#pragma unroll
  for (int i = 0; i < N; ++i) r.d[i] = (a.d[i] - r.v * b.d[i]) * ib;
  return r;
}
template <int N>
__device__ __forceinline__ Dual<N> operator+(const Dual<N>& a, double b) { return a + cst<N>(b); }
template <int N>
__device__ __forceinline__ Dual<N> operator+(double a, const Dual<N>& b) { return cst<N>(a) + b; }
template <int N>
__device__ __forceinline__ Dual<N> operator-(const Dual<N>& a, double b) { return a - cst<N>(b); }
template <int N>
__device__ __forceinline__ Dual<N> operator-(double a, const Dual<N>& b) { return cst<N>(a) - b; }
template <int N>
__device__ __forceinline__ Dual<N> operator*(const Dual<N>& a, double b) {
  Dual<N> r; r.v = a.v * b;
#pragma unroll
  for (int i = 0; i < N; ++i) r.d[i] = a.d[i] * b;
  return r;
}
template <int N>
__device__ __forceinline__ Dual<N> operator*(double a, const Dual<N>& b) { return b * a; }
template <int N>
__device__ __forceinline__ Dual<N> operator/(const Dual<N>& a, double b) { return a * (1.0 / b); }
template <int N>
__device__ __forceinline__ Dual<N> operator/(double a, const Dual<N>& b) { return cst<N>(a) / b; }
template <int N>
__device__ __forceinline__ Dual<N> chain(const Dual<N>& a, double f, double df) {
  Dual<N> r; r.v = f;
#pragma unroll
  for (int i = 0; i < N; ++i) r.d[i] = df * a.d[i];
  return r;
}
template <int N>
__device__ __forceinline__ Dual<N> dexp(const Dual<N>& a) { const double e = exp(a.v); return chain(a, e, e); }
template <int N>
__device__ __forceinline__ Dual<N> dlog(const Dual<N>& a) { return chain(a, log(a.v), 1.0 / a.v); }
template <int N>
__device__ __forceinline__ Dual<N> dpow(const Dual<N>& a, double y) {
  const double p = pow(a.v, y);
  return chain(a, p, y * p / a.v);
}
template <int N>
__device__ __forceinline__ Dual<N> dcbrt(const Dual<N>& a) {
  const double c = cbrt(a.v);
  return chain(a, c, c / (3.0 * a.v));
}
__device__ __forceinline__ double dexp(double a) { return exp(a); }
__device__ __forceinline__ double dlog(double a) { return log(a); }
__device__ __forceinline__ double dpow(double a, double y) { return pow(a, y); }
__device__ __forceinline__ double dcbrt(double a) { return cbrt(a); }
__device__ __forceinline__ double val(double a) { return a; }
template <int N>
__device__ __forceinline__ double val(const Dual<N>& a) { return a.v; }
// a constant of scalar type S
template <class S>
struct Const {
  static __device__ __forceinline__ S of(double v) { return v; }
};
template <int N>
struct Const<Dual<N>> {
  static __device__ __forceinline__ Dual<N> of(double v) { return cst<N>(v); }
};

// ---- cell ambient from Theta and r_v (integration.py:402-484, 359-400) ----
struct GridConst {
  double p_ref, p_ref_inv, V;
};
template <class S>
struct Amb {
  S T, p, Sat, e_s, K, D_v, L_v, sigw, rhow, lap0, lbp0, c1, c2;
};
template <class S>
__device__ __forceinline__ Amb<S> ambient(const S& Th, const S& r_v, double rho_d,
                                          const GridConst& g) {
  Amb<S> a;
  const S pdr = dpow(rho_d * Th * (LC_R_D * g.p_ref_inv), LC_KAPPA_FACTOR);
  a.T = Th * dpow(pdr, LC_KAPPA_AIR_DRY);
  a.p = pdr * g.p_ref * (1.0 + r_v / LC_EPSILON_GC);
  a.e_s = 2.53E11 * dexp(-5420.0 / a.T);
  a.Sat = rho_d * r_v * a.T * LC_R_V / a.e_s;
  a.K = 4.1868E-3 * (5.69 + 0.017 * (a.T - 273.15));
  a.D_v = 4.01218E-5 * dpow(a.T, 1.94) / a.p;
  a.L_v = 1.0E3 * (2500.82 - 2.358 * (a.T - 273.0));
  const S tau = 1.0 - a.T / 647.096;
  a.sigw = 0.2358 * dpow(tau, 1.256) * (1.0 - 0.625 * tau);
  const S dT = a.T - LC_PAR_WATER_DENS_2;
  a.rhow = LC_PAR_WATER_DENS_0 + LC_PAR_WATER_DENS_1 * (dT * dT);
  a.lap0 = (LC_C_ALPHA_1 + LC_C_ALPHA_2 * (a.T - LC_T_ALPHA_0)) * a.K / a.p;
  a.lbp0 = LC_C_BETA_1 * (1.0 + LC_C_BETA_2 * (a.T - LC_T_ALPHA_0)) * a.D_v;
  a.c1 = a.L_v * a.L_v / (LC_R_V * a.K * a.T * a.T);
  a.c2 = LC_R_V * a.T / (a.D_v * a.e_s);
  return a;
}

// ---- mass rate of an ammonium-sulfate SIP (microphysics.py:1359-1469) with
// the kappa scaling; gamma in fg/s and (for S = double) dgamma/dm_w ----
template <class S, class M>
__device__ __forceinline__ S mass_rate(const M& m, const S& m_s, const S& ks, const Amb<S>& a,
                                       S* dg_out) {
  const S m_p = m + m_s;
  const S w_s = m_s / m_p;
  S pr = LC_PAR_RHO_AS_0 * w_s + LC_PAR_RHO_AS_1;
  pr = pr * w_s + LC_PAR_RHO_AS_2;
  pr = pr * w_s + LC_PAR_RHO_AS_3;
  const S rho_p = a.rhow * pr;
  const S R_p = dcbrt(LC_FOUR_PI_OVER_THREE_INV * m_p / rho_p);
  const S sigma_p = a.sigw * (1.0 + LC_PAR_SIGMA_AS * w_s / (1.0 - w_s));
  const S l_a = 1.0E-6 * (R_p + a.lap0);
  const S l_b = 1.0E-6 * (R_p + a.lbp0);
  const S m_p_inv_SI = 1.0E18 / m_p;
  const S wfac = w_s / ((1.0 - w_s) * (1.0 - w_s));
  S pd = LC_PAR_RHO_DERIV_AS_0 * w_s + LC_PAR_RHO_DERIV_AS_1;
  pd = pd * w_s + LC_PAR_RHO_DERIV_AS_2;
  const S drho_dm_over_rho = -1.0 * a.rhow * m_p_inv_SI / rho_p * w_s * pd;
  S aw = LC_PAR_WAT_ACT_AS_0 * w_s + LC_PAR_WAT_ACT_AS_1;
  aw = aw * w_s + LC_PAR_WAT_ACT_AS_2;
  aw = aw * w_s + LC_PAR_WAT_ACT_AS_3;
  const S aw_m1 = ks * (aw * w_s);                    // a_w - 1, scaled by kappa / 0.6
  const S a_w = 1.0 + aw_m1;
  S da = LC_PAR_WAT_ACT_DERIV_AS_0 * w_s + LC_PAR_WAT_ACT_DERIV_AS_1;
  da = da * w_s + LC_PAR_WAT_ACT_DERIV_AS_2;
  da = da * w_s + LC_PAR_WAT_ACT_DERIV_AS_3;
  const S da_w_dm = -1.0 * ks * m_p_inv_SI * w_s * da;
  const S dsigma_dm = -LC_PAR_SIGMA_AS * a.sigw * m_p_inv_SI * wfac;
  const S dR_dm_over_R = LC_ONE_THIRD * (m_p_inv_SI - drho_dm_over_rho);
  const S dR_dm = 1.0E-6 * dR_dm_over_R * R_p;
  const S eps_k = 2.0E6 * sigma_p / (LC_R_V * a.T * rho_p * R_p);
  const S kel = dexp(eps_k);
  const S S_eq = a_w * kel;
  const S f3 = 1.0 / (l_a * S_eq * a.c1 + l_b * a.c2);
  const S f1f3 = LC_FOUR_PI * R_p * R_p * f3;
  const S f2 = a.Sat - S_eq;
  if (dg_out) {   // dgamma/dm_w in the arithmetic of S (second derivatives for duals)
    const S dSeq = da_w_dm * kel + S_eq * eps_k * (dsigma_dm / sigma_p - drho_dm_over_rho -
                                                   dR_dm_over_R);
    const S dg1 = (dSeq * l_a + S_eq * dR_dm) * a.c1 + dR_dm * a.c2;
    *dg_out = 1.0E-12 * f1f3 * (f2 * (2.0 * dR_dm_over_R - f3 * dg1) - dSeq);
  }
  return 1.0E6 * f1f3 * f2;
}

// the implicit Euler step solved to convergence; returns the new mass and
// whether it sits on the efflorescence floor
// (no_iter > 0: exactly no_iter evaluations, the map of integration.py:728-836
// the time step uses; 0: to convergence)
__device__ __forceinline__ double solve_step(double m_w, double m_s, double ks,
                                             const Amb<double>& a, double dt, int no_iter,
                                             bool* floored) {
  const double m_eff = m_s * (LC_W_S_MAX_AS_INV - 1.0);
  double dg;
  double g = mass_rate<double>(m_w, m_s, ks, a, &dg);
  double x = dt * dg;
  double m = m_w + dt * g * ((x < 0.9) ? 1.0 / (1.0 - x) : 10.0);
  if (!(m >= m_eff)) m = m_eff;
  const int iters = no_iter > 0 ? no_iter - 1 : 40;
  for (int it = 0; it < iters; ++it) {
    g = mass_rate<double>(m, m_s, ks, a, &dg);
    x = dt * dg;
    double mn = m + (dt * g + m_w - m) * ((x < 0.9) ? 1.0 / (1.0 - x) : 10.0);
    if (!(mn >= m_eff)) mn = m_eff;
    const double step = fabs(mn - m);
    m = mn;
    if (no_iter == 0 && step <= 1e-15 * fabs(m)) break;
  }
  *floored = !(m > m_eff);
  return m;
}

// the time step's own map (integration.py:786-836): no_iter evaluations of the
// damped Newton, each floored at the efflorescence mass, in the arithmetic of
// S (duals: the exact derivative of the map, branches taken as evaluated)
template <class S>
__device__ __forceinline__ S newton_map(const S& m_w, const S& m_s, const S& ks, const Amb<S>& a,
                                        double dt, int no_iter) {
  const S m_eff = m_s * (LC_W_S_MAX_AS_INV - 1.0);
  S dg;
  S g = mass_rate<S>(m_w, m_s, ks, a, &dg);
  S x = dt * dg;
  S m = m_w + dt * g * ((val(x) < 0.9) ? 1.0 / (1.0 - x) : Const<S>::of(10.0));
  if (!(val(m) >= val(m_eff))) m = m_eff;
  for (int it = 0; it < no_iter - 1; ++it) {
    g = mass_rate<S>(m, m_s, ks, a, &dg);
    x = dt * dg;
    m = m + (dt * g + m_w - m) * ((val(x) < 0.9) ? 1.0 / (1.0 - x) : Const<S>::of(10.0));
    if (!(val(m) >= val(m_eff))) m = m_eff;
  }
  return m;
}

// cell update (integration.py:402-438): Theta and r_v after the sub-step
template <class S, class F>
__device__ __forceinline__ void cell_update(const S& Th, const S& r_v, const S& dml, double rho_d,
                                            double mdi, const F& dTh, const F& drv,
                                            const GridConst& g, S* Th_out, S* rv_out) {
  const Amb<S> a = ambient<S>(Th, r_v, rho_d, g);   // L_v before the update
  const S Th1 = Th + dTh;
  const S rv1 = r_v + drv - dml * mdi;
  const S ToT = dpow(g.p_ref_inv * LC_R_D * rho_d * Th1, LC_KAPPA_FACTOR2);
  *Th_out = Th1 + ToT * (a.L_v * dml) / (LC_C_PD * rho_d * g.V * (1.0 + rv1 * LC_HEAT_FACTOR_R_V));
  *rv_out = rv1;
}

// The derivatives of a cell's terms (CellFF) by Theta (T) and r_v (r), cx and
// ce by their logarithms
struct CellGrad {
  ff S_T, lcx_T, lce_T, la_T, lb_T, c1_T, c2_T;
  ff S_r, la_r, lb_r, c2_r;
  double pad[5];
};
static_assert(sizeof(CellGrad) == 128, "one line");

// dt gamma and dt dgamma/dm of mass_rate_ff (ammonium sulfate, a_w - 1 scaled by
// ks) and the reverse of its evaluation: with the adjoints gb of dt gamma and xb
// of x = dt dgamma/dm, the adjoints of the mass (returned), of m_s, ks and of the
// cell's terms (added to acc).  The reverse follows the forward's lines upwards;
// with b(.) the adjoint, the products that recur are
//   e = b(eps) eps, X = b(x_r) x_r = (b(R) R - e) / 3 (x_r = 3 m_p / (4 pi rho)),
// and 1 / rho, 1 / m_p enter through u, e, X, x and w alone.
struct RevAcc {
  ff ms, ks, S, lcx, lce, la, lb, c1, c2;
};
__device__ __forceinline__ ff two(ff a) { return ff{2.0f * a.h, 2.0f * a.l}; }
struct MassRate {
  // the forward values the reverse reads
  ff imp, im, wf, q, ipr, isg, z, R, eps, kel, am1, f2, Seq, pd, da, u, t, v, A, B, y, z3, D, iden,
      N, E, G, k1, k2, gd, x, P;
};
__device__ __forceinline__ bool mass_rate_fwd(double m, double ms, ff msf, const CellFF& c, ff gdt,
                                              double ks, ff ksf, MassRate& r) {
  const double mp = m + ms;
  const ff mpf = d2ff(mp);
  r.imp = ff_rcp(mpf);
  r.wf = ff_mul(msf, r.imp);
  double w = ff2d(r.wf);
  w = fma(fma(-w, mp, ms), f2d_int(r.imp.h), w);
  r.im = ff_rcp(d2ff(m));
  r.q = ff_mul(msf, r.im);
  const double P = w * (((LC_PAR_WAT_ACT_AS_0 * w + LC_PAR_WAT_ACT_AS_1) * w +
                         LC_PAR_WAT_ACT_AS_2) * w + LC_PAR_WAT_ACT_AS_3);
  r.P = d2ff(P);
  const double aw_m1 = ks * P;
  r.am1 = ff_add(d2ff(aw_m1), 1.0f);   // a_w
  ff da = ff_add(FFC(LC_PAR_WAT_ACT_DERIV_AS_1), ff_mul(FFC(LC_PAR_WAT_ACT_DERIV_AS_0), r.wf));
  da = ff_add(FFC(LC_PAR_WAT_ACT_DERIV_AS_2), ff_mul(da, r.wf));
  r.da = ff_add(FFC(LC_PAR_WAT_ACT_DERIV_AS_3), ff_mul(da, r.wf));
  ff pd = ff_horner(FFC(LC_PAR_RHO_DERIV_AS_1), FFC(LC_PAR_RHO_DERIV_AS_0), r.wf);
  r.pd = ff_horner(FFC(LC_PAR_RHO_DERIV_AS_2), pd, r.wf);
  ff pr = ff_horner(FFC(LC_PAR_RHO_AS_1), FFC(LC_PAR_RHO_AS_0), r.wf);
  pr = ff_horner(FFC(LC_PAR_RHO_AS_2), pr, r.wf);
  r.ipr = ff_rcp(ff_one_plus(ff_mul(pr, r.wf)));
  const ff sq = ff_mul(FFC(LC_PAR_SIGMA_AS), r.q);
  const ff sg = ff_add(sq, 1.0f);
  r.isg = ff_rcp(sg);
  const ff xr = ff_mul(ff_mul(c.cx, mpf), r.ipr);
  r.z = ff_icbrt(xr);
  r.R = ff_mul(ff_mul(xr, r.z), r.z);
  r.eps = ff_mul(ff_mul(c.ce, sg), ff_mul(r.ipr, r.z));
  const ff em1 = ff_expm1(r.eps);
  r.kel = ff_one_plus(em1);
  const double sm1 = fma(1.0 + aw_m1, ff2d(em1), aw_m1);
  r.f2 = d2ff(c.S_m1 - sm1);
  r.Seq = ff_add(d2ff(sm1), 1.0f);
  r.u = ff_mul(ff_mul(r.wf, r.pd), r.ipr);
  r.t = ff_mul(ff_add(r.u, 1.0f), FFC(1.0 / 3.0));
  r.v = ff_mul(r.R, r.t);
  r.A = ff_add(c.la, r.R);
  r.B = ff_add(c.lb, r.R);
  r.y = ff_mul(ff_mul(sq, ff_add(r.q, 1.0f)), r.isg);
  r.z3 = ff_sub(ff_add(two(r.t), -1.0f), r.y);
  r.D = ff_sub(ff_mul(ff_mul(r.Seq, r.eps), r.z3),
               ff_mul(ff_mul(ff_mul(r.wf, r.da), ksf), r.kel));
  r.E = ff_mul(r.A, r.Seq);
  r.iden = ff_rcp(ff_add(ff_mul(r.E, c.c1), ff_mul(r.B, c.c2)));
  r.N = ff_add(ff_mul(ff_add(ff_mul(r.D, r.A), ff_mul(r.Seq, r.v)), c.c1), ff_mul(r.v, c.c2));
  r.G = ff_mul(ff_mul(gdt, ff_mul(r.R, r.R)), r.iden);
  r.k1 = ff_sub(two(r.t), ff_mul(r.N, r.iden));
  r.k2 = ff_sub(ff_mul(r.f2, r.k1), r.D);
  r.gd = ff_mul(r.G, r.f2);
  r.x = ff_mul(ff_mul(r.G, r.imp), r.k2);
  return r.eps.h < 0.25f;
}
__device__ __forceinline__ ff mass_rate_rev(const MassRate& r, const CellFF& c, ff msf, ff ksf,
                                            ff gb, ff xb, RevAcc& acc) {
  const ff Gi = ff_mul(r.G, r.imp);
  const ff kb2 = ff_mul(xb, Gi);
  // b(G) G and b(1/den) / den follow from gd, x, G and H = N / den
  const ff xx = ff_mul(xb, r.x);                        // xb x
  const ff GbG = ff_add(ff_mul(gb, r.gd), xx);          // b(G) G
  ff fb2 = ff_add(ff_mul(gb, r.G), ff_mul(kb2, r.k1));
  const ff kb1 = ff_mul(kb2, r.f2);
  ff Db = ff_neg(kb2);
  ff tb = two(kb1);
  const ff Nb = ff_neg(ff_mul(kb1, r.iden));
  // den: b(den) = -(b(G) G + b(H) H) / den, b(H) = -kb1
  const ff H = ff_mul(r.N, r.iden);
  const ff db = ff_neg(ff_mul(ff_sub(GbG, ff_mul(kb1, H)), r.iden));
  ff RbR = two(GbG);                                    // b(R) R
  const ff Q = ff_add(ff_mul(r.D, r.A), ff_mul(r.Seq, r.v));
  const ff Qb = ff_mul(Nb, c.c1);
  acc.c1 = ff_add(acc.c1, ff_add(ff_mul(Nb, Q), ff_mul(db, r.E)));
  acc.c2 = ff_add(acc.c2, ff_add(ff_mul(Nb, r.v), ff_mul(db, r.B)));
  const ff vb = ff_add(ff_mul(Nb, c.c2), ff_mul(Qb, r.Seq));
  Db = ff_add(Db, ff_mul(Qb, r.A));
  const ff Eb = ff_mul(db, c.c1);
  const ff Ab = ff_add(ff_mul(Qb, r.D), ff_mul(Eb, r.Seq));
  const ff Bb = ff_mul(db, c.c2);
  ff Sb = ff_add(ff_mul(Qb, r.v), ff_mul(Eb, r.A));     // b(S_eq)
  const ff DSe = ff_mul(Db, r.eps);
  Sb = ff_add(Sb, ff_mul(DSe, r.z3));
  const ff zb3 = ff_mul(DSe, r.Seq);
  ff e = ff_mul(zb3, r.z3);                             // b(eps) eps
  const ff wda = ff_mul(r.wf, r.da);
  const ff Wb = ff_neg(ff_mul(Db, r.kel));              // b(ks w a_w')
  ff mb1 = ff_neg(ff_mul(Db, ff_mul(wda, ksf)));        // b(expm1) through e^eps
  tb = ff_add(tb, two(zb3));
  // y = s q (1 + q) / (1 + s q): dy/dq = s (1 + 2q - y) / (1 + s q)
  ff qb = ff_neg(ff_mul(ff_mul(zb3, FFC(LC_PAR_SIGMA_AS)),
                        ff_mul(ff_sub(ff_add(two(r.q), 1.0f), r.y), r.isg)));
  acc.la = ff_add(acc.la, Ab);
  acc.lb = ff_add(acc.lb, Bb);
  RbR = ff_add(RbR, ff_mul(ff_add(ff_add(Ab, Bb), ff_mul(vb, r.t)), r.R));
  tb = ff_add(tb, ff_mul(vb, r.R));
  const ff ub = ff_mul(tb, FFC(1.0 / 3.0));
  const ff uw = ff_mul(ub, r.ipr);
  ff wb = ff_mul(uw, r.pd);
  const ff pdb = ff_mul(uw, r.wf);
  acc.S = ff_add(acc.S, fb2);
  const ff Sq = ff_sub(Sb, fb2);
  const ff ab = ff_mul(Sq, r.kel);                      // b(a_w)
  mb1 = ff_add(mb1, ff_mul(Sq, r.am1));
  e = ff_add(e, ff_mul(ff_mul(mb1, r.kel), r.eps));
  acc.ks = ff_add(acc.ks, ff_add(ff_mul(ab, r.P), ff_mul(Wb, wda)));
  // a_w' and its derivative
  ff dd = ff_add(FFC(2.0 * LC_PAR_WAT_ACT_DERIV_AS_1),
                 ff_mul(FFC(3.0 * LC_PAR_WAT_ACT_DERIV_AS_0), r.wf));
  dd = ff_add(FFC(LC_PAR_WAT_ACT_DERIV_AS_2), ff_mul(dd, r.wf));
  wb = ff_add(wb, ff_mul(ksf, ff_add(ff_mul(ab, r.da),
                                     ff_mul(Wb, ff_add(r.da, ff_mul(r.wf, dd))))));
  acc.lce = ff_add(acc.lce, e);
  qb = ff_add(qb, ff_mul(ff_mul(e, r.isg), FFC(LC_PAR_SIGMA_AS)));
  const ff X = ff_mul(ff_sub(RbR, e), FFC(1.0 / 3.0));
  acc.lcx = ff_add(acc.lcx, X);
  // rho / rho_w: b = -(b(u) u + e + X) / (rho / rho_w)
  const ff pb = ff_neg(ff_mul(ff_add(ff_add(ff_mul(ub, r.u), e), X), r.ipr));
  const ff pdd = ff_add(FFC(LC_PAR_RHO_DERIV_AS_1),
                        ff_mul(FFC(2.0 * LC_PAR_RHO_DERIV_AS_0), r.wf));
  wb = ff_add(wb, ff_add(ff_mul(pb, r.pd), ff_mul(pdb, pdd)));
  const ff mpb = ff_mul(r.imp, ff_sub(ff_sub(X, xx), ff_mul(wb, r.wf)));
  const ff qm = ff_mul(qb, r.im);
  acc.ms = ff_add(acc.ms, ff_add(ff_add(qm, ff_mul(wb, r.imp)), mpb));
  return ff_sub(mpb, ff_mul(qm, r.q));
}

struct Args {
  int64_t n, C;
  double* m_w;          // [n] in/out
  const double* m_s;    // [n]
  const double* xi;     // [n]
  const int32_t* cell;  // [n] this sub-step's cells (negative: not condensing)
  double* Th;           // [C] in/out
  double* r_v;          // [C] in/out
  const double* rho_d;  // [C]
  const double* mdi;    // [C] mass_dry_inv
  const double* dTh;    // [C] per sub-step forcing, or null
  const double* drv;    // [C]
  double* dml;          // [C] scratch
  double dt, ks;
  GridConst g;
  int no_iter;          // 0: implicit step to convergence, else the step's map
  CellFF* rec;          // [C] the map's cell terms (no_iter > 0 and scratch), else null
  CellGrad* grad;       // [C] their derivatives (reverse sweep)
  CellFast* fast;       // [C] the terms in FP64 (forward sweep)
};

__device__ __forceinline__ CellFast fast_of(const CellState& s) {
  CellAmb m;
  m.T = s.T; m.S = s.S; m.sigw = s.t.sigw; m.rhow = s.t.rhow; m.lap0 = s.t.lap0;
  m.lbp0 = s.t.lbp0; m.c1 = s.t.c1; m.c2 = s.t.c2;
  return cell_fast(SOL_AS, m);
}
// a cell's terms for the sub-step that starts from Theta and r_v, as the time
// step forms them, and (GRAD) their derivatives
template <bool GRAD>
__device__ __forceinline__ void write_cell(const Args& a, int64_t c, double Th, double rv) {
  const double rho_d = a.rho_d[c];
  const CellState s = cell_state64(Th, rv, rho_d, a.g.p_ref, a.g.p_ref_inv);
  write_rec64(a.rec + c, s.T, s.S, s.L_v, s.mu, s.rho_f, s.t);
  if (!GRAD) {
    a.fast[c] = fast_of(s);
  }
  if (GRAD) {
    // logarithmic derivatives: T ~ Theta^kf (kf = 1 / (1 - kappa)), p the same
    // and 1 + r_v / eps, e_s' / e_s = 5420 / T^2
    CellGrad* const g = a.grad + c;
    const double iTh = rcp64(Th), iT = rcp64(s.T);
    const double lT = LC_KAPPA_FACTOR * iTh, T_T = lT * s.T;
    const double lp_r = rcp64(LC_EPSILON_GC + rv);
    const double les = 5420.0 * iT * iT * T_T;
    const double lK = 4.1868E-3 * 0.017 * T_T * rcp64(s.K);
    const double lD = 1.94 * lT - lT;              // D_v ~ T^1.94 / p
    const double lL = -2358.0 * T_T * rcp64(s.L_v);
    const double tau = 1.0 - s.T * (1.0 / 647.096);
    const double lsig = (1.256 * rcp64(tau) - 0.625 * rcp64(1.0 - 0.625 * tau)) *
                        (-1.0 / 647.096) * T_T;
    const double lrho = 2.0 * LC_PAR_WATER_DENS_1 * (s.T - LC_PAR_WATER_DENS_2) * T_T *
                        rcp64(s.t.rhow);
    const double dT = s.T - LC_T_ALPHA_0;
    g->S_T = d2ff(s.S * (lT - les));
    g->S_r = d2ff(rho_d * s.T * LC_R_V * rcp64(s.e_s));   // S / r_v, for r_v = 0 too
    g->lcx_T = d2ff(-lrho);
    g->lce_T = d2ff(lsig - lrho - lT);
    g->la_T = d2ff(s.t.lap0 * (LC_C_ALPHA_2 * T_T * rcp64(LC_C_ALPHA_1 + LC_C_ALPHA_2 * dT) + lK -
                               lT));
    g->la_r = d2ff(-s.t.lap0 * lp_r);
    g->lb_T = d2ff(s.t.lbp0 * (LC_C_BETA_2 * T_T * rcp64(1.0 + LC_C_BETA_2 * dT) + lD));
    g->lb_r = d2ff(-s.t.lbp0 * lp_r);
    g->c1_T = d2ff(s.t.c1 * (2.0 * (lL - lT) - lK));
    g->c2_T = d2ff(s.t.c2 * (lT - lD - les));
    g->c2_r = d2ff(s.t.c2 * lp_r);
  }
}
__global__ void k_cell_terms(Args a) {
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < a.C;
       c += (int64_t)gridDim.x * blockDim.x)
    write_cell<false>(a, c, a.Th[c], a.r_v[c]);
}
__device__ __forceinline__ CellFF load_cell(const CellFF* rec) {
  CellFF cf;
  const float4* src = (const float4*)rec;
  float4* dst = (float4*)&cf;
#pragma unroll
  for (int q = 0; q < 6; ++q) dst[q] = __ldg(src + q);
  return cf;
}

// one condensation step in FP64: to convergence (no_iter = 0), or of a SIP
// outside the two-float range
__device__ __noinline__ double fwd_step64(const Args& a, int32_t c, double mw, double ms) {
  if (a.fast && ff_mass_ok(mw) && ff_mass_ok(ms))
    return newton_fast(SOL_AS, a.dt, a.no_iter, mw, ms, a.fast[c], a.ks);
  const Amb<double> am = ambient<double>(a.Th[c], a.r_v[c], a.rho_d[c], a.g);
  bool fl;
  return solve_step(mw, ms, a.ks, am, a.dt, a.no_iter, &fl);
}

// The SIPs of a forward sub-step.  MAP: the time step's map as the time step runs
// it (newton_ff; FULL as there), else the converged step, or the map in FP64 without
// scratch.  SIPs whose step needs plain FP64 wait in the block's queue, as in the
// time step.  Bound by issue and the FP64 pipe; 720,000 SIPs took 1326 us a launch
// with the cell's ambient terms and the Newton per SIP in FP64, 190 us with plain
// FP64 in place, 140 us gathered, 117 us with the cell's FP64 terms stored beside its
// record.
constexpr int FQ = 1024;
template <bool MAP, bool FULL>
__global__ void __launch_bounds__(128) k_fwd_sips(const __grid_constant__ Args a, double* tape_m) {
  __shared__ int32_t s_q[MAP ? FQ : 1];
  __shared__ int s_n;
  if (MAP) {
    if (threadIdx.x == 0) s_n = 0;
    __syncthreads();
  }
  const ff gdt = d2ff(LC_FOUR_PI * 1.0E12 * a.dt);
  auto put = [&](int64_t k, int32_t c, double mw, double m) {
    a.m_w[k] = m;
    atomicAdd(a.dml + c, (m - mw) * a.xi[k]);
  };
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < a.n;
       k += (int64_t)gridDim.x * blockDim.x) {
    const double mw = a.m_w[k];
    if (tape_m) tape_m[k] = mw;
    const int32_t c = a.cell[k];
    if (c < 0) continue;
    const double ms = a.m_s[k];
    double m;
    if (MAP) {
      const CellFF cf = load_cell(a.rec + c);   // beside the loads of the masses
      bool ok = ff_mass_ok(mw) && ff_mass_ok(ms);
      if (ok) m = newton_ff<true, FULL>(SOL_AS, a.no_iter, mw, ms, cf, gdt, a.ks, &ok);
      if (!ok) {
        const int at = atomicAdd(&s_n, 1);
        if (at < FQ) {
          s_q[at] = (int32_t)k;
          continue;
        }
        m = fwd_step64(a, c, mw, ms);
      }
    } else {
      m = fwd_step64(a, c, mw, ms);
    }
    put(k, c, mw, m);
  }
  if (MAP) {
    __syncthreads();
    const int end = s_n < FQ ? s_n : FQ;
    for (int q = threadIdx.x; q < end; q += blockDim.x) {
      const int64_t k = s_q[q];
      const int32_t c = a.cell[k];
      const double mw = a.m_w[k];
      put(k, c, mw, fwd_step64(a, c, mw, a.m_s[k]));
    }
  }
}

// The cells of a forward sub-step, four lanes each for the map (cell_state64_x4;
// 1240 cells: 13.7 us a launch with one thread each, 10.5 us now).
__global__ void __launch_bounds__(32) k_fwd_cells(Args a, double* tape_c) {
  const int role = threadIdx.x & 3;
  for (int64_t c0 = (int64_t)blockIdx.x * 8; c0 < a.C; c0 += (int64_t)gridDim.x * 8) {
    int64_t c = c0 + (threadIdx.x >> 2);
    const bool in = c < a.C;
    if (!in) c = a.C - 1;
    const double Th = a.Th[c], rv = a.r_v[c];
    const double dml = a.dml[c] * 1.0E-18;
    const double fT = a.dTh ? a.dTh[c] : 0.0, fr = a.drv ? a.drv[c] : 0.0;
    double Th2 = Th, rv2 = rv;
    CellState s;
    double irho = 0.0, kelvin = 0.0;
    if (a.rec) {
      const double L_v = a.rec[c].L_v;
      __syncwarp();   // all lanes have read the cell
      cell_step64(&Th2, &rv2, a.rho_d[c], a.mdi[c], L_v, fT, fr, dml, a.g.V, a.g.p_ref_inv);
      s = cell_state64_x4(Th2, rv2, a.rho_d[c], a.g.p_ref, a.g.p_ref_inv, &irho, &kelvin);
    } else {
      __syncwarp();
      cell_update<double, double>(Th, rv, dml, a.rho_d[c], a.mdi[c], fT, fr, a.g, &Th2, &rv2);
    }
    if (!in) continue;
    if (role == 0) {
      if (tape_c) { tape_c[c] = Th; tape_c[a.C + c] = rv; }
      a.dml[c] = 0.0;
      a.Th[c] = Th2;
      a.r_v[c] = rv2;
    } else if (a.rec && role == 1) {
      write_rec64(a.rec + c, s.T, s.S, s.L_v, s.mu, s.rho_f, s.t, irho, kelvin);
    } else if (a.rec && role == 2) {
      a.fast[c] = fast_of(s);
    }
  }
}

// reverse of one sub-step.  In: lam_m [n], lam_Th, lam_rv [C] (adjoints of the
// state after the sub-step), tape_m (m_w before), tape_c (Theta, r_v before),
// m_after [n] (m_w after).  Out: the same adjoints for the state before;
// grad_ms [n] and grad_ks [1] accumulate.
// lam_inc (optional, [2][C]) accumulates the adjoints of the increments
// (dTh, drv), which every sub-step of a half step shares
__global__ void k_bwd_cells(Args a, const double* tape_c, const double* m_before,
                            const double* m_after, double* lam_Th, double* lam_rv,
                            double* lam_dml, double* lam_inc) {
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < a.C;
       c += (int64_t)gridDim.x * blockDim.x) {
    const double Th = tape_c[c], rv = tape_c[a.C + c];
    const double dml = a.dml[c] * 1.0E-18;   // recomputed forward sum of this sub-step
    const double fT = a.dTh ? a.dTh[c] : 0.0, fr = a.drv ? a.drv[c] : 0.0;
    const double lT = lam_Th[c], lr = lam_rv[c];
    double Tv[5], rvv[5];   // partials of the new Theta and r_v by Theta, r_v, dml, dTh, drv
    if (a.rec) {
      write_cell<true>(a, c, Th, rv);
      // cell_step64: Theta' = Th1 + A, A = (c Th1)^kf2 L_v dml / (C (1 + h r_v'))
      const double L_v = a.rec[c].L_v;
      const double Th1 = Th + fT, rv1 = rv + (fr - dml * a.mdi[c]);
      const double ToT = exp64(LC_KAPPA_FACTOR2 * log64(a.g.p_ref_inv * LC_R_D * a.rho_d[c] * Th1));
      const double ih = rcp64(1.0 + rv1 * LC_HEAT_FACTOR_R_V);
      const double B = ToT * ih * rcp64(LC_C_PD * a.rho_d[c] * a.g.V);   // A = B L_v dml
      const double A = B * L_v * dml;
      const double T = 273.0 + (2500.82 - L_v * 1.0E-3) * (1.0 / 2.358);
      const double Ar = -A * LC_HEAT_FACTOR_R_V * ih;
      Tv[3] = 1.0 + A * LC_KAPPA_FACTOR2 * rcp64(Th1);
      Tv[0] = Tv[3] - B * dml * 2358.0 * LC_KAPPA_FACTOR * T * rcp64(Th);
      Tv[1] = Tv[4] = Ar;
      Tv[2] = B * L_v - Ar * a.mdi[c];
      rvv[0] = rvv[3] = 0.0;
      rvv[1] = rvv[4] = 1.0;
      rvv[2] = -a.mdi[c];
    } else {
      Dual<5> Th2, rv2;
      cell_update<Dual<5>, Dual<5>>(var<5>(Th, 0), var<5>(rv, 1), var<5>(dml, 2), a.rho_d[c],
                                    a.mdi[c], var<5>(fT, 3), var<5>(fr, 4), a.g, &Th2, &rv2);
      for (int q = 0; q < 5; ++q) { Tv[q] = Th2.d[q]; rvv[q] = rv2.d[q]; }
    }
    lam_Th[c] = lT * Tv[0] + lr * rvv[0];
    lam_rv[c] = lT * Tv[1] + lr * rvv[1];
    lam_dml[c] = (lT * Tv[2] + lr * rvv[2]) * 1.0E-18;   // per fg of dm*xi
    if (lam_inc) {
      lam_inc[c] += lT * Tv[3] + lr * rvv[3];
      lam_inc[a.C + c] += lT * Tv[4] + lr * rvv[4];
    }
    a.dml[c] = 0.0;
  }
}

__global__ void k_bwd_sum_dml(Args a, const double* m_before, const double* m_after) {
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < a.n;
       k += (int64_t)gridDim.x * blockDim.x) {
    const int32_t c = a.cell[k];
    if (c >= 0) atomicAdd(a.dml + c, (m_after[k] - m_before[k]) * a.xi[k]);
  }
}

// the partial derivatives of a SIP's new mass by m_w, m_s, ks, Theta and r_v
struct SipGrad {
  double m, ms, ks, Th, rv;
};
// in FP64 by duals: the time step's map (no_iter > 0), differentiated exactly
__device__ __noinline__ SipGrad map_grad64(const Args& a, double Th, double rv, double rho_d,
                                           double mw, double ms) {
  const Amb<Dual<5>> am = ambient<Dual<5>>(var<5>(Th, 3), var<5>(rv, 4), rho_d, a.g);
  const Dual<5> mn = newton_map<Dual<5>>(var<5>(mw, 0), var<5>(ms, 1), var<5>(a.ks, 2), am, a.dt,
                                         a.no_iter);
  return SipGrad{mn.d[0], mn.d[1], mn.d[2], mn.d[3], mn.d[4]};
}
// the converged step: implicit-function theorem
__device__ __noinline__ SipGrad root_grad64(const Args& a, double Th, double rv, double rho_d,
                                            double m, double ms) {
  const double m_eff = ms * (LC_W_S_MAX_AS_INV - 1.0);
  if (!(m > m_eff)) return SipGrad{0.0, LC_W_S_MAX_AS_INV - 1.0, 0.0, 0.0, 0.0};
  const Amb<Dual<4>> am = ambient<Dual<4>>(var<4>(Th, 2), var<4>(rv, 3), rho_d, a.g);
  double dg;
  {
    const Amb<double> a0 = ambient<double>(Th, rv, rho_d, a.g);
    mass_rate<double>(m, ms, a.ks, a0, &dg);
  }
  const Dual<4> gam = mass_rate<Dual<4>>(m, var<4>(ms, 0), var<4>(a.ks, 1), am, nullptr);
  const double inv = 1.0 / (1.0 - a.dt * dg), t = a.dt * inv;
  return SipGrad{inv, t * gam.d[0], t * gam.d[1], t * gam.d[2], t * gam.d[3]};
}

// The time step's map backwards: the masses m_1 .. m_{no_iter - 1} forwards
// (newton_ff's), then from the last evaluation to the first.  An evaluation is
//   m_{i+1} = max(m_eff, m_i + (dt gamma_i + m_w - m_i) / (1 - x_i)), m_0 = m_w.
constexpr int REV_MAX = 8;   // evaluations held; more take map_grad64
__device__ __forceinline__ bool map_grad(const Args& a, const CellFF& cf, const CellGrad* gr, ff gdt,
                                         double mw, double ms, SipGrad* out) {
  const double floor_m = ms * (LC_W_S_MAX_AS_INV - 1.0);
  const ff msf = d2ff(ms), ksf = d2ff(a.ks);
  double mi[REV_MAX];
  bool good = ff_mass_ok(mw) && ff_mass_ok(ms);
  {
    double m = mw;
#pragma unroll 1
    for (int it = 0; it < a.no_iter - 1; ++it) {
      mi[it] = m;
      ff gd, x;
      good = mass_rate_ff<true, false>(SOL_AS, false, m, ms, msf, cf, gdt, a.ks, gd, x) && good;
      const ff res = it == 0 ? gd : ff_sub(gd, d2ff(m - mw));
      m = np_max(floor_m, m + ff2d(ff_mul(res, damp_ff(x))));
    }
    mi[a.no_iter - 1] = m;
    good = good && m < 1e29;
  }
  const ff zero = {0.0f, 0.0f};
  RevAcc acc = {zero, zero, zero, zero, zero, zero, zero, zero, zero};
  ff mu = {1.0f, 0.0f};       // adjoint of m_{i+1}
  ff m0b = zero;              // of m_w, beyond m_0's
#pragma unroll 1
  for (int it = a.no_iter - 1; it >= 0; --it) {
    const double m = mi[it];
    MassRate r;
    good = mass_rate_fwd(m, ms, msf, cf, gdt, a.ks, ksf, r) && good;
    const ff dn = damp_ff(r.x);
    const ff res = it == 0 ? r.gd : ff_sub(r.gd, d2ff(m - mw));
    const double mn = m + ff2d(ff_mul(res, dn));
    if (!(mn >= floor_m)) {   // floored: only m_s is left
      acc.ms = ff_add(acc.ms, ff_mul(mu, FFC(LC_W_S_MAX_AS_INV - 1.0)));
      mu = zero;
      break;
    }
    const ff gb = ff_mul(mu, dn);
    ff xb = ff_mul(ff_mul(gb, dn), res);
    if (!(r.x.h < 0.9f)) xb = zero;
    const ff mb = mass_rate_rev(r, cf, msf, ksf, gb, xb, acc);
    if (it > 0) {
      m0b = ff_add(m0b, gb);
      mu = ff_add(ff_sub(mu, gb), mb);
    } else {
      mu = ff_add(mu, mb);
    }
  }
  auto ld = [&](int q) { const float2 v = __ldg((const float2*)gr + q); return ff{v.x, v.y}; };
  ff T = ff_add(ff_mul(acc.S, ld(0)), ff_mul(acc.lcx, ld(1)));
  T = ff_add(T, ff_add(ff_mul(acc.lce, ld(2)), ff_mul(acc.la, ld(3))));
  T = ff_add(T, ff_add(ff_mul(acc.lb, ld(4)), ff_mul(acc.c1, ld(5))));
  T = ff_add(T, ff_mul(acc.c2, ld(6)));
  ff V = ff_add(ff_mul(acc.S, ld(7)), ff_mul(acc.la, ld(8)));
  V = ff_add(V, ff_add(ff_mul(acc.lb, ld(9)), ff_mul(acc.c2, ld(10))));
  *out = SipGrad{ff2d(ff_add(mu, m0b)), ff2d(acc.ms), ff2d(acc.ks), ff2d(T), ff2d(V)};
  return good;
}

// The SIPs of a reverse sub-step.  Bound by FP32 issue at 8 warps an SM (255
// registers hold an evaluation's forward values); 720,000 SIPs took 4330 us a
// launch with duals of five directions through the ambient terms and the
// evaluations in FP64, 276 us now.
template <bool MAP>
__global__ void __launch_bounds__(128) k_bwd_sips(const __grid_constant__ Args a,
                                                  const double* tape_c, const double* m_before,
                                                  const double* m_after, double* lam_m,
                                                  const double* lam_dml, double* lam_Th_pre,
                                                  double* lam_rv_pre, double* grad_ms,
                                                  double* grad_ks) {
  double gk = 0.0;
  const ff gdt = d2ff(LC_FOUR_PI * 1.0E12 * a.dt);
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < a.n;
       k += (int64_t)gridDim.x * blockDim.x) {
    const int32_t c = a.cell[k];
    if (c < 0) continue;   // not condensing: m_w passes through
    const double ms = a.m_s[k];
    SipGrad g;
    if (MAP) {
      const double mw = m_before[k];
      const CellFF cf = load_cell(a.rec + c);
      if (a.no_iter > REV_MAX || !ff_mass_ok(mw) || !ff_mass_ok(ms) ||
          !map_grad(a, cf, a.grad + c, gdt, mw, ms, &g))
        g = map_grad64(a, tape_c[c], tape_c[a.C + c], a.rho_d[c], mw, ms);
    } else if (a.no_iter > 0) {
      g = map_grad64(a, tape_c[c], tape_c[a.C + c], a.rho_d[c], m_before[k], ms);
    } else {
      g = root_grad64(a, tape_c[c], tape_c[a.C + c], a.rho_d[c], m_after[k], ms);
    }
    // total adjoint of the new mass: the state after, and the cell sum
    const double ld = lam_dml[c] * a.xi[k];
    const double lm = lam_m[k] + ld;
    grad_ms[k] += lm * g.ms;
    gk += lm * g.ks * (1.0 / 0.6);   // ks = kappa / 0.6
    atomicAdd(lam_Th_pre + c, lm * g.Th);
    atomicAdd(lam_rv_pre + c, lm * g.rv);
    lam_m[k] = lm * g.m - ld;
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) gk += __shfl_down_sync(0xffffffffu, gk, off);
  if ((threadIdx.x & 31) == 0 && gk != 0.0) atomicAdd(grad_ks, gk);
}

// ---- advective increments of Theta and r_v (integration.py:80-287 with the
// sub-step increments of :1483-1508 and :1536-1561) in the arithmetic of S ----
__device__ __forceinline__ double dfmin(double x, double y) { return fmin(x, y); }
template <int N>
__device__ __forceinline__ Dual<N> dfmin(const Dual<N>& x, const Dual<N>& y) {
  if (isnan(x.v)) return y;   // C fmin: a NaN operand is ignored
  if (isnan(y.v)) return x;
  return (y.v < x.v) ? y : x;
}
__device__ __forceinline__ double dmax0(double z) { return np_max(0.0, z); }
template <int N>
__device__ __forceinline__ Dual<N> dmax0(const Dual<N>& z) {   // np.maximum(0, z)
  return (0.0 >= z.v) ? cst<N>(0.0) : z;
}
// integration.py:113-148 limiter of the Hundsdorfer et al. (1995) scheme
template <class S>
__device__ __forceinline__ S limiter_of(const S& a0, const S& a1, const S& a2) {
  const S r = (fabs(val(a1) - val(a2)) > 1.0E-8 * fabs(val(a0) - val(a1)))
                  ? (a0 - a1) / (a1 - a2)
                  : (a0 - a1) * 1.0E8 * np_sign(val(a1) - val(a2));
  const S K = (1.0 + 2.0 * r) * LC_ONE_THIRD;
  return dmax0(dfmin(2.0 * r, dfmin(K, Const<S>::of(2.0))));
}
// flux through the face left of stencil value a0 (integration.py:204-228)
template <class S>
__device__ __forceinline__ S face_flux_of(double u, const S& am2, const S& am1, const S& a0,
                                          const S& ap1) {
  if (u >= 0.0) return u * (am1 + 0.5 * limiter_of(a0, am1, am2) * (am1 - am2));
  return u * (a0 + 0.5 * limiter_of(am1, a0, ap1) * (a0 - ap1));
}
__device__ __forceinline__ int64_t wrap_idx(int64_t i, int64_t N, int bc) {
  if (bc == 0) { i %= N; return i < 0 ? i + N : i; }
  return i < 0 ? 0 : (i > N - 1 ? N - 1 : i);
}
// the four face fluxes of cell (i, j) (x: periodic, z: solid walls) and the
// flat indices of their stencils
struct Stencil {
  double u[4];
  int64_t idx[4][4];
  bool zero[4];
};
__device__ __forceinline__ Stencil stencil_of(const double* flux, int64_t nx, int64_t nz,
                                              int64_t i, int64_t j) {
  Stencil st;
  for (int s = 0; s < 2; ++s) {
    const int64_t fi = i + s, fj = j + s;
    st.u[s] = flux[fi * (nz + 1) + j];
    st.zero[s] = false;
    st.u[2 + s] = flux[(nx + 1) * (nz + 1) + i * (nz + 1) + fj];
    st.zero[2 + s] = (fj == 0 || fj == nz);
    for (int t = 0; t < 4; ++t) {
      st.idx[s][t] = wrap_idx(fi - 2 + t, nx, 0) * nz + j;
      st.idx[2 + s][t] = i * nz + wrap_idx(fj - 2 + t, nz, 1);
    }
  }
  return st;
}

struct IncArgs {
  const double* f[2];     // Theta, r_v [C]
  const double* rdi;      // rho_dry_inv [C]
  const double* flux;     // mass flux at the faces [2][nx+1][nz+1]
  const double* trel;     // relaxation time [nz] or null (no relaxation)
  const double* prof[2];  // initial profiles of Theta and r_v [nz]
  int64_t nx, nz;
  double dx, dz, dt;
};

// increments of a half step: second = 0: inc = -dt div rdi + relax;
// second = 1: inc = -2 dt div rdi - inc_prev + 2 relax (inc holds inc_prev)
__global__ void k_increments(IncArgs a, int second, double* inc_Th, double* inc_rv) {
  const int64_t C = a.nx * a.nz;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < 2 * C;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int fld = t < C ? 0 : 1;
    const int64_t c = t - fld * C, i = c / a.nz, j = c - i * a.nz;
    const double* f = a.f[fld];
    const Stencil st = stencil_of(a.flux, a.nx, a.nz, i, j);
    double F[4];
    for (int q = 0; q < 4; ++q)
      F[q] = st.zero[q] ? 0.0
                        : face_flux_of<double>(st.u[q], f[st.idx[q][0]], f[st.idx[q][1]],
                                               f[st.idx[q][2]], f[st.idx[q][3]]);
    const double div = (F[1] - F[0]) / a.dx + (F[3] - F[2]) / a.dz;
    double relax = 0.0;
    if (a.trel) {   // integration.py:325-354, column sum in x order
      double sum = f[j];
      for (int64_t ii = 1; ii < a.nx; ++ii) sum += f[ii * a.nz + j];
      relax = a.dt * (a.prof[fld][j] - sum / (double)a.nx) / a.trel[j];
    }
    double* out = fld == 0 ? inc_Th : inc_rv;
    double v;
    if (!second) {
      v = -a.dt * div * a.rdi[c];
      if (a.trel) v += relax;
    } else {
      v = -2.0 * a.dt * div * a.rdi[c] - out[c];
      if (a.trel) v += 2. * relax;
    }
    out[c] = v;
  }
}

// vector-Jacobian product of factor * (advective + relaxation increment):
// lam_f += factor J^T lam_inc for both fields; grad_s += factor lam_inc .
// (advective increment) / flux_scale, the derivative by a common factor s of
// the mass flux (the flux passed is s times the unscaled one)
__global__ void k_increments_vjp(IncArgs a, double factor, double flux_scale,
                                 const double* lam_inc, double* lam_Th, double* lam_rv,
                                 double* grad_s) {
  const int64_t C = a.nx * a.nz;
  double gs = 0.0;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < 2 * C;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int fld = t < C ? 0 : 1;
    const int64_t c = t - fld * C, i = c / a.nz, j = c - i * a.nz;
    const double* f = a.f[fld];
    double* lam_f = fld == 0 ? lam_Th : lam_rv;
    const double li = lam_inc[fld * C + c];
    if (li == 0.0) continue;
    const Stencil st = stencil_of(a.flux, a.nx, a.nz, i, j);
    const double ld = factor * li * (-a.dt * a.rdi[c]);   // adjoint of div(c)
    double div = 0.0;
    for (int q = 0; q < 4; ++q) {
      if (st.zero[q]) continue;
      const Dual<4> F = face_flux_of<Dual<4>>(st.u[q], var<4>(f[st.idx[q][0]], 0),
                                              var<4>(f[st.idx[q][1]], 1),
                                              var<4>(f[st.idx[q][2]], 2),
                                              var<4>(f[st.idx[q][3]], 3));
      const double w = (q & 1 ? 1.0 : -1.0) / (q < 2 ? a.dx : a.dz);
      div += w * F.v;
      for (int m = 0; m < 4; ++m)
        if (F.d[m] != 0.0) atomicAdd(lam_f + st.idx[q][m], ld * w * F.d[m]);
    }
    gs += factor * li * (-a.dt * div * a.rdi[c]) / flux_scale;
    if (a.trel) {   // relax_j depends on the column mean of field j
      const double lr = -factor * li * a.dt / (a.trel[j] * (double)a.nx);
      for (int64_t ii = 0; ii < a.nx; ++ii) atomicAdd(lam_f + ii * a.nz + j, lr);
    }
  }
  if (gs != 0.0) atomicAdd(grad_s, gs);
}

// ---- collisions as recorded events (collision/all_or_nothing.py:577-633) ----
struct EvRec {
  int32_t imin, imax, kind, pad;
  double a, b;
};

__device__ __forceinline__ void prefetch_l1(const void* p) {
  asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
}
// One warp per group, the group's records in order, in the collision step's own
// operation order: lanes 0 to 2 take the water and solute masses and the
// multiplicities.  Bound by the chain of the longest group, so its records share
// no warp with other groups' (32 groups a warp ran every kind of record for each
// of their steps), and the next record's SIPs are on their way to L1 while one is
// worked on (a raining run, 36 collision steps: 70 us a launch with one thread
// per group, 17 us now).
__global__ void __launch_bounds__(32) k_ev_forward(const EvRec* ev, const int64_t* off, int64_t G,
                                                   double* MW, double* MS, double* XI) {
  const int lane = threadIdx.x;
  if (lane > 2) return;
  constexpr unsigned LANES = 7u;
  double* const A = lane == 0 ? MW : (lane == 1 ? MS : XI);
  for (int64_t g = blockIdx.x; g < G; g += gridDim.x) {
    const int64_t end = off[g + 1];
    int64_t q = off[g];
    if (q >= end) continue;
    EvRec r = ev[q], next = ev[q + 1 < end ? q + 1 : q];
    for (; q < end; ++q) {
      const EvRec after = ev[q + 2 < end ? q + 2 : end - 1];
      prefetch_l1(A + next.imin);
      prefetch_l1(A + next.imax);
      const double lo = A[r.imin], hi = A[r.imax];
      if (r.kind == 1) {
        const double xi_min = XI[r.imin], xi_max = XI[r.imax];
        const double xi_ges = xi_min + xi_max;
        __syncwarp(LANES);   // all lanes have read the multiplicities
        if (lane < 2) {
          const double m = 2.0 * (xi_min * lo + xi_max * hi) / xi_ges;
          A[r.imin] = m;
          A[r.imax] = m;
        } else {
          const double x = 0.5 * 0.7 * xi_ges;
          A[r.imax] = x;
          A[r.imin] = 0.5 * xi_ges - x;
        }
      } else {
        const double f = r.kind == 2 ? r.a : 1.0;
        if (lane < 2) A[r.imin] = lo + f * hi;
        else A[r.imax] = hi - f * lo;
      }
      __syncwarp(LANES);
      r = next;
      next = after;
    }
  }
}

// the transposed maps, records in reverse order; lanes 0 and 1 take the adjoints of
// the water and the solute masses
__global__ void __launch_bounds__(32) k_ev_backward(const EvRec* ev, const int64_t* off, int64_t G,
                                                    double* LW, double* LS) {
  if (threadIdx.x > 1) return;
  double* const A = threadIdx.x ? LS : LW;
  for (int64_t g = blockIdx.x; g < G; g += gridDim.x) {
    const int64_t first = off[g];
    int64_t q = off[g + 1] - 1;
    if (q < first) continue;
    EvRec r = ev[q], next = ev[q > first ? q - 1 : q];
    for (; q >= first; --q) {
      const EvRec after = ev[q > first + 1 ? q - 2 : first];
      prefetch_l1(A + next.imin);
      prefetch_l1(A + next.imax);
      const double lo = A[r.imin], hi = A[r.imax];
      if (r.kind == 1) {   // both take 2 (xi_min m_min + xi_max m_max) / xi_ges
        const double xi_ges = r.a + r.b, s = lo + hi;
        A[r.imin] = 2.0 * r.a / xi_ges * s;
        A[r.imax] = 2.0 * r.b / xi_ges * s;
      } else {   // m_min += f m_max, f = p_crit (kind 2) or 1
        A[r.imax] = hi + (r.kind == 2 ? r.a : 1.0) * lo;
      }
      r = next;
      next = after;
    }
  }
}

static inline int ev_blocks(int64_t groups) { return (int)(groups < 152 * 64 ? groups : 152 * 64); }
static inline int nb(int64_t n, int t) {
  int64_t b = (n + t - 1) / t;
  return (int)(b < 1 ? 1 : (b > 152 * 16 ? 152 * 16 : b));
}

}  // namespace adj
}  // namespace lacmo

using namespace lacmo;
using namespace lacmo::adj;

static Args make_args(int64_t n, int64_t C, double* m_w, const double* m_s, const double* xi,
                      const int32_t* cell, double* Th, double* r_v, const double* rho_d,
                      const double* mdi, const double* dTh, const double* drv, double* dml,
                      double dt, double kappa, double p_ref, double V, int no_iter) {
  Args a;
  a.no_iter = no_iter;
  a.n = n; a.C = C; a.m_w = m_w; a.m_s = m_s; a.xi = xi; a.cell = cell; a.Th = Th; a.r_v = r_v;
  a.rho_d = rho_d; a.mdi = mdi; a.dTh = dTh; a.drv = drv; a.dml = dml; a.dt = dt;
  a.ks = kappa / 0.6;
  a.g.p_ref = p_ref; a.g.p_ref_inv = 1.0 / p_ref; a.g.V = V;
  a.rec = nullptr; a.grad = nullptr; a.fast = nullptr;
  return a;
}

extern "C" {

int lacmo_adj_forward(int64_t n, int64_t C, double* m_w, const double* m_s, const double* xi,
                      const int32_t* cell, int64_t cell_stride, double* Th, double* r_v,
                      const double* rho_d, const double* mdi, const double* dTh,
                      const double* drv, double* dml, double dt_sub, double kappa, double p_ref,
                      double V, int n_sub, int no_iter, double* tape_m, double* tape_c,
                      void* stream) {
  if (n <= 0 || C <= 0 || !m_w || !m_s || !xi || !cell || !Th || !r_v || !rho_d || !mdi || !dml ||
      n_sub < 0 || cell_stride < 0 || no_iter < 0 || !(kappa > 0.0) || !(p_ref > 0.0))
    return LACMO_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  Args a = make_args(n, C, m_w, m_s, xi, cell, Th, r_v, rho_d, mdi, dTh, drv, dml, dt_sub, kappa,
                     p_ref, V, no_iter);
  if (cudaMemsetAsync(dml, 0, 8 * C, s) != cudaSuccess) return LACMO_ERR_CUDA;
  Scratch scratch(s);
  // without scratch for the cells' terms every SIP forms its own, in FP64
  if (no_iter > 0 && n_sub > 0)
    a.rec = (CellFF*)scratch.get((sizeof(CellFF) + sizeof(CellFast)) * (size_t)C);
  if (a.rec) {
    a.fast = (CellFast*)(a.rec + C);
    k_cell_terms<<<nb(C, 32), 32, 0, s>>>(a);
    note_launches(1);
  }
  static std::atomic<int> cached[64];
  int res = 0;   // blocks of k_fwd_sips resident at once
  if (resident_blocks((const void*)k_fwd_sips<true, true>, 128, 0, cached, &res) != cudaSuccess)
    return LACMO_ERR_CUDA;
  for (int k = 0; k < n_sub; ++k) {
    a.cell = cell + (size_t)k * cell_stride;
    double* const tm = tape_m ? tape_m + (size_t)k * n : nullptr;
    if (!a.rec) k_fwd_sips<false, false><<<nb(n, 128), 128, 0, s>>>(a, tm);
    else if (n > 128 * (int64_t)res) k_fwd_sips<true, true><<<res, 128, 0, s>>>(a, tm);
    else k_fwd_sips<true, false><<<nb(n, 128), 128, 0, s>>>(a, tm);
    k_fwd_cells<<<nb(4 * C, 32), 32, 0, s>>>(a, tape_c ? tape_c + (size_t)k * 2 * C : nullptr);
    note_launches(2);
  }
  if (tape_m) {   // the state after the last sub-step closes the tape
    if (cudaMemcpyAsync(tape_m + (size_t)n_sub * n, m_w, 8 * n, cudaMemcpyDeviceToDevice, s) !=
        cudaSuccess)
      return LACMO_ERR_CUDA;
  }
  return cudaGetLastError() == cudaSuccess ? LACMO_OK : LACMO_ERR_CUDA;
}

int lacmo_adj_backward(int64_t n, int64_t C, const double* m_s, const double* xi,
                       const int32_t* cell, int64_t cell_stride, const double* rho_d,
                       const double* mdi, const double* dTh, const double* drv, double* dml,
                       double dt_sub, double kappa, double p_ref, double V, int n_sub,
                       int no_iter, const double* tape_m, const double* tape_c, double* lam_m,
                       double* lam_Th, double* lam_rv, double* lam_dml, double* grad_ms,
                       double* grad_kappa, double* lam_inc, void* stream) {
  if (n <= 0 || C <= 0 || !m_s || !xi || !cell || !rho_d || !mdi || !dml || n_sub < 0 ||
      cell_stride < 0 || no_iter < 0 || !tape_m || !tape_c || !lam_m || !lam_Th || !lam_rv ||
      !lam_dml || !grad_ms || !grad_kappa || !(kappa > 0.0))
    return LACMO_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  Args a = make_args(n, C, nullptr, m_s, xi, cell, nullptr, nullptr, rho_d, mdi, dTh, drv, dml,
                     dt_sub, kappa, p_ref, V, no_iter);
  if (cudaMemsetAsync(dml, 0, 8 * C, s) != cudaSuccess) return LACMO_ERR_CUDA;
  Scratch scratch(s);
  if (no_iter > 0 && n_sub > 0)   // as in lacmo_adj_forward
    a.rec = (CellFF*)scratch.get((sizeof(CellFF) + sizeof(CellGrad)) * (size_t)C);
  if (a.rec) a.grad = (CellGrad*)(a.rec + C);
  for (int k = n_sub - 1; k >= 0; --k) {
    a.cell = cell + (size_t)k * cell_stride;
    const double* mb = tape_m + (size_t)k * n;
    const double* ma = tape_m + (size_t)(k + 1) * n;
    const double* tc = tape_c + (size_t)k * 2 * C;
    k_bwd_sum_dml<<<nb(n, 128), 128, 0, s>>>(a, mb, ma);
    k_bwd_cells<<<nb(C, 32), 32, 0, s>>>(a, tc, mb, ma, lam_Th, lam_rv, lam_dml, lam_inc);
    if (a.rec)
      k_bwd_sips<true><<<nb(n, 128), 128, 0, s>>>(a, tc, mb, ma, lam_m, lam_dml, lam_Th, lam_rv,
                                                  grad_ms, grad_kappa);
    else
      k_bwd_sips<false><<<nb(n, 128), 128, 0, s>>>(a, tc, mb, ma, lam_m, lam_dml, lam_Th, lam_rv,
                                                   grad_ms, grad_kappa);
    note_launches(3);
  }
  return cudaGetLastError() == cudaSuccess ? LACMO_OK : LACMO_ERR_CUDA;
}

static bool inc_args(IncArgs* a, const double* Th, const double* r_v, const double* rdi,
                     const double* flux, int64_t nx, int64_t nz, double dx, double dz,
                     double dt_sub, const double* prof_Th, const double* prof_rv,
                     const double* t_relax) {
  if (!Th || !r_v || !rdi || !flux || nx <= 0 || nz <= 0 || !(dx > 0.0) || !(dz > 0.0))
    return false;
  if (t_relax && (!prof_Th || !prof_rv)) return false;
  a->f[0] = Th; a->f[1] = r_v; a->rdi = rdi; a->flux = flux; a->trel = t_relax;
  a->prof[0] = prof_Th; a->prof[1] = prof_rv;
  a->nx = nx; a->nz = nz; a->dx = dx; a->dz = dz; a->dt = dt_sub;
  return true;
}

int lacmo_adj_increments(const double* Th, const double* r_v, const double* rho_dry_inv,
                         const double* flux, int64_t nx, int64_t nz, double dx, double dz,
                         double dt_sub, const double* prof_Th, const double* prof_rv,
                         const double* t_relax, int second, double* inc_Th, double* inc_rv,
                         void* stream) {
  IncArgs a;
  if (!inc_args(&a, Th, r_v, rho_dry_inv, flux, nx, nz, dx, dz, dt_sub, prof_Th, prof_rv,
                t_relax) || !inc_Th || !inc_rv)
    return LACMO_ERR_ARG;
  k_increments<<<nb(2 * nx * nz, 128), 128, 0, (cudaStream_t)stream>>>(a, second ? 1 : 0,
                                                                       inc_Th, inc_rv);
  note_launches(1);
  return cudaGetLastError() == cudaSuccess ? LACMO_OK : LACMO_ERR_CUDA;
}

int lacmo_adj_increments_vjp(const double* Th, const double* r_v, const double* rho_dry_inv,
                             const double* flux, int64_t nx, int64_t nz, double dx, double dz,
                             double dt_sub, const double* prof_Th, const double* prof_rv,
                             const double* t_relax, double factor, double flux_scale,
                             const double* lam_inc, double* lam_Th, double* lam_rv,
                             double* grad_s, void* stream) {
  IncArgs a;
  if (!inc_args(&a, Th, r_v, rho_dry_inv, flux, nx, nz, dx, dz, dt_sub, prof_Th, prof_rv,
                t_relax) || !lam_inc || !lam_Th || !lam_rv || !grad_s || !(flux_scale > 0.0))
    return LACMO_ERR_ARG;
  k_increments_vjp<<<nb(2 * nx * nz, 128), 128, 0, (cudaStream_t)stream>>>(
      a, factor, flux_scale, lam_inc, lam_Th, lam_rv, grad_s);
  note_launches(1);
  return cudaGetLastError() == cudaSuccess ? LACMO_OK : LACMO_ERR_CUDA;
}

int lacmo_adj_collisions_forward(const void* events, const int64_t* off, int64_t n_groups,
                                 double* m_w, double* m_s, double* xi, void* stream) {
  if (n_groups < 0 || (n_groups > 0 && (!events || !off || !m_w || !m_s || !xi)))
    return LACMO_ERR_ARG;
  if (n_groups == 0) return LACMO_OK;
  k_ev_forward<<<ev_blocks(n_groups), 32, 0, (cudaStream_t)stream>>>(
      (const EvRec*)events, off, n_groups, m_w, m_s, xi);
  note_launches(1);
  return cudaGetLastError() == cudaSuccess ? LACMO_OK : LACMO_ERR_CUDA;
}

int lacmo_adj_collisions_backward(const void* events, const int64_t* off, int64_t n_groups,
                                  double* lam_w, double* lam_s, void* stream) {
  if (n_groups < 0 || (n_groups > 0 && (!events || !off || !lam_w || !lam_s)))
    return LACMO_ERR_ARG;
  if (n_groups == 0) return LACMO_OK;
  k_ev_backward<<<ev_blocks(n_groups), 32, 0, (cudaStream_t)stream>>>(
      (const EvRec*)events, off, n_groups, lam_w, lam_s);
  note_launches(1);
  return cudaGetLastError() == cudaSuccess ? LACMO_OK : LACMO_ERR_CUDA;
}

}  // extern "C"
