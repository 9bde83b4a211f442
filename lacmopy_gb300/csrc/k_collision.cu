// All-or-nothing (AON) collision kernels, bit-exact with the reference.
//
// The reference visits the pairs (i, j), i < j, of a cell in lexicographic
// order and each pair may update SIPs i and j (collision/all_or_nothing.py:
// 553-633).  Two pairs that share no SIP commute exactly, and every pair that
// shares a SIP with (i, j) and comes earlier lexicographically has a smaller
// index sum i + j, every later one a larger sum.  So processing the
// anti-diagonals s = i + j = 1 .. 2n-3 in order, the pairs of one diagonal in
// parallel, gives the sequential result bit for bit: 2n-3 barrier steps of at
// most n/2 independent pairs.  The collision counters are integer sums.
//
// Bit-exactness also needs the reference's floating-point operation order
// (this file is compiled with -fmad=false, so no a*b+c is fused) and the same
// pow/log values: the radius (3/(4 pi) m/rho)^(1/3) and the kernel bin
// int((log R - a)/b + 0.5) use the correctly-rounded routines of
// lacmo_crmath.h.  Draws come either from an injected buffer in the
// reference's consumption order or from Philox4x32-10.
#include <cuda_runtime.h>

#include <atomic>

#include "lacmo_colmath.cuh"

namespace lacmo {

// ---------------------------------------------------------------------------
// 2-D cells: one warp per cell (collision/all_or_nothing.py:498-635, 637-751,
// 754-846).  SIP state of cells with up to CELL_SMEM SIPs lives in shared
// memory; larger cells use per-SIP global scratch.
constexpr int CELL_SMEM = 256;
constexpr int CELL_WARPS = 8;

// one collection of the sequential order, as a log record for the adjoint's
// replay (recorded events): kind 0 ordinary, 1 equal-xi split (a, b: xi of
// imin and imax before), 2 multiple collection (a: p_crit)
struct EvRec {
  int32_t imin, imax, kind, pad;
  double a, b;
};

struct CellArgs {
  EvRec* log;                       // event log (single states), or null
  int64_t log_cap;
  unsigned long long* log_count;
  double *xi, *m_w, *m_s;
  const double* vel;
  const double* T;
  const int32_t *start, *perm;
  const int64_t* draw_off;
  int64_t n, C;
  double dtdv;
  const double* E;
  double E_const;
  int64_t nb;
  double lo, bl;
  int sol;
  const double* draws;
  int64_t n_draws;
  uint64_t seed;
  const int64_t *cursor, *col_step, *total_pairs;
  int64_t* no_cols;
  uint32_t* flags;
  double *gR, *grho;   // per slot: exact radius and density
  int32_t* gk;         // per slot: exact kernel bin, GK_NONE or GK_STALE
  float dtdv_f, lo_f, inv_bl_f, E_const_f;   // FP32 copies for the screen
  float bin_margin;    // distance from a bin edge below which the FP32 bin is not trusted
  const float* Ef;     // FP32 efficiency table, or null (then E is read and rounded)
  const int32_t* cell_order;   // cells, largest first
  int32_t* cell_ctr;           // next cell_order entry to take
  float* gcopy;                // [6][n] FP32 copies by slot, for cells above CELL_SMEM
  float4* gstats;              // block statistics of cells above CELL_SMEM (thinned draws)
  const float* erow;           // largest FP32 efficiency of each table row (thinned draws)
  const float* ecap;           // the same as a bound: infinity for a row with a NaN
  int thin;                    // thinned Philox draws (lacmo_thin.h)
  float cmax;                  // surely_skips' factor for the whole table
  int64_t draw_base;           // *cursor
  uint64_t cstep;              // *col_step
};

// A block's dynamic shared memory: its arguments (all its warps belong to one
// member), then a slice per warp.
constexpr size_t CELL_ARGS_BYTES = (sizeof(CellArgs) + 15) / 16 * 16;
constexpr size_t CELL_WARP_BYTES = (size_t)CELL_SMEM * (4 * 4 + 4 + 4) + (CELL_SMEM / 32) * 32;
__device__ __forceinline__ CellArgs& cell_args() {
  extern __shared__ float4 fsm[];
  return *(CellArgs*)fsm;
}

// the parameters a collision step shares across members
struct CellCommon {
  EvRec* log;
  int64_t log_cap;
  unsigned long long* log_count;
  double dtdv;
  const double* E;
  double E_const;
  int64_t nb;
  double lo, bl;
  int sol;
  const double* draws;
  int64_t n_draws;
  float dtdv_f, lo_f, inv_bl_f, E_const_f, bin_margin;
  const float* Ef;
  const float *erow, *ecap;
  int thin;
};
struct CK {
  MRef m;
  CellCommon cc;
};
__device__ __forceinline__ void make_cellargs(CellArgs& a, const Member& mb, const CellCommon& cc) {
  a.log = cc.log; a.log_cap = cc.log_cap; a.log_count = cc.log_count;
  a.xi = mb.sp.xi; a.m_w = mb.sp.m_w; a.m_s = mb.sp.m_s; a.vel = mb.sp.vel;
  a.T = mb.g.scalar_fields;
  a.start = mb.w.start; a.perm = mb.w.perm; a.draw_off = mb.w.draw_off;
  a.n = mb.sp.n; a.C = mb.g.nx * mb.g.nz;
  a.dtdv = cc.dtdv; a.E = cc.E; a.E_const = cc.E_const; a.nb = cc.nb; a.lo = cc.lo; a.bl = cc.bl;
  a.sol = cc.sol; a.draws = cc.draws; a.n_draws = cc.n_draws; a.seed = mb.seed;
  a.cursor = mb.w.cursor; a.col_step = mb.w.col_step; a.total_pairs = mb.w.total_pairs;
  a.no_cols = mb.sp.no_cols; a.flags = mb.w.flags;
  a.gR = mb.w.colR; a.grho = mb.w.colrho; a.gk = mb.w.colk;
  a.dtdv_f = cc.dtdv_f; a.lo_f = cc.lo_f; a.inv_bl_f = cc.inv_bl_f; a.E_const_f = cc.E_const_f;
  a.bin_margin = cc.bin_margin;
  a.Ef = cc.Ef;
  a.cell_order = mb.w.cell_order; a.cell_ctr = mb.w.cell_ctr;
  a.gcopy = mb.w.gcopy;
  a.gstats = (float4*)mb.w.gstats;
  a.erow = cc.erow;
  a.ecap = cc.ecap;
  a.thin = cc.thin;
}

// Exact per-SIP collision data (collision/all_or_nothing.py:812-826), kept
// in gR / grho / gk by slot (a cell's lie side by side) and computed on first
// need.  The density belongs to the step-start masses and the cell temperature
// (the reference keeps it for the whole step); the radius and its kernel bin
// follow from the current masses and that density, which the reference
// recomputes after every collection (all_or_nothing.py:596-633).  A radius only
// matters when an exact evaluation reads it, so after a collection it is
// recomputed lazily:
//   gk = GK_NONE:  nothing computed; the masses are still those of the step's start
//                  (whoever changes them computes the density first)
//   gk = GK_STALE: grho holds the density; gR, gk are out of date
//   gk >= 0:       gR, gk are the exact radius and bin of the current masses
constexpr int32_t GK_NONE = -1, GK_STALE = -2;
__device__ __forceinline__ double density_of(const CellArgs& a, double m_p, double ms, double Tc) {
  const double w_s = ms / m_p;
  return (a.sol == SOL_AS) ? density_water(Tc) * poly_rho_AS(w_s)
                           : density_NaCl_solution(w_s, Tc);
}
__device__ __noinline__ void compute_density(int32_t id, int32_t s, double Tc) {
  const CellArgs& a = cell_args();
  const double ms = a.m_s[id];
  a.grho[s] = density_of(a, a.m_w[id] + ms, ms, Tc);
  a.gk[s] = GK_STALE;
}
__device__ __forceinline__ void ensure_density(const CellArgs& a, int32_t id, int32_t s, double Tc) {
  if (a.gk[s] == GK_NONE) compute_density(id, s, Tc);
}
__device__ __noinline__ void compute_exact(int32_t id, int32_t s, double Tc,
                                           bool use_E) {
  const CellArgs& a = cell_args();
  ensure_density(a, id, s, Tc);
  const double R = col_radius(a.m_w[id] + a.m_s[id], a.grho[s]);
  a.gR[s] = R;
  a.gk[s] = use_E ? col_bin_f(R, a.lo, a.bl, a.nb, a.lo_f, a.inv_bl_f, a.bin_margin) : 0;
}
// the exact kernel bin of SIP id from its current masses, stored nowhere
__device__ __noinline__ int32_t exact_bin_of(int32_t id, double Tc) {
  const CellArgs& a = cell_args();
  const double m_p = a.m_w[id] + a.m_s[id];
  return col_bin(col_radius(m_p, density_of(a, m_p, a.m_s[id], Tc)), a.lo, a.bl, a.nb);
}
__device__ __forceinline__ void ensure_exact(const CellArgs& a, int32_t id, int32_t s, double Tc,
                                             bool use_E) {
  if (a.gk[s] < 0) compute_exact(id, s, Tc, use_E);
}

// FP32 copies of a cell's SIPs: v = (xi, R, u, w) per SIP, the kernel bin
// and the SIP ID, and for thinned draws the statistics of block b at st[2b],
// st[2b + 1]; base is the cell's first slot.  They lie in a warp's shared-memory
// slice or, for cells above its size (BIG), in the cell's slots of the global
// scratch.  The slice is known by the warp's index and the arguments by their
// place in shared memory: pointers to either held some ten registers of every
// thread, and what they pushed out to local memory did not fit into L1 beside the
// slices (a step of the 64-member ensemble 4.10 ms with pointers, 3.91 ms without;
// of 12 raining members, thinned, 3.28 and 3.08 ms).
template <bool BIG>
struct Cell;
template <>
struct Cell<false> {
  int w;
  int32_t base;
  __device__ __forceinline__ float4* v() const {
    extern __shared__ float4 fsm[];
    return (float4*)((char*)fsm + CELL_ARGS_BYTES + (size_t)w * CELL_WARP_BYTES);
  }
  __device__ __forceinline__ int32_t* sk() const { return (int32_t*)(v() + CELL_SMEM); }
  __device__ __forceinline__ int32_t* sid() const { return sk() + CELL_SMEM; }
  __device__ __forceinline__ float4* st() const { return (float4*)(sid() + CELL_SMEM); }
};
template <>
struct Cell<true> {
  float4* v_;
  int32_t *sk_, *sid_;
  float4* st_;
  int32_t base;
  __device__ __forceinline__ float4* v() const { return v_; }
  __device__ __forceinline__ int32_t* sk() const { return sk_; }
  __device__ __forceinline__ int32_t* sid() const { return sid_; }
  __device__ __forceinline__ float4* st() const { return st_; }
};

// SIP id's masses changed in a collection: its exact radius and bin become
// stale, and its FP32 copies at slot l of the cell follow now from the FP32 masses
// and the step-start density (the radius within the screen's 1e-6, as at the
// cell's load; a bin near an edge is computed exactly, as there).
template <bool BIG>
__device__ __noinline__ void masses_changed(Cell<BIG> S, int32_t id,
                                            int l, double Tc, bool use_E) {
  const CellArgs& a = cell_args();
  const int32_t s = S.base + l;
  a.gk[s] = GK_STALE;
  const float Rf = lt_cbrtf((float)LC_FOUR_PI_OVER_THREE_INV * d2f_rn(a.m_w[id] + a.m_s[id]) /
                            d2f_rn(a.grho[s]));
  int32_t kb = 0;
  if (use_E) {
    const float v = (__logf(Rf) - a.lo_f) * a.inv_bl_f + 0.5f;
    const float fl = floorf(v);
    if (v - fl > a.bin_margin && (fl + 1.0f) - v > a.bin_margin && v > -1e6f && v < 1e6f &&
        Rf > 0.f) {
      kb = __float2int_rz(fl);
      kb = kb < 0 ? 0 : (kb > a.nb - 1 ? (int32_t)a.nb - 1 : kb);
    } else {
      compute_exact(id, s, Tc, use_E);
      kb = a.gk[s];
    }
  }
  S.v()[l].y = Rf;
  S.sk()[l] = kb;
}

// append a collection to the event log; a cell's events come from one warp
// in its sequential order, one at a time, so their slots increase in that
// order (slots past the capacity are counted, not written)
__device__ __noinline__ void log_event(int32_t imin, int32_t imax, int kind,
                                       double x, double y) {
  const CellArgs& a = cell_args();
  const unsigned long long slot = atomicAdd(a.log_count, 1ull);
  if (slot < (unsigned long long)a.log_cap) {
    EvRec r;
    r.imin = imin; r.imax = imax; r.kind = kind; r.pad = 0; r.a = x; r.b = y;
    a.log[slot] = r;
  }
}

// One ordinary collection (p_crit <= 1 and p_crit > r) of the pair imin/imax
// (collision/all_or_nothing.py:607-633), at the cell's slots lmin/lmax; the
// density of imin must be known.
template <bool BIG>
__device__ __forceinline__ void collect_once(const CellArgs& a, Cell<BIG> S, int32_t imin,
                                             int32_t imax, int lmin, int lmax, double Tc,
                                             bool use_E) {
  double *XI = a.xi, *MW = a.m_w, *MS = a.m_s;
  const int32_t smin = S.base + lmin, smax = S.base + lmax;
  const double xi_min = XI[imin], xi_max = XI[imax];
  const double m_w_min = MW[imin], m_w_max = MW[imax];
  const double m_s_min = MS[imin], m_s_max = MS[imax];
  const double xi_rel_dev = (xi_max - xi_min) / xi_max;
  if (xi_rel_dev < 1.0E-5) {
    if (a.log) log_event(imin, imax, 1, xi_min, xi_max);
    // both radii follow from imin's density (all_or_nothing.py:615-624):
    // computed now, not left stale
    ensure_density(a, imax, smax, Tc);
    const double xi_ges = xi_min + xi_max;
    MW[imin] = 2.0 * (xi_min * m_w_min + xi_max * m_w_max) / xi_ges;
    MS[imin] = 2.0 * (xi_min * m_s_min + xi_max * m_s_max) / xi_ges;
    MW[imax] = MW[imin];
    MS[imax] = MS[imin];
    const double R = col_radius((MW[imin] + MS[imin]), a.grho[smin]);
    XI[imax] = 0.5 * 0.7 * xi_ges;
    XI[imin] = 0.5 * xi_ges - XI[imax];
    const int32_t gk =
        use_E ? col_bin_f(R, a.lo, a.bl, a.nb, a.lo_f, a.inv_bl_f, a.bin_margin) : 0;
    a.gR[smin] = a.gR[smax] = R;
    a.gk[smin] = a.gk[smax] = gk;
    S.v()[lmin].x = d2f_rn(XI[imin]); S.v()[lmax].x = d2f_rn(XI[imax]);
    S.v()[lmin].y = S.v()[lmax].y = d2f_rn(R);
    S.sk()[lmin] = S.sk()[lmax] = gk;
  } else {
    if (a.log) log_event(imin, imax, 0, 0.0, 0.0);
    MW[imin] += m_w_max;
    MS[imin] += m_s_max;
    XI[imax] -= xi_min;
    masses_changed(S, imin, lmin, Tc, use_E);
    S.v()[lmax].x = d2f_rn(XI[imax]);
  }
}

// Exact FP64 evaluation of the pair ii/jj (collision/all_or_nothing.py:
// 553-633) in the reference's operation order, at the cell's slots li/lj.
// Returns 0 (no collision), 1 (one collection) or 2 (multiple collection).
template <bool BIG>
__device__ __noinline__ int exact_pair(Cell<BIG> S, int32_t ii, int32_t jj,
                                       int li, int lj, double Tc, bool use_E, double r) {
  const CellArgs& a = cell_args();
  const int32_t si = S.base + li, sj = S.base + lj;
  ensure_exact(a, ii, si, Tc, use_E);
  ensure_exact(a, jj, sj, Tc, use_E);
  double *XI = a.xi, *MW = a.m_w, *MS = a.m_s;
  const double *U = a.vel, *W = a.vel + a.n;
  int32_t imin, imax;
  int lmin, lmax;
  if (XI[ii] <= XI[jj]) { imin = ii; imax = jj; lmin = li; lmax = lj; }
  else { imin = jj; imax = ii; lmin = lj; lmax = li; }
  const double xi_min = XI[imin], xi_max = XI[imax];
  const double Rs = a.gR[si] + a.gR[sj];
  const double e = use_E ? __ldg(a.E + (int64_t)a.gk[si] * a.nb + a.gk[sj]) : a.E_const;
  const double du = U[ii] - U[jj], dw = W[ii] - W[jj];
  const double dv = sqrt(du * du + dw * dw);
  const double p_crit = xi_max * a.dtdv * (LC_PI * Rs * Rs * e * dv * 1.0E-12);
  if (p_crit > 1.0) {
    if (a.log) log_event(imin, imax, 2, p_crit, 0.0);
    const double xi_col = p_crit * xi_min;
    MW[imin] = MW[imin] + p_crit * MW[imax];
    MS[imin] = MS[imin] + p_crit * MS[imax];
    XI[imax] -= xi_col;
    masses_changed(S, imin, lmin, Tc, use_E);
    S.v()[lmax].x = d2f_rn(XI[imax]);
    return 2;
  }
  if (!(p_crit > r)) return 0;
  collect_once(a, S, imin, imax, lmin, lmax, Tc, use_E);
  return 1;
}

// A pair the FP32 bounds place certainly in an ordinary collection.
template <bool BIG>
__device__ __noinline__ void certain_collection(Cell<BIG> S, int i, int j,
                                                double Tc, bool use_E) {
  const CellArgs& a = cell_args();
  const int32_t ii = S.sid()[i], jj = S.sid()[j];
  const bool lo_i = a.xi[ii] <= a.xi[jj];
  const int32_t imin = lo_i ? ii : jj, imax = lo_i ? jj : ii;
  const int lmin = lo_i ? i : j, lmax = lo_i ? j : i;
  ensure_density(a, imin, S.base + lmin, Tc);
  collect_once(a, S, imin, imax, lmin, lmax, Tc, use_E);
}

// all_or_nothing.py:609-610 (out of line: the compiler would run the quotient's
// chain of FP64 operations in every event)
__device__ __noinline__ bool equal_multiplicities(double xi_min, double xi_max) {
  return (xi_max - xi_min) / xi_max < 1.0E-5;
}
// One event of a cell's sequential order, taken by a whole warp: the pair of slots
// (l0, l1) with draw r, either placed certainly in an ordinary collection by the
// FP32 bounds (certain) or evaluated exactly.  Even lanes hold SIP l0, odd lanes
// SIP l1 (lanes 0 and 1 write): both SIPs' loads, densities and radii run side by
// side, and the updated masses stay in registers for the FP32 copies instead of
// being read back, so an event costs one round of loads and one chain of FP64
// operations (its latency is what a raining cell waits for; some 100 cycles an
// operation, so the test for equal multiplicities runs in FP32 and the density of
// imax is left out where nothing reads it). Keeping SIP l0 in registers over all
// events of its row, its partners' data formed in all lanes at once, was slower (a
// step of the raining 75 x 75 x 128 state 1.20 ms against 0.94 ms): most rows hold
// one event.  Same decisions and operation order as exact_pair and collect_once.
// Returns 0 (no collision), 1 (one collection) or 2 (multiple collection), the same
// in all lanes.
template <bool THIN, bool BIG>
__device__ __forceinline__ int warp_event(Cell<BIG> S, int l0, int l1, double Tc,
                                       bool use_E, double r, bool certain) {
  const CellArgs& a = cell_args();
  constexpr unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, me = lane & 1;
  const bool writes = lane < 2;
  const int l = me ? l1 : l0;
  const int32_t id = S.sid()[l];
  // one round of independent loads
  double xi = a.xi[id];
  double mw = a.m_w[id], ms = a.m_s[id];
  const int32_t s = S.base + l;
  int32_t gk = a.gk[s];
  double R = a.gR[s], rho = a.grho[s];
  const double u = certain ? 0.0 : a.vel[id], w = certain ? 0.0 : a.vel[a.n + id];
  const double xo = __shfl_xor_sync(FULL, xi, 1);
  // imin is l0's SIP when XI[ii] <= XI[jj], else l1's
  const double x0 = me ? xo : xi, x1 = me ? xi : xo;
  const bool lo0 = x0 <= x1;
  const bool is_min = (me == 0) == lo0;
  if (gk == GK_NONE && (!certain || is_min)) {
    rho = density_of(a, mw + ms, ms, Tc);
    gk = GK_STALE;
    if (writes) { a.grho[s] = rho; a.gk[s] = gk; }
  }
  double p_crit = 0.0;
  if (!certain) {
    if (gk < 0) {
      R = col_radius(mw + ms, rho);
      gk = use_E ? col_bin_f(R, a.lo, a.bl, a.nb, a.lo_f, a.inv_bl_f, a.bin_margin) : 0;
      if (writes) { a.gR[s] = R; a.gk[s] = gk; }
    }
    const int32_t go = __shfl_xor_sync(FULL, gk, 1);
    const double Ro = __shfl_xor_sync(FULL, R, 1);
    const double e = use_E ? __ldg(a.E + (int64_t)(me ? go : gk) * a.nb + (me ? gk : go))
                           : a.E_const;
    const double du = u - __shfl_xor_sync(FULL, u, 1), dw = w - __shfl_xor_sync(FULL, w, 1);
    const double dv = sqrt(du * du + dw * dw);
    const double Rs = R + Ro;
    const double xi_max = lo0 ? x1 : x0;
    p_crit = xi_max * a.dtdv * (LC_PI * Rs * Rs * e * dv * 1.0E-12);
    if (!(p_crit > 1.0) && !(p_crit > r)) {
      __syncwarp();   // orders the scratch writes before the next event's loads
      return 0;
    }
  }
  const double mwo = __shfl_xor_sync(FULL, mw, 1), mso = __shfl_xor_sync(FULL, ms, 1);
  const int32_t ido = __shfl_xor_sync(FULL, id, 1);
  const int32_t imin = is_min ? id : ido, imax = is_min ? ido : id;
  const double xi_min = lo0 ? x0 : x1, xi_max = lo0 ? x1 : x0;
  int out = 1;
  bool split = false;
  if (p_crit > 1.0) {
    out = 2;
    if (a.log && lane == 0) log_event(imin, imax, 2, p_crit, 0.0);
    if (is_min) {
      mw = mw + p_crit * mwo;
      ms = ms + p_crit * mso;
    } else {
      xi -= p_crit * xi_min;
    }
  } else {
    // xi_rel_dev < 1e-5: the FP32 copies decide where they are clear of the limit
    const float xf = d2f_flush(xi), xof = __shfl_xor_sync(FULL, xf, 1);
    const float xmaxf = fmaxf(xf, xof);
    if (!(xmaxf - fminf(xf, xof) > 2.0E-5f * xmaxf && xmaxf < 3.0E38f && fminf(xf, xof) > 0.0f))
      split = equal_multiplicities(xi_min, xi_max);
    if (!split) {
      if (a.log && lane == 0) log_event(imin, imax, 0, 0.0, 0.0);
      if (is_min) {
        mw += mwo;
        ms += mso;
      } else {
        xi -= xi_min;
      }
    } else {
      if (a.log && lane == 0) log_event(imin, imax, 1, xi_min, xi_max);
      if (gk == GK_NONE) {
        // imax's density belongs to its step-start masses
        rho = density_of(a, mw + ms, ms, Tc);
        if (writes) a.grho[s] = rho;
      }
      const double rhoo = __shfl_xor_sync(FULL, rho, 1);
      const double xi_ges = xi_min + xi_max;
      const double w_min = is_min ? mw : mwo, w_max = is_min ? mwo : mw;
      const double s_min = is_min ? ms : mso, s_max = is_min ? mso : ms;
      mw = 2.0 * (xi_min * w_min + xi_max * w_max) / xi_ges;
      ms = 2.0 * (xi_min * s_min + xi_max * s_max) / xi_ges;
      // both radii follow from imin's density (all_or_nothing.py:615-624)
      R = col_radius(mw + ms, is_min ? rho : rhoo);
      const double xm = 0.5 * 0.7 * xi_ges;
      xi = is_min ? 0.5 * xi_ges - xm : xm;
      gk = use_E ? col_bin_f(R, a.lo, a.bl, a.nb, a.lo_f, a.inv_bl_f, a.bin_margin) : 0;
    }
  }
  // the FP32 copies.  imin's exact radius and bin become stale (masses_changed);
  // everything is formed before the first store, after which the compiler reads
  // a's and S's members again
  float Rf = 0.0f;
  int32_t kb = 0;
  const float xif = d2f_rn(xi);
  bool exact = split;   // R and gk are new
  if (split) {
    Rf = d2f_rn(R);
    kb = gk;
  } else {
    const float mf = (float)LC_FOUR_PI_OVER_THREE_INV * d2f_rn(mw + ms), rf = d2f_rn(rho);
    Rf = THIN ? lt_cbrtf(mf / rf) : f_cbrt(mf * f_rcp(rf));
    gk = GK_STALE;
    if (use_E) {
      const float v = (__logf(Rf) - a.lo_f) * a.inv_bl_f + 0.5f;
      const float fl = floorf(v);
      if (v - fl > a.bin_margin && (fl + 1.0f) - v > a.bin_margin && v > -1e6f && v < 1e6f &&
          Rf > 0.f) {
        kb = __float2int_rz(fl);
        kb = kb < 0 ? 0 : (kb > a.nb - 1 ? (int32_t)a.nb - 1 : kb);
      } else if (is_min) {
        R = col_radius(mw + ms, rho);
        kb = gk = col_bin_f(R, a.lo, a.bl, a.nb, a.lo_f, a.inv_bl_f, a.bin_margin);
        exact = true;
      }
    }
  }
  if (writes) {
    if (is_min || split) {
      a.m_w[id] = mw;
      a.m_s[id] = ms;
      if (exact) a.gR[s] = R;
      a.gk[s] = gk;
      S.v()[l].y = Rf;
      S.sk()[l] = kb;
    }
    if (!is_min || split) {
      a.xi[id] = xi;
      S.v()[l].x = xif;
    }
  }
  __syncwarp();   // orders the stores before the next event's loads
  return out;
}

__device__ __noinline__ double philox_from_bits(uint64_t k53) {
  return (double)k53 * (1.0 / 9007199254740992.0);
}
// a pair's draw from its two words: an injected double's bits, or Philox's
__device__ __forceinline__ double draw_of(bool injected, uint64_t w) {
  if (injected) return __longlong_as_double((long long)w);
  return philox_from_bits((w >> 37) * 67108864ull + (uint64_t)((uint32_t)w >> 6));
}

// FP32 screen of the pair (i, j): 0 = certainly no collision, 1 = certainly
// one ordinary collection (0 < p_crit <= 1 and p_crit > r), 2 = undecided
// (the exact FP64 evaluation decides).  Two-sided bounds of p_crit: the FP32
// radii are within 1e-6 (relative) of the exact ones, every other FP32
// operation and conversion within 2^-24, the velocity difference carries an
// absolute slack for its cancellation, and the bounds are widened by 2^-14
// relative (and 1e-36 absolute); |du| + |dw| in place of the Euclidean norm
// gives a looser upper bound that decides most skips alone.  Non-positive
// multiplicities (left by multiple collections) are undecided.  [r_lo, r_hi]
// brackets the draw.
__device__ __forceinline__ int screen_pair(const CellArgs& a, bool use_E, float4 vi, int32_t ki,
                                           float4 vj, int32_t kj, float r_lo, float r_hi) {
  const float du = vi.z - vj.z, dw = vi.w - vj.w;
  const float adu = fabsf(du), adw = fabsf(dw);
  const float slack = 0x1p-21f * (fabsf(vi.z) + fabsf(vj.z) + fabsf(vi.w) + fabsf(vj.w));
  const float rs = vi.y + vj.y;
  float ef = a.E_const_f;
  if (use_E) {
    const int64_t ke = (int64_t)ki * a.nb + kj;
    ef = a.Ef ? __ldg(a.Ef + ke) : d2f_flush(__ldg(a.E + ke));
  }
  const float core = ((fmaxf(vi.x, vj.x) * a.dtdv_f) * (float)(LC_PI * 1.0E-12)) * rs * rs * ef;
  const bool sane = vi.x > 0.0f && vj.x > 0.0f && core >= 1e-30f;
  // common case first: |du| + |dw| >= |(du, dw)| gives an upper bound without
  // the square root, enough to skip the pair when the draw is above it
  const float p_l1 = core * ((adu + adw) + slack) * (1.0f + 0x1p-14f) + 1e-36f;
  if (sane && p_l1 < 1.0f && p_l1 < r_lo) return 0;
  const float dvm = sqrtf(du * du + dw * dw);
  const float p_hi = core * (dvm + slack) * (1.0f + 0x1p-14f) + 1e-36f;
  const float p_lo = core * fmaxf(dvm - slack, 0.0f) * (1.0f - 0x1p-14f);
  const bool ok = sane && p_hi < 1.0f;
  if (ok && p_hi < r_lo) return 0;
  if (ok && p_lo > r_hi) return 1;
  return 2;
}
// draw intervals: Philox bits (exact: r - r_lo < 2^-24) or an injected draw
// (an injected draw outside [0, 1) gives an empty interval: undecided)
__device__ __forceinline__ void philox_interval(uint64_t k53, float& r_lo, float& r_hi) {
  r_lo = (float)(uint32_t)(k53 >> 29) * 0x1p-24f;
  r_hi = r_lo + 0x1p-24f;
}
__device__ __forceinline__ void injected_interval(double r, float& r_lo, float& r_hi) {
  const uint64_t rb = (uint64_t)__double_as_longlong(r);
  const bool in01 = rb < 0x3ff0000000000000ull;
  r_lo = in01 ? d2f_down_pos(r) : 2.0f;
  r_hi = in01 ? r_lo + 0x1p-24f : -1.0f;
}

// First screen of the per-pair draws, without a table look-up: the pair of
// SIPs vi and vj is certainly no collision when screen_pair's upper bound with
// the table's largest efficiency (folded into cmax with dt/dV, pi 1e-12 and the
// bound's 2^-14 slack) lies below r, a lower bound of the draw that is 0 or at
// least 2^-24 (a product flushed to zero belongs to a p_crit far below that).
// NaN and non-positive multiplicities never pass.
__device__ __forceinline__ bool surely_skips(float4 vi, float4 vj, float cmax, float r) {
  const float dv = fabsf(vi.z - vj.z) + fabsf(vi.w - vj.w);
  const float sl = (fabsf(vi.z) + fabsf(vi.w)) + (fabsf(vj.z) + fabsf(vj.w));
  const float rs = vi.y + vj.y;
  const float p = ((fmaxf(vi.x, vj.x) * cmax) * (rs * rs)) * (dv + 0x1p-21f * sl) + 1e-36f;
  return p < r && vi.x > 0.0f && vj.x > 0.0f;
}
// no exact data yet for the cell's n SIPs
template <bool BIG>
__device__ __forceinline__ void init_exact_scratch(const CellArgs& a, Cell<BIG> S, int n,
                                                   int lane) {
  for (int q = lane; q < n; q += 32) a.gk[S.base + q] = GK_NONE;
  __syncwarp();
}

// The events of one window of the per-pair draws (k_collide_cells), taken in their
// order: screen_pair places the pairs the first screen left (bits of ev.m), the
// first one it does not skip is the next event, and after a collection the window's
// later pairs are screened again with the draws they already have; an event that
// changes nothing leaves the later screens valid.  Out of line: the window loop
// around it then reloads nothing (a step of 5625 cells of 64 SIPs, fresh: 124 us
// with the events in the loop, 74 us without).  An event costs one more screen of
// its window, where letting every lane run on to its own first hit cost a screen of
// the whole rest of the cell: a step of a raining 75 x 75 x 128 state (14
// collections per cell on average, 190 in the heaviest, whose chain of events of
// some 5 us each is what the step waits for) took 10.6 ms, 0.78 ms now.
// Returns false when a limit is passed, of collections or of undecided pairs that
// change nothing (ev.pos: the first rank left).
struct PairEvents {
  int pos, events, idle, c0, c1;
  uint32_t m;
};
__device__ __noinline__ PhiloxBlock injected_couple(const double* rnd, int p, int P) {
  PhiloxBlock x = {0, 0, 0, 0};
  if (p < P) {
    const uint64_t q = (uint64_t)__double_as_longlong(rnd[p]);
    x.x0 = (uint32_t)(q >> 32); x.x1 = (uint32_t)q;
  }
  if (p + 1 < P) {
    const uint64_t q = (uint64_t)__double_as_longlong(rnd[p + 1]);
    x.x2 = (uint32_t)(q >> 32); x.x3 = (uint32_t)q;
  }
  return x;
}
template <bool BIG>
__device__ __noinline__ bool window_events(Cell<BIG> S, int n, int P, int w0,
                                           int i, int j, PhiloxBlock x, float cmax, double Tc,
                                           bool use_E, bool injected, int event_limit,
                                           int idle_limit, PairEvents& ev) {
  const CellArgs& a = cell_args();
  constexpr unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const bool same = j < n - 1;
  const int i2 = same ? i : i + 1, j2 = same ? j + 1 : i + 2;
  const int p = w0 + 2 * lane;
  uint32_t m = ev.m;
  ev.c0 = ev.c1 = 0;
  for (;;) {
    uint32_t sc = 0;   // screen_pair's answers, two bits per pair
    float r_lo, r_hi;
    if (m & 1u) {
      if (injected) injected_interval(__hiloint2double((int)x.x0, (int)x.x1), r_lo, r_hi);
      else philox_interval(philox_half53(x, false), r_lo, r_hi);
      sc = (uint32_t)screen_pair(a, use_E, S.v()[i], S.sk()[i], S.v()[j], S.sk()[j], r_lo, r_hi);
    }
    if (m & 2u) {
      if (injected) injected_interval(__hiloint2double((int)x.x2, (int)x.x3), r_lo, r_hi);
      else philox_interval(philox_half53(x, true), r_lo, r_hi);
      sc |= (uint32_t)screen_pair(a, use_E, S.v()[i2], S.sk()[i2], S.v()[j2], S.sk()[j2], r_lo, r_hi) << 2;
    }
    int done = w0;
    bool changed = false;
    unsigned hits;
    while (!changed && (hits = __ballot_sync(FULL, sc != 0)) != 0) {
      if (ev.events == 0) {
        init_exact_scratch(a, S, n, lane);
        ev.events = 1;
      }
      const int L = __ffs(hits) - 1;
      const uint32_t scL = __shfl_sync(FULL, sc, L);
      const bool sec = (scL & 3u) == 0;
      const uint64_t dr = ((uint64_t)(sec ? x.x2 : x.x0) << 32) | (sec ? x.x3 : x.x1);
      const int o = warp_event<false>(S, __shfl_sync(FULL, sec ? i2 : i, L),
                               __shfl_sync(FULL, sec ? j2 : j, L), Tc, use_E,
                               draw_of(injected, __shfl_sync(FULL, dr, L)),
                               (sec ? scL >> 2 : scL & 3u) == 1u);
      if (lane == L) {
        ev.c0 += o == 1;
        ev.c1 += o == 2;
        sc &= sec ? 3u : 12u;
      }
      done = w0 + 2 * L + (sec ? 2 : 1);
      changed = o != 0;
      if (changed ? ++ev.events > event_limit : ++ev.idle > idle_limit) {
        ev.pos = done;
        return false;
      }
    }
    if (!changed) break;
    const float r0 = injected ? low_of_double(__hiloint2double((int)x.x0, (int)x.x1))
                              : low_of_word(x.x0);
    const float r1 = injected ? low_of_double(__hiloint2double((int)x.x2, (int)x.x3))
                              : low_of_word(x.x2);
    m = 0;
    if (p < P && p >= done && !surely_skips(S.v()[i], S.v()[j], cmax, r0)) m = 1;
    if (p + 1 < P && p + 1 >= done && !surely_skips(S.v()[i2], S.v()[j2], cmax, r1)) m |= 2;
  }
  ev.pos = w0 + 64;
  return true;
}

// order-preserving keys of non-NaN floats (for warp min/max reductions)
__device__ __forceinline__ uint32_t ord_key(float f) {
  const uint32_t b = __float_as_uint(f);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float ord_val(uint32_t k) {
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

// statistics (lt_block_stats) of block b, slots [32 b, min(32 b + 32, n)),
// from the FP32 copies, warp-cooperative: st[2b] = (xmax, Rmax, umin, umax),
// st[2b + 1] = (wmin, wmax, ok, 0)
template <bool BIG>
__device__ __forceinline__ void block_stats(Cell<BIG> S, int n, int b, int lane) {
  constexpr unsigned FULL = 0xffffffffu;
  const int q = (b << 5) + lane;
  const bool in = q < n;
  const float4 v = in ? S.v()[q] : make_float4(1.0f, 0.0f, 0.0f, 0.0f);
  const bool bad = in && !(v.x > 0.0f && v.y == v.y && v.z == v.z && v.w == v.w);
  const int ok = __ballot_sync(FULL, bad) == 0u;
  const uint32_t xk = __reduce_max_sync(FULL, in ? ord_key(v.x) : 0u);
  const uint32_t Rk = __reduce_max_sync(FULL, in ? ord_key(v.y) : 0u);
  const uint32_t ulo = __reduce_min_sync(FULL, in ? ord_key(v.z) : 0xffffffffu);
  const uint32_t uhi = __reduce_max_sync(FULL, in ? ord_key(v.z) : 0u);
  const uint32_t wlo = __reduce_min_sync(FULL, in ? ord_key(v.w) : 0xffffffffu);
  const uint32_t whi = __reduce_max_sync(FULL, in ? ord_key(v.w) : 0u);
  if (lane == 0) {
    S.st()[2 * b] = make_float4(ord_val(xk), ord_val(Rk), ord_val(ulo), ord_val(uhi));
    S.st()[2 * b + 1] = make_float4(ord_val(wlo), ord_val(whi), __int_as_float(ok), 0.0f);
  }
}

// pair_rank within a cell of at most 65535 SIPs
__device__ __forceinline__ uint32_t rank32(int i, int j, int n) {
  const uint32_t u = (uint32_t)i;
  return u * (uint32_t)n - ((u * (u + 1u)) >> 1) + (uint32_t)(j - i - 1);
}
// segment (i, b) moved forward by `adv` segments (row i holds the segments
// b = (i + 1) / 32 .. B - 1); past the cell's last segment b >= B
__device__ __forceinline__ void advance_seg(int n, int B, int& i, int& b, int adv) {
  b += adv;
  while (b > B - 1 && i < n - 2) {
    ++i;
    b += ((i + 1) >> 5) - B;
  }
}

// surely_skips' factor for an efficiency of at most em
__device__ __forceinline__ float skip_factor(const CellArgs& a, float em) {
  return ((a.dtdv_f * (float)(LC_PI * 1.0E-12)) * fmaxf(em, 0.0f)) * (1.0f + 0x1p-13f);
}
// warp_event out of line, for thin_cell's two kinds of events
template <bool BIG>
__device__ __noinline__ int event_call(Cell<BIG> S, int l0, int l1, double Tc, bool use_E, double r,
                                       bool certain) {
  return warp_event<true>(S, l0, l1, Tc, use_E, r, certain);
}

// The thinned draws of lacmo_thin.h for one cell, warp-cooperative.  A round
// takes 32 consecutive segments, one per lane (lane 0 the current part of the
// current segment): each lane bounds its segment from SIP i and the block
// statistics and, when the bound is below LACMO_THIN_TAU, draws the uniform
// that decides whether the segment holds a draw below q.  Segments with
// neither such a hit nor per-pair draws are done; the first one with either
// is then processed by the warp: per-pair draws screened in parallel, or the
// hit's first-hit draws evaluated by all lanes at once and the hit pair by
// one lane.  The statistics of the blocks it may have changed are refreshed,
// and the next round starts after it.
template <bool BIG>
__device__ __forceinline__ int2 thin_cell(Cell<BIG> S, int n, double Tc,
                                       bool use_E, uint64_t pc1, int lane) {
  const CellArgs& a = cell_args();
  static_assert(LACMO_THIN_L == 32, "one block of slots per warp");
  int c0 = 0, c1 = 0;   // this lane's outcome counts
  constexpr unsigned FULL = 0xffffffffu;
  const int B = (n + 31) >> 5;
  for (int b = 0; b < B; ++b) block_stats(S, n, b, lane);
  __syncwarp();
  int si = 0, sb = 0, sj = 1, ssub = 0;   // current segment, its part start and counter
  bool scratch = false;
  for (;;) {
    // Lane l takes the l-th segment from (si, sb) on.  Rows r with one (r + 1) / 32
    // = g hold B - g segments each, so beyond row si the row and block follow
    // from one quotient; 32 segments reach into no third such group (a sum over
    // the rows and a search in it took a chain of 12 shuffles: a step of the
    // 64-member ensemble 3.90 ms with it, 3.51 ms without).
    int i = si, b = sb + lane;
    bool valid = b < B;
    if (!valid) {
      int l = b - B, g = (si + 2) >> 5, cnt = B - g;
      int r = si + 1;
      const int rows = ((g + 1) << 5) - (r + 1);   // left of this group
      if (l >= rows * cnt) {
        l -= rows * cnt;
        r += rows;
        ++g;
        --cnt;
      }
      const int q = cnt > 0 ? __float2int_rz(((float)l + 0.5f) * f_rcp((float)cnt)) : 0;
      i = r + q;
      b = g + l - q * cnt;
      valid = cnt > 0 && i <= n - 2;
    }
    const int blo = b << 5;
    const int jfirst = blo > i + 1 ? blo : i + 1;
    const int j = lane ? jfirst : sj;
    const int jend = blo + 32 < n ? blo + 32 : n;
    const uint32_t sub = lane ? 0u : (uint32_t)ssub;
    bool indiv = false, hit = false;
    int e = 0;
    if (valid) {
      const float4 vi = S.v()[i];
      const float4 s0 = S.st()[2 * b], s1 = S.st()[2 * b + 1];
      const lt_block_t st{s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, __float_as_int(s1.z)};
      const float er = use_E ? __ldg(a.erow + S.sk()[i]) : a.E_const_f;
      const float Q = lt_segment_bound(vi.x, vi.y, vi.z, vi.w, &st, er, a.dtdv_f);
      indiv = !(Q >= 0.0f && Q < LACMO_THIN_TAU);
      if (!indiv) {
        e = lt_exponent(Q);
        const uint64_t u = lt_bits53(a.seed, (uint64_t)rank32(i, jfirst, n), sub, 0u, pc1);
        hit = u < __ldg(&LACMO_THIN_HT[e - LACMO_THIN_E_MIN][jend - j - 1]);
      }
    }
    const unsigned ev = __ballot_sync(FULL, valid && (indiv || hit));
    const bool all_valid = __ballot_sync(FULL, valid) == FULL;
    // the lane's segment, packed into three words for the event loop
    // (n <= 65535 so i, j < 2^16; B <= 2048; e < 128; sub <= 32)
    const uint32_t pk_ij = (uint32_t)i | ((uint32_t)j << 16);
    const uint32_t pk_fe = (uint32_t)jfirst | ((uint32_t)jend << 16);
    const uint32_t pk_b = ((uint32_t)b & 0x7ffu) | ((uint32_t)e << 11) | ((uint32_t)indiv << 18) |
                          (sub << 19);
    // the round's segments with an event, in order.  An event that changes
    // nothing (no collection) leaves the state, and so the bounds and hit
    // draws of the later lanes, as they were: the next event of the round is
    // processed at once.  A collection (or a hit whose segment has pairs
    // left, a new part with its own draw) ends the round; the next one
    // starts after it.
    unsigned pend = ev;
    bool restart = false, cell_done = false;
    while (pend) {
      const int L = __ffs(pend) - 1;
      pend &= pend - 1u;
      const uint32_t qij = __shfl_sync(FULL, pk_ij, L), qfe = __shfl_sync(FULL, pk_fe, L);
      const uint32_t qb = __shfl_sync(FULL, pk_b, L);
      const int ei = (int)(qij & 0xffffu), ej = (int)(qij >> 16);
      const int ejf = (int)(qfe & 0xffffu), eend = (int)(qfe >> 16);
      const int eb = (int)(qb & 0x7ffu), ee = (int)((qb >> 11) & 0x7fu);
      const bool eind = ((qb >> 18) & 1u) != 0;
      const uint32_t esub = qb >> 19;
      int next_j = eend;
      bool changed = false;
      if (eind) {
        // per-pair draws of the rest of the segment (pair ej + lane per
        // lane, drawn once), screened in parallel; the candidates are
        // processed in order, and the rest is screened again only after a
        // state change
        const int q = ej + lane;
        const bool mine = q < eend;
        uint64_t k53 = 0;
        float r_lo = 0.0f, r_hi = 0.0f;
        if (mine) {
          k53 = philox_bits53(a.seed, (uint64_t)rank32(ei, q, n), pc1);
          philox_interval(k53, r_lo, r_hi);
        }
        unsigned todo = __ballot_sync(FULL, mine);   // pairs not processed yet
        while (todo) {
          // SIP ei's row bounds the efficiency
          const float cmax = skip_factor(a, use_E ? __ldg(a.ecap + S.sk()[ei]) : a.E_const_f);
          int sc = 0;
          const float4 ve = S.v()[ei];
          const bool left = ((todo >> lane) & 1u) && !surely_skips(ve, S.v()[q], cmax, r_lo);
          if (!__any_sync(FULL, left)) break;
          if (left) sc = screen_pair(a, use_E, ve, S.sk()[ei], S.v()[q], S.sk()[q], r_lo, r_hi);
          unsigned cand = __ballot_sync(FULL, sc != 0);
          bool col_now = false;
          while (cand) {
            if (!scratch) { init_exact_scratch(a, S, n, lane); scratch = true; }
            const int t = __ffs(cand) - 1;
            const int o = event_call(S, ei, ej + t, Tc, use_E,
                                     philox_from_bits(__shfl_sync(FULL, k53, t)),
                                     __shfl_sync(FULL, sc, t) == 1);
            if (lane == t) {
              c0 += o == 1;
              c1 += o == 2;
            }
            todo &= ~((2u << t) - 1u);   // pairs up to t are done
            if (o) { col_now = true; break; }
            cand &= cand - 1u;   // no change: the later screens still hold
          }
          if (!col_now) break;
          changed = true;
        }
      } else {
        // the hit: first-hit draws of all lanes, then the pair with r = q u
        const int m = eend - ej;
        const uint64_t chunk = (uint64_t)rank32(ei, ejf, n);
        bool succ = false;
        if (lane < m - 1)
          succ = lt_bits53(a.seed, chunk, esub, (uint32_t)(1 + lane), pc1) <
                 __ldg(&LACMO_THIN_PT[ee - LACMO_THIN_E_MIN][m - lane - 1]);
        const unsigned bal = __ballot_sync(FULL, succ);
        const int g = bal ? __ffs(bal) - 1 : m - 1;
        const uint32_t jd = g < m - 1 ? (uint32_t)(g + 2) : (uint32_t)m;
        const double r = ldexp((double)lt_bits53(a.seed, chunk, esub, jd, pc1) *
                                   (1.0 / 9007199254740992.0), -ee);
        // a float interval around r: truncation and the next float up
        // (below the normal range: [0, 2^-126])
        const bool normal = r >= 0x1p-126;
        const float r_lo = normal ? d2f_down_pos(r) : 0.0f;
        const float r_hi = normal ? __uint_as_float(__float_as_uint(r_lo) + 1u) : 0x1p-126f;
        const int hj = ej + g;
        const int sc = screen_pair(a, use_E, S.v()[ei], S.sk()[ei], S.v()[hj], S.sk()[hj], r_lo, r_hi);
        if (sc != 0) {
          if (!scratch) { init_exact_scratch(a, S, n, lane); scratch = true; }
          const int o = event_call(S, ei, hj, Tc, use_E, r, sc == 1);
          if (lane == 0) {
            c0 += o == 1;
            c1 += o == 2;
          }
          changed = o != 0;
        }
        next_j = ej + g + 1;
      }
      const bool part_left = !eind && next_j < eend;
      if (!changed && !part_left) continue;   // the round goes on
      if (changed) {
        // the statistics of the blocks the event may have changed
        block_stats(S, n, ei >> 5, lane);
        if ((ei >> 5) != eb) block_stats(S, n, eb, lane);
        __syncwarp();
      }
      si = ei; sb = eb;
      if (part_left) {
        sj = next_j;
        ssub = (int)esub + 1;
      } else {
        advance_seg(n, B, si, sb, 1);
        if (sb >= B) { cell_done = true; break; }
        sj = (sb << 5) > si + 1 ? (sb << 5) : si + 1;
        ssub = 0;
      }
      restart = true;
      break;
    }
    if (cell_done) break;
    if (restart) continue;
    // every segment of the round is done
    if (!all_valid) break;   // the cell's last segment is done
    si = (int)(__shfl_sync(FULL, pk_ij, 31) & 0xffffu);
    sb = (int)(__shfl_sync(FULL, pk_b, 31) & 0x7ffu);
    advance_seg(n, B, si, sb, 1);
    if (sb >= B) break;
    sj = (sb << 5) > si + 1 ? (sb << 5) : si + 1;
    ssub = 0;
  }
  return make_int2((int)c0, (int)c1);
}

// One cell by one warp: the pairs are screened in parallel in lexicographic
// order and only the events of the sequential order (collections and undecided
// pairs) are processed one at a time.  Returns this lane's outcome counts.
template <bool THIN, bool BIG>
__device__ __forceinline__ int2 collide_cell(const Cell<BIG> S, int64_t c, int n, int lane) {
  const CellArgs& a = cell_args();
  const bool use_E = a.E != nullptr;
  const double Tc = a.T[c];
  const uint64_t pc1 = (a.cstep << 32) | (uint64_t)c;
  const int32_t* ids = a.perm + S.base;
  // FP32 copies, FP32 radius and bin (exact when near a bin edge).  Thinned draws
  // bound segments with the radius' bits; per-pair screens take it within 1e-6
  const float Tf = d2f_rn(Tc);
  const float rhow_f = (float)LC_PAR_WATER_DENS_0 +
                       (float)LC_PAR_WATER_DENS_1 * ((Tf - (float)LC_PAR_WATER_DENS_2) *
                                                      (Tf - (float)LC_PAR_WATER_DENS_2));
  // The next slot's data are fetched while this one is worked on: the gathers
  // by SIP ID waited for memory slot after slot (a step of the 64-member
  // ensemble, 51.9 million SIPs: 5.00 ms before, 4.31 ms with them in flight).
  int32_t id_n = lane < n ? ids[lane] : 0;
  double mw_n = 0.0, ms_n = 0.0, xi_n = 0.0, u_n = 0.0, w_n = 0.0;
  if (lane < n) {
    mw_n = a.m_w[id_n]; ms_n = a.m_s[id_n]; xi_n = a.xi[id_n];
    u_n = a.vel[id_n]; w_n = a.vel[a.n + id_n];
  }
  for (int q = lane; q < n; q += 32) {
    const int32_t id = id_n;
    const double mw_q = mw_n, ms_q = ms_n, xi_q = xi_n, u_q = u_n, w_q = w_n;
    if (q + 32 < n) {
      id_n = ids[q + 32];
      mw_n = a.m_w[id_n]; ms_n = a.m_s[id_n]; xi_n = a.xi[id_n];
      u_n = a.vel[id_n]; w_n = a.vel[a.n + id_n];
    }
    const float mwf = d2f_rn(mw_q), msf = d2f_rn(ms_q);
    const float mpf = mwf + msf;
    const float wsf = THIN ? msf / mpf : msf * f_rcp(mpf);
    const float rho = (a.sol == SOL_AS)
                          ? rhow_f * ((((float)LC_PAR_RHO_AS_0 * wsf + (float)LC_PAR_RHO_AS_1) *
                                           wsf + (float)LC_PAR_RHO_AS_2) * wsf +
                                      (float)LC_PAR_RHO_AS_3)
                          : (float)LC_PAR_SOL_DENS_NACL_0 + (float)LC_PAR_SOL_DENS_NACL_1 * wsf +
                                (float)LC_PAR_SOL_DENS_NACL_2 * Tf +
                                (float)LC_PAR_SOL_DENS_NACL_3 * wsf * wsf +
                                (float)LC_PAR_SOL_DENS_NACL_4 * wsf * Tf +
                                (float)LC_PAR_SOL_DENS_NACL_5 * Tf * Tf;
    const float V = (float)LC_FOUR_PI_OVER_THREE_INV * mpf;
    const float Rf = THIN ? lt_cbrtf(V / rho) : f_cbrt(V * f_rcp(rho));
    int32_t kb = 0;
    if (use_E) {
      const float v = (__logf(Rf) - a.lo_f) * a.inv_bl_f + 0.5f;
      const float fl = floorf(v);
      if (v - fl > a.bin_margin && (fl + 1.0f) - v > a.bin_margin && v > -1e6f && v < 1e6f &&
          Rf > 0.f) {
        kb = __float2int_rz(fl);
        kb = kb < 0 ? 0 : (kb > a.nb - 1 ? (int32_t)a.nb - 1 : kb);
      } else {
        kb = exact_bin_of(id, Tc);
      }
    }
    S.v()[q] = make_float4(d2f_rn(xi_q), Rf, d2f_rn(u_q), d2f_rn(w_q));
    S.sk()[q] = kb;
    S.sid()[q] = id;
  }
  __syncwarp();
  if constexpr (THIN) {
    return thin_cell(S, n, Tc, use_E, pc1, lane);
  } else {
    int c0 = 0, c1 = 0;
    const float cmax = a.cmax;
    const double* rnd = a.draws ? a.draws + a.draw_base + a.draw_off[c] : nullptr;
    const int P = (int)((int64_t)n * (n - 1) / 2);
    // Speculative sequential order, one window of 64 pairs (lexicographic
    // order) at a time: lane l draws the couple of ranks (w0 + 2l, w0 + 2l + 1),
    // one Philox block per couple, and screens both pairs with the current
    // state (surely_skips).  The few left go to window_events, which takes the
    // window's events in their order.  A cell with many events finishes with the
    // anti-diagonal schedule from its current position: the sequence costs a
    // chain of some 4 us per event, the 2n - 3 diagonals about as much each.
    const int event_limit = 64 + 2 * n;
    // Undecided pairs that change nothing (multiplicities below zero, NaN) take some
    // 2 us each where they fill a cell, the diagonals 10 us each: 250 SIPs, all of
    // them negative, 64.7 ms a step without this limit, 5.4 ms with it.
    const int idle_limit = min(16 + P / 64, 10 * n);
    PairEvents ev;
    ev.pos = 0;            // first rank not processed yet
    ev.events = ev.idle = 0;
    bool diagonal = false;
    int i = 0, j = 1 + 2 * lane;   // the pair of rank w0 + 2 lane
    float4 vi = S.v()[0];
    for (int w0 = 0; w0 < P; w0 += 64, j += 64) {
      if (j > n - 1) {
        while (j > n - 1 && i < n - 2) { j += i + 2 - n; ++i; }
        vi = S.v()[i];
      }
      const int p = w0 + 2 * lane;
      // the next pair in lexicographic order: the same row, or the next one's first
      const bool same = j < n - 1;
      const int i2 = same ? i : i + 1, j2 = same ? j + 1 : i + 2;
      PhiloxBlock x;   // the couple's draws (injected ones as their bits)
      float r0, r1;
      if (rnd) {
        x = injected_couple(rnd, p, P);
        r0 = low_of_double(__hiloint2double((int)x.x0, (int)x.x1));
        r1 = low_of_double(__hiloint2double((int)x.x2, (int)x.x3));
      } else {
        x = philox_block(a.seed, (uint64_t)(p >> 1), pc1);
        r0 = low_of_word(x.x0);
        r1 = low_of_word(x.x2);
      }
      bool m0 = false, m1 = false;
      if (p < P) m0 = !surely_skips(vi, S.v()[j], cmax, r0);
      if (p + 1 < P) m1 = !surely_skips(same ? vi : S.v()[i2], S.v()[j2], cmax, r1);
      if (!__any_sync(0xffffffffu, m0 | m1)) continue;
      ev.m = (m0 ? 1 : 0) | (m1 ? 2 : 0);
      const bool go_on = window_events(S, n, P, w0, i, j, x, cmax, Tc, use_E, rnd != nullptr,
                                       event_limit, idle_limit, ev);
      c0 += ev.c0;
      c1 += ev.c1;
      diagonal = !go_on;
      if (diagonal) break;
      vi = S.v()[i];   // SIP i may have changed
    }
    if (diagonal) {
      const int pos = ev.pos;
      // anti-diagonal schedule of the pairs from rank pos on
      for (int s = 1; s <= 2 * n - 3; ++s) {
        const int ilo = s - (n - 1) > 0 ? s - (n - 1) : 0;
        const int ihi = (s - 1) >> 1;
        for (int i = ilo + lane; i <= ihi; i += 32) {
          const int j = s - i;
          const uint32_t rk = rank32(i, j, n);
          if (rk < (uint32_t)pos) continue;
          uint64_t k53 = 0;
          float r_lo, r_hi;
          if (rnd) {
            injected_interval(rnd[rk], r_lo, r_hi);
          } else {
            k53 = philox_bits53(a.seed, (uint64_t)rk, pc1);
            philox_interval(k53, r_lo, r_hi);
          }
          const int sc = screen_pair(a, use_E, S.v()[i], S.sk()[i], S.v()[j], S.sk()[j], r_lo, r_hi);
          if (sc == 0) continue;
          if (sc == 1) {
            certain_collection(S, i, j, Tc, use_E);
            c0 += 1;
            continue;
          }
          const int o = exact_pair(S, S.sid()[i], S.sid()[j], i, j, Tc, use_E,
                                   rnd ? rnd[rk] : philox_from_bits(k53));
          c0 += o == 1;
          c1 += o == 2;
        }
        __threadfence_block();
        __syncwarp();
      }
    }
    return make_int2(c0, c1);
  }
}
// cells above the shared-memory size, out of line
template <bool THIN>
__device__ __noinline__ int2 collide_big(int64_t c, int32_t b, int n) {
  const CellArgs& a = cell_args();
  Cell<true> S;
  S.base = b;
  S.v_ = (float4*)a.gcopy + b;
  S.sk_ = (int32_t*)((float4*)a.gcopy + a.n) + b;
  S.sid_ = S.sk_ + a.n;
  S.st_ = a.gstats + 2 * ((int64_t)(b >> 5) + c);
  return collide_cell<THIN>(S, c, n, threadIdx.x & 31);
}

// THIN: the thinned draws, else per-pair draws.  MINB: resident blocks per
// SM the register budget is set for (the TUNE_COLLISION_BLOCKS knob picks the
// instance; 3 by default)
template <bool THIN, int MINB>
__global__ void __launch_bounds__(CELL_WARPS * 32, MINB)
    k_collide_cells(const __grid_constant__ CK x) {
  CellArgs& a = cell_args();
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (threadIdx.x == 0) {
    make_cellargs(a, x.m.get(), x.cc);
    a.draw_base = a.draws ? *a.cursor : 0;
    a.cstep = (uint64_t)*a.col_step;
  }
  __syncthreads();
  if (a.draws && a.draw_base + *a.total_pairs > a.n_draws) {
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(a.flags, LACMO_FLAG_DRAWS_SHORT);
    return;
  }
  if constexpr (!THIN) {   // surely_skips' factor
    if (wid == 0) {
      float em = a.E_const_f;
      if (a.E) {
        // the largest of the row bounds (infinity without them: every pair is screened)
        em = a.ecap ? 0.0f : __uint_as_float(0x7f800000u);
        if (a.ecap) {
          for (int64_t q = lane; q < a.nb; q += 32) em = fmaxf(em, __ldg(a.ecap + q));
          em = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(em)));
        }
      }
      if (lane == 0) a.cmax = skip_factor(a, em);
    }
    __syncthreads();
  }
  // persistent warps take the member's cells, largest first, from a counter
  for (;;) {
    int idx = 0;
    if (lane == 0) idx = atomicAdd(a.cell_ctr, 1);
    idx = __shfl_sync(0xffffffffu, idx, 0);
    if (idx >= a.C) break;
    const int64_t c = a.cell_order[idx];
    const int32_t b = a.start[c];
    const int n = a.start[c + 1] - b;
    if (n < 2) break;   // the remaining cells hold fewer than two SIPs
    if (n > 65535) {    // pair ranks would leave 32 bits
      if (lane == 0) atomicOr(a.flags, LACMO_FLAG_CELL_TOO_BIG);
      continue;
    }
    const int2 k = n > CELL_SMEM ? collide_big<THIN>(c, b, n)
                                 : collide_cell<THIN>(Cell<false>{wid, b}, c, n, lane);
    __syncwarp();
    // counters (integer sums commute)
    if (__any_sync(0xffffffffu, k.x | k.y)) {
      const unsigned k0 = __reduce_add_sync(0xffffffffu, (unsigned)k.x);
      const unsigned k1 = __reduce_add_sync(0xffffffffu, (unsigned)k.y);
      if (lane == 0) {
        atomicAdd((unsigned long long*)a.no_cols, (unsigned long long)k0);
        atomicAdd((unsigned long long*)(a.no_cols + 1), (unsigned long long)k1);
      }
    }
  }
}

__global__ void k_col_advance(const __grid_constant__ MRef mr, int draws) {
  const Ws& w = mr.get().w;
  if (draws && !(*w.flags & LACMO_FLAG_DRAWS_SHORT)) *w.cursor += *w.total_pairs;
  *w.col_step += 1;
  *w.cell_ctr = 0;
}

// ---------------------------------------------------------------------------
static inline int nblk(int64_t n, int t) {
  int64_t b = (n + t - 1) / t;
  if (b < 1) b = 1;
  return (int)(b < 152 * 32 ? b : 152 * 32);
}
static const size_t CELL_SMEM_BYTES = CELL_ARGS_BYTES + (size_t)CELL_WARPS * CELL_WARP_BYTES;

// The FP32 copy of the efficiency table and the largest FP32 efficiency of
// each row, one warp per row: the maximum of the row's positive values by a
// warp reduction; a row with a NaN, or whose largest value is not positive
// (where the sign of a zero or the place of a NaN decides), is taken in column
// order by one lane, as the oracle does.  ecap bounds the row from above whatever
// it holds: a row with a NaN gets infinity (in column order a NaN hides the values
// before it)
__global__ void k_table_float(const double* __restrict__ E, float* __restrict__ Ef,
                              float* __restrict__ erow, float* __restrict__ ecap, int64_t nb) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t k = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5); k < nb;
       k += warps) {
    const double* row = E + k * nb;
    uint32_t mk = 0;
    bool nan = false;
    for (int64_t q = lane; q < nb; q += 32) {
      const float v = (float)__ldg(row + q);
      Ef[k * nb + q] = v;
      nan |= v != v;
      if (v > 0.0f) mk = max(mk, __float_as_uint(v));   // positive floats order as integers
    }
    mk = __reduce_max_sync(0xffffffffu, mk);
    nan = __any_sync(0xffffffffu, nan);
    if (lane == 0) {
      if (nan || mk == 0) {
        float mx = (float)row[0];
        for (int64_t q = 1; q < nb; ++q) mx = lt_max(mx, (float)row[q]);
        erow[k] = mx;
        ecap[k] = nan ? __uint_as_float(0x7f800000u) : mx;
      } else {
        erow[k] = ecap[k] = __uint_as_float(mk);
      }
    }
  }
}

// persistent blocks: as many as are resident at once, split over members
template <bool THIN, int MINB>
static cudaError_t launch_cells(const Bt& B, const CK& x, cudaStream_t s) {
  static std::atomic<int> resident[64];
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  int res = dev < 64 ? resident[dev].load() : 0;
  if (res <= 0) {
    e = cudaFuncSetAttribute(k_collide_cells<THIN, MINB>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CELL_SMEM_BYTES);
    if (e != cudaSuccess) return e;
    int per_sm = 0, sms = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_collide_cells<THIN, MINB>,
                                                      CELL_WARPS * 32, CELL_SMEM_BYTES);
    if (e != cudaSuccess) return e;
    e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    res = per_sm * sms > 0 ? per_sm * sms : 1;
    if (dev < 64) resident[dev].store(res);
  }
  const int64_t C = B.nx * B.nz;
  int64_t bx = res / B.M;
  const int64_t need = (C + CELL_WARPS - 1) / CELL_WARPS;
  if (bx > need) bx = need;
  if (bx < 1) bx = 1;
  k_collide_cells<THIN, MINB><<<dim3((unsigned)bx, (unsigned)B.M), CELL_WARPS * 32,
                                CELL_SMEM_BYTES, s>>>(x);
  note_launches(1);
  return cudaGetLastError();
}

// the event log of single-state collision steps (lacmo_collision_event_log)
static std::atomic<EvRec*> g_log{nullptr};
static std::atomic<int64_t> g_log_cap{0};
static std::atomic<unsigned long long*> g_log_count{nullptr};

cudaError_t launch_collide_cells(const Bt& B, const lacmo_params_t& p, const lacmo_draws_t& d,
                                 cudaStream_t s) {
  if (B.M > 1 && d.draws) return cudaErrorInvalidValue;   // batches draw from Philox
  CellCommon cc;
  cc.log = B.M == 1 ? g_log.load() : nullptr;
  cc.log_cap = g_log_cap.load();
  cc.log_count = g_log_count.load();
  if (!cc.log_count) cc.log = nullptr;
  cc.dtdv = p.dt_col_over_dV; cc.E = p.E_col_grid; cc.E_const = p.E_col_const;
  cc.nb = p.no_kernel_bins; cc.lo = p.R_kernel_low_log; cc.bl = p.bin_factor_R_log;
  cc.sol = p.solute; cc.draws = d.draws; cc.n_draws = d.n_draws;
  cc.dtdv_f = (float)cc.dtdv; cc.lo_f = (float)cc.lo; cc.inv_bl_f = (float)(1.0 / cc.bl);
  cc.bin_margin = fp32_bin_margin(cc.lo, cc.bl, cc.nb);
  cc.E_const_f = (float)cc.E_const;
  cc.Ef = nullptr;
  cc.erow = cc.ecap = nullptr;
  float* Ef = B.one.w.Ef;   // member 0's slot serves the whole batch
  if (p.E_col_grid && Ef && p.no_kernel_bins <= LACMO_MAX_KERNEL_BINS) {
    float* erow = Ef + (int64_t)LACMO_MAX_KERNEL_BINS * LACMO_MAX_KERNEL_BINS;
    k_table_float<<<nblk(p.no_kernel_bins * 32, 128), 128, 0, s>>>(
        p.E_col_grid, Ef, erow, erow + LACMO_MAX_KERNEL_BINS, p.no_kernel_bins);
    note_launches(1);
    cc.Ef = Ef;
    cc.erow = erow;
    cc.ecap = erow + LACMO_MAX_KERNEL_BINS;
  }
  // thinned draws need the row maxima of a tabulated efficiency
  cc.thin = (p.thin_draws != 0 && d.draws == nullptr && (!p.E_col_grid || cc.erow)) ? 1 : 0;
  CK x{B.ref(), cc};
  cudaError_t e;
  const int minb = tune_value(TUNE_COLLISION_BLOCKS);
  if (cc.thin) {
    e = minb == 2 ? launch_cells<true, 2>(B, x, s)
                  : (minb == 4 ? launch_cells<true, 4>(B, x, s) : launch_cells<true, 3>(B, x, s));
  } else {
    e = minb == 2 ? launch_cells<false, 2>(B, x, s)
                  : (minb == 4 ? launch_cells<false, 4>(B, x, s)
                               : launch_cells<false, 3>(B, x, s));
  }
  if (e != cudaSuccess) return e;
  k_col_advance<<<dim3(1, B.M), 1, 0, s>>>(B.ref(), d.draws ? 1 : 0); note_launches(1);
  return cudaGetLastError();
}
}  // namespace lacmo

extern "C" int lacmo_collision_event_log(void* events, int64_t capacity,
                                         unsigned long long* count) {
  if (events && (capacity < 0 || !count)) return LACMO_ERR_ARG;
  lacmo::g_log_count.store(events ? count : nullptr);
  lacmo::g_log_cap.store(events ? capacity : 0);
  lacmo::g_log.store((lacmo::EvRec*)events);
  return LACMO_OK;
}
