// Box-model collision steps (one cell, up to thousands of SIPs), bit-exact
// with the reference's loop over the pairs (i, j), i < j, in lexicographic
// order (collision/all_or_nothing.py:109-185, 269-390, 392-491).
//
// A step evaluates n(n-1)/2 pairs (12.5 million for 5000 SIPs) and collects a
// few tens of them, so the work is the uniform draw of every pair and a screen
// against it, and the order only matters among the few pairs left.  A step is
//   1. k_box_prep (tabulated kernels): kernel bins and FP32 copies of the SIPs,
//      the largest value of each table row;
//   2. k_box_screen, the whole GPU: every pair's draw against a certified FP32
//      upper bound of its p_crit from the step-start state; pairs not ruled out
//      become candidates (their key i << 16 | j orders them as the reference
//      does);
//   3. k_box_step, one CTA: takes the candidates in order and evaluates each
//      exactly (FP64, the reference's operation order) with the state at its
//      turn.  After a collection the SIPs whose p_crit may have grown are
//      screened again against all their later pairs, and what the screen does
//      not rule out joins the candidates: at any time every pair to come that
//      would collect is among them.  A collected SIP that only lost
//      multiplicity, and is not left below zero, is not screened: max(xi) falls and
//      nothing else changed.
// Bounds: the screen is limited by the Philox blocks (about 65 of some 100
// instructions per couple of pairs); the event loop by its latency (3.6 us per
// collection of 5000 SIPs: one exact evaluation, up to n screened pairs).
// Measured on GB300, ms per step, before (one CTA, FP64 on every pair, diagonal
// by diagonal) and now: Golovin, 4968 SIPs, 22 / 646 / 3850 / 136,937
// collections 34.7 -> 0.24, 34.9 -> 2.3, 35.5 -> 18.3, 44.5 -> 31.8; 500 SIPs
// 0.77 -> 0.05; Hall efficiencies, 2980 SIPs, 7 collections 20.0 -> 0.14.
// Up to BOX_SELF pairs the one CTA screens them itself, two launches less: 100
// SIPs take 56 us a step with Hall efficiencies; at 362 SIPs it took 101 us
// against 47 us with the screen on the whole GPU.
// Many candidates (more than n) mean that the event chain would be longer than
// the anti-diagonal schedule, which then runs the step (18 ms for 4968 SIPs, the
// chain's 3.6 us n the same): pairs that share no SIP
// commute exactly, every pair that shares a SIP with (i, j) and comes earlier
// has a smaller index sum i + j and every later one a larger, so the diagonals
// s = i + j = 1 .. 2n - 3 in order, the pairs of one diagonal in parallel,
// give the sequential result: 2n - 3 barrier steps.
#include <cuda_runtime.h>

#include <atomic>

#include "lacmo_colmath.cuh"

namespace lacmo {
namespace {

enum { BOX_GOLOVIN, BOX_KGRID, BOX_ECOL };
constexpr int BOX_THREADS = 1024;
constexpr int BOX_CAND = 4096;       // candidates k_box_step holds in shared memory
constexpr int BOX_SELF = 8192;       // pairs one CTA screens itself
constexpr int SCREEN_THREADS = 512;
constexpr uint32_t NO_KEY = 0xffffffffu;

// what a step needs; scratch (count .. erow) is null when k_box_step works
// alone
struct BoxArgs {
  double *X, *M, *R;
  const double *V, *Rho;
  const double* K;     // kernel table K(m1, m2) or efficiency table E(R1, R2), [nb][nb]
  int n;
  int64_t nb;
  double lo, bl, dtdv;
  int64_t* no_cols;
  const double* rnd;
  uint64_t seed, step;
  float dtdv_f;
  int screened;        // candidates come from k_box_screen
  int limit;           // more candidates than this: the anti-diagonal schedule
  uint32_t* count;
  uint32_t* cand;      // [BOX_CAND]
  float4* f;           // [n] FP32 copies: (xi, row bound) or (xi, R, v, row bound)
  int32_t* bin;        // [n]
  float* erow;         // [nb]
};

__device__ __forceinline__ uint32_t key_of(int i, int j) { return ((uint32_t)i << 16) | (uint32_t)j; }
__device__ __forceinline__ float absmax(float a, float b) { return fmaxf(fabsf(a), fabsf(b)); }

// the draw of pair rank k and the lower bound the screens compare with
struct Draw {
  uint32_t hi, lo;
};
__device__ __forceinline__ Draw pair_draw(const BoxArgs& a, int64_t k) {
  if (a.rnd) {
    const uint64_t q = (uint64_t)__double_as_longlong(a.rnd[k]);
    return Draw{(uint32_t)(q >> 32), (uint32_t)q};
  }
  const PhiloxBlock b = philox_block(a.seed, (uint64_t)(k >> 1), a.step);
  return (k & 1) ? Draw{b.x2, b.x3} : Draw{b.x0, b.x1};
}
__device__ __forceinline__ float draw_low(const BoxArgs& a, Draw d) {
  return a.rnd ? low_of_double(__hiloint2double((int)d.hi, (int)d.lo)) : low_of_word(d.hi);
}
__device__ __forceinline__ double draw_value(const BoxArgs& a, Draw d) {
  if (a.rnd) return __hiloint2double((int)d.hi, (int)d.lo);
  return (double)((uint64_t)(d.hi >> 5) * 67108864ull + (uint64_t)(d.lo >> 6)) *
         (1.0 / 9007199254740992.0);
}

// Certified upper bound of |p_crit| from FP32 copies (each within 2^-24 of its
// value, or infinite beyond the FP32 range) and kf, an upper bound of the
// table's value (1 for Golovin): at most ten roundings of 2^-24 against the
// factor's 2^-14, magnitudes throughout so that no cancellation enters, an
// absolute slack for the velocity difference, and 1e-30 for products flushed to
// zero.  A draw's lower bound is 0 or at least 2^-24: a smaller p_crit than
// that never collects unless the bound keeps the pair.  NaN compares false:
// the pair stays a candidate.
template <int KIND>
__device__ __forceinline__ float p_bound(const BoxArgs& a, float4 fi, float4 fj, float kf) {
  float p;
  if (KIND == BOX_GOLOVIN) {
    p = ((absmax(fi.x, fj.x) * (fabsf(fi.y) + fabsf(fj.y))) * 1.5E-18f) * a.dtdv_f;
  } else if (KIND == BOX_KGRID) {
    p = (absmax(fi.x, fj.x) * fabsf(kf)) * a.dtdv_f;
  } else {
    const float rs = fabsf(fi.y) + fabsf(fj.y);
    const float dv = fabsf(fi.z - fj.z) + 0x1p-21f * (fabsf(fi.z) + fabsf(fj.z));
    p = ((absmax(fi.x, fj.x) * a.dtdv_f) * (float)(LC_PI * 1.0E-12)) * (rs * rs) *
        (fabsf(kf) * dv);
  }
  return p * (1.0f + 0x1p-14f) + 1e-30f;
}

__global__ void k_box_prep(const BoxArgs a, int kind) {
  if (blockIdx.x == 0 && threadIdx.x == 0) *a.count = 0;
  const int lane = threadIdx.x & 31;
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t T = (int64_t)gridDim.x * blockDim.x;
  for (int64_t q = t; q < a.n; q += T) {
    const double m = kind == BOX_KGRID ? a.M[q] : a.R[q];
    a.bin[q] = col_bin(m, a.lo, a.bl, a.nb);
    float4 f = make_float4(d2f_flush(a.X[q]), 0.0f, 0.0f, 0.0f);
    if (kind == BOX_ECOL) { f.y = d2f_flush(m); f.z = d2f_flush(a.V[q]); }
    a.f[q] = f;
  }
  for (int64_t r = t >> 5; r < a.nb; r += T >> 5) {   // |largest| value of each row
    float mx = 0.0f;
    for (int64_t q = lane; q < a.nb; q += 32) mx = fmaxf(mx, fabsf(d2f_flush(a.K[r * a.nb + q])));
    mx = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(mx)));
    if (lane == 0) a.erow[r] = mx;
  }
}

__device__ __forceinline__ void add_candidate(const BoxArgs& a, int i, int j) {
  const uint32_t s = atomicAdd(a.count, 1u);
  if (s < (uint32_t)BOX_CAND) a.cand[s] = key_of(i, j);
}

// Every warp walks a run of windows of 64 ranks (one couple per lane, one
// Philox block per couple); the SIPs' FP32 copies lie in shared memory.
template <int KIND>
__global__ void __launch_bounds__(SCREEN_THREADS, 2) k_box_screen(const BoxArgs a) {
  extern __shared__ float4 sm4[];
  float2* s2 = (float2*)sm4;                                   // Golovin, kgrid
  int32_t* sb = KIND == BOX_KGRID ? (int32_t*)(s2 + a.n) : (int32_t*)(sm4 + a.n);
  const int n = a.n;
  for (int q = threadIdx.x; q < n; q += SCREEN_THREADS) {
    if (KIND == BOX_GOLOVIN) {
      s2[q] = make_float2(d2f_flush(a.X[q]), d2f_flush(a.M[q]));
    } else {
      float4 f = a.f[q];
      const int32_t b = a.bin[q];
      const float e = a.erow[b];
      sb[q] = b;
      if (KIND == BOX_KGRID) s2[q] = make_float2(f.x, e);
      else { f.w = e; sm4[q] = f; }
    }
  }
  __syncthreads();
  auto get = [&](int q) {
    if (KIND == BOX_ECOL) return sm4[q];
    const float2 v = s2[q];
    return make_float4(v.x, v.y, 0.0f, KIND == BOX_KGRID ? v.y : 1.0f);
  };
  const int lane = threadIdx.x & 31;
  const int W = (int)(gridDim.x * (SCREEN_THREADS / 32));
  const int w = (int)(blockIdx.x * (SCREEN_THREADS / 32) + (threadIdx.x >> 5));
  const int64_t P = (int64_t)n * (n - 1) / 2;
  const int64_t windows = (P + 63) / 64, per = (windows + W - 1) / W;
  const int64_t k_end = min((w + 1) * per * 64, P);
  int64_t k = w * per * 64 + 2 * lane;
  if (k >= k_end) return;
  // the pair of rank k: the row i with i (2n - i - 1) / 2 <= k
  const double b = 2.0 * n - 1.0;
  int i = (int)((b - sqrt(fmax(b * b - 8.0 * (double)k, 0.0))) * 0.5);
  i = i < 0 ? 0 : (i > n - 2 ? n - 2 : i);
  while (i > 0 && (int64_t)i * (2 * n - i - 1) / 2 > k) --i;
  while (i < n - 2 && (int64_t)(i + 1) * (2 * n - i - 2) / 2 <= k) ++i;
  int j = (int)(k - (int64_t)i * (2 * n - i - 1) / 2) + i + 1;
  float4 fi = get(i);
  for (; k < k_end; k += 64, j += 64) {
    if (j > n - 1) {
      while (j > n - 1 && i < n - 2) { j += i + 2 - n; ++i; }
      fi = get(i);
    }
    Draw d0, d1 = {0, 0};
    const bool has1 = k + 1 < P;   // the couple's second pair: this row's next, or a new row
    if (a.rnd) {
      d0 = pair_draw(a, k);
      if (has1) d1 = pair_draw(a, k + 1);
    } else {
      const PhiloxBlock x = philox_block(a.seed, (uint64_t)(k >> 1), a.step);
      d0 = Draw{x.x0, x.x1};
      d1 = Draw{x.x2, x.x3};
    }
    const bool same = j < n - 1;
    const int i2 = same ? i : i + 1, j2 = same ? j + 1 : i + 2;
    const float4 fj = get(j);
    const bool m0 = !(p_bound<KIND>(a, fi, fj, fi.w) < draw_low(a, d0));
    bool m1 = false;
    if (has1) {
      const float4 g = same ? fi : get(i2);
      m1 = !(p_bound<KIND>(a, g, get(j2), g.w) < draw_low(a, d1));
    }
    if (m0 | m1) {
      // the few left: with the pair's own table value
      auto own = [&](int p, int q) {
        return KIND == BOX_GOLOVIN ? 1.0f : d2f_flush(__ldg(a.K + (int64_t)sb[p] * a.nb + sb[q]));
      };
      if (m0 && !(p_bound<KIND>(a, fi, fj, own(i, j)) < draw_low(a, d0))) add_candidate(a, i, j);
      if (m1 && !(p_bound<KIND>(a, get(i2), get(j2), own(i2, j2)) < draw_low(a, d1)))
        add_candidate(a, i2, j2);
    }
  }
}

// the step's state in shared memory
template <int KIND>
struct BoxSm {
  double *X, *M, *R, *V, *Rh;
  int32_t* B;
  __device__ __forceinline__ BoxSm(double* sm, int n) {
    X = sm; M = sm + n; R = V = Rh = nullptr; B = nullptr;
    if (KIND == BOX_KGRID) B = (int32_t*)(sm + 2 * n);
    if (KIND == BOX_ECOL) { R = sm + 2 * n; V = sm + 3 * n; Rh = sm + 4 * n; B = (int32_t*)(sm + 5 * n); }
  }
  __device__ __forceinline__ float4 f(int q) const {
    float4 r = make_float4(d2f_flush(X[q]), 0.0f, 0.0f, 0.0f);
    if (KIND == BOX_GOLOVIN) r.y = d2f_flush(M[q]);
    if (KIND == BOX_ECOL) { r.y = d2f_flush(R[q]); r.z = d2f_flush(V[q]); }
    return r;
  }
  // pair (i, j), i < j, may collect with its draw (a certified screen)
  __device__ __forceinline__ bool may_collect(const BoxArgs& a, int i, int j, Draw d) const {
    const float r = draw_low(a, d);
    const float4 fi = f(i), fj = f(j);
    if (KIND != BOX_GOLOVIN) {
      if (a.erow && p_bound<KIND>(a, fi, fj, a.erow[B[i]]) < r) return false;
      return !(p_bound<KIND>(a, fi, fj, d2f_flush(__ldg(a.K + (int64_t)B[i] * a.nb + B[j]))) < r);
    }
    return !(p_bound<KIND>(a, fi, fj, 1.0f) < r);
  }
  // the pair (i, j) evaluated exactly: 0 none, 1 collection, 2 multiple
  // collection; imin is the SIP that gained mass, split whether both changed
  __device__ __forceinline__ int pair(const BoxArgs& a, int i, int j, double r, int* imin_out,
                                      bool* split) const {
    int imin, imax;
    if (X[i] <= X[j]) { imin = i; imax = j; } else { imin = j; imax = i; }
    *imin_out = imin;
    *split = false;
    const double xi_min = X[imin], xi_max = X[imax];
    const double m_min = M[imin], m_max = M[imax];
    double p_crit;
    if (KIND == BOX_GOLOVIN) {
      p_crit = xi_max * ((m_min + m_max) * 1.5E-18) * a.dtdv;
    } else if (KIND == BOX_KGRID) {
      p_crit = xi_max * __ldg(a.K + (int64_t)B[i] * a.nb + B[j]) * a.dtdv;
    } else {
      const double Rs = R[i] + R[j];
      p_crit = xi_max * a.dtdv *
               (LC_PI * Rs * Rs * __ldg(a.K + (int64_t)B[i] * a.nb + B[j]) * fabs(V[i] - V[j]) *
                1.0E-12);
    }
    if (p_crit > 1.0) {
      const double xi_col = p_crit * xi_min;
      M[imin] = (xi_min * m_min + xi_col * m_max) / xi_min;
      X[imax] -= xi_col;
      update(a, imin);
      return 2;
    }
    if (!(p_crit > r)) return 0;
    const double xi_rel_dev = (xi_max - xi_min) / xi_max;
    if (xi_rel_dev < 1.0E-5) {
      const double xi_ges = xi_min + xi_max;
      M[imin] = 2.0 * (xi_min * m_min + xi_max * m_max) / xi_ges;
      M[imax] = M[imin];
      X[imax] = 0.5 * 0.7 * xi_ges;
      X[imin] = 0.5 * xi_ges - X[imax];
      update(a, imin);
      if (KIND == BOX_ECOL) R[imax] = R[imin];
      if (KIND != BOX_GOLOVIN) B[imax] = B[imin];
      *split = true;
    } else {
      M[imin] += m_max;
      X[imax] -= xi_min;
      update(a, imin);
    }
    return 1;
  }
  // radius and bin after a mass change
  __device__ __forceinline__ void update(const BoxArgs& a, int q) const {
    if (KIND == BOX_KGRID) B[q] = col_bin(M[q], a.lo, a.bl, a.nb);
    if (KIND == BOX_ECOL) {
      R[q] = col_radius(M[q], Rh[q]);
      B[q] = col_bin(R[q], a.lo, a.bl, a.nb);
    }
  }
};

template <int KIND>
__global__ void __launch_bounds__(BOX_THREADS) k_box_step(const BoxArgs a) {
  extern __shared__ double sm[];
  const int n = a.n;
  const BoxSm<KIND> S(sm, n);
  uint32_t* const cand = (uint32_t*)(sm + (KIND == BOX_ECOL ? 5 * n : 2 * n)) +
                         (KIND == BOX_GOLOVIN ? 0 : n);
  __shared__ uint32_t s_min[BOX_THREADS / 32];
  __shared__ uint32_t s_cnt;
  __shared__ int s_chg[2];
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
  const uint32_t found = a.screened ? *a.count : 0;
  if (t == 0) s_cnt = found;
  for (int q = t; q < n; q += BOX_THREADS) {
    S.X[q] = a.X[q]; S.M[q] = a.M[q];
    if (KIND == BOX_ECOL) { S.R[q] = a.R[q]; S.V[q] = a.V[q]; S.Rh[q] = a.Rho[q]; }
    if (KIND != BOX_GOLOVIN)
      S.B[q] = a.screened ? a.bin[q]
                          : col_bin(KIND == BOX_KGRID ? S.M[q] : S.R[q], a.lo, a.bl, a.nb);
  }
  __syncthreads();
  const int64_t P = (int64_t)n * (n - 1) / 2;
  if (a.screened) {
    for (int q = t; q < (int)min(found, (uint32_t)BOX_CAND); q += BOX_THREADS) cand[q] = a.cand[q];
  } else if (P <= BOX_SELF) {
    for (int r = t; r < (int)P; r += BOX_THREADS) {
      const float b = 2.0f * n - 1.0f;
      int i = (int)((b - sqrtf(fmaxf(b * b - 8.0f * (float)r, 0.0f))) * 0.5f);
      i = i < 0 ? 0 : (i > n - 2 ? n - 2 : i);
      while (i > 0 && i * (2 * n - i - 1) / 2 > r) --i;
      while (i < n - 2 && (i + 1) * (2 * n - i - 2) / 2 <= r) ++i;
      const int j = r - i * (2 * n - i - 1) / 2 + i + 1;
      if (S.may_collect(a, i, j, pair_draw(a, r))) {
        const uint32_t s = atomicAdd(&s_cnt, 1u);
        if (s < (uint32_t)BOX_CAND) cand[s] = key_of(i, j);
      }
    }
  }
  __syncthreads();
  // keys below `next` are done
  uint32_t next = 0;
  bool diagonal = !a.screened && P > BOX_SELF;
  int64_t c0 = 0, c1 = 0;
  int events = 0;
  uint32_t cnt = s_cnt;
  if (cnt > (uint32_t)min(a.limit, BOX_CAND)) diagonal = true;
  const int event_limit = 2 * (int)min(cnt, (uint32_t)BOX_CAND) + 64;
  while (!diagonal) {
    // the next candidate in order
    uint32_t best = NO_KEY;
    for (uint32_t q = t; q < cnt; q += BOX_THREADS) {
      const uint32_t k = cand[q];
      if (k >= next) best = min(best, k);
    }
    best = __reduce_min_sync(0xffffffffu, best);
    if (lane == 0) s_min[wid] = best;
    __syncthreads();
    best = __reduce_min_sync(0xffffffffu, s_min[lane]);
    if (best == NO_KEY) break;
    const int i = (int)(best >> 16), j = (int)(best & 0xffffu);
    next = best + 1;
    if (t == 0) {
      int imin;
      bool split;
      const double xi_i = S.X[i], xi_j = S.X[j];
      const int o = S.pair(a, i, j, draw_value(a, pair_draw(a, pair_rank(i, j, n))), &imin, &split);
      c0 += o == 1;
      c1 += o == 2;
      // the SIPs whose p_crit may have grown: the one that gained mass, and the
      // other one unless it only lost multiplicity and still has some (it gains from
      // a SIP whose multiplicity is negative)
      const int imax = imin == i ? j : i;
      const bool less = S.X[imax] >= 0.0 && S.X[imax] <= (imin == i ? xi_j : xi_i);
      s_chg[0] = o ? imin : -1;
      s_chg[1] = o && (split || !less) ? imax : -1;
    }
    __syncthreads();
    if (s_chg[0] < 0) continue;
    for (int c = 0; c < 2; ++c) {
      const int s = s_chg[c];
      if (s < 0) continue;
      // later pairs of s: (q, s) in rows q >= i below s, (s, q) in its own row
      for (int q = i + t; q < n; q += BOX_THREADS) {
        if (q == s) continue;
        const int p0 = q < s ? q : s, p1 = q < s ? s : q;
        if (key_of(p0, p1) < next) continue;
        if (S.may_collect(a, p0, p1, pair_draw(a, pair_rank(p0, p1, n)))) {
          const uint32_t at = atomicAdd(&s_cnt, 1u);
          if (at < (uint32_t)BOX_CAND) cand[at] = key_of(p0, p1);
        }
      }
    }
    __syncthreads();
    cnt = s_cnt;
    if (cnt > (uint32_t)BOX_CAND || ++events > event_limit) diagonal = true;
    __syncthreads();
  }
  if (diagonal) {
    // every pair with a key from `next` on, diagonal by diagonal
    for (int s = 1; s <= 2 * n - 3; ++s) {
      const int ilo = s - (n - 1) > 0 ? s - (n - 1) : 0;
      const int ihi = (s - 1) >> 1;
      for (int i = ilo + t; i <= ihi; i += BOX_THREADS) {
        const int j = s - i;
        if (key_of(i, j) < next) continue;
        const Draw d = pair_draw(a, pair_rank(i, j, n));
        if (!S.may_collect(a, i, j, d)) continue;
        int imin;
        bool split;
        const int o = S.pair(a, i, j, draw_value(a, d), &imin, &split);
        c0 += o == 1;
        c1 += o == 2;
      }
      __syncthreads();
    }
  }
  __syncthreads();
  for (int q = t; q < n; q += BOX_THREADS) {
    a.X[q] = S.X[q]; a.M[q] = S.M[q];
    if (KIND == BOX_ECOL) a.R[q] = S.R[q];
  }
  for (int off = 16; off > 0; off >>= 1) {
    c0 += __shfl_down_sync(0xffffffffu, c0, off);
    c1 += __shfl_down_sync(0xffffffffu, c1, off);
  }
  if (lane == 0 && (c0 | c1)) {
    atomicAdd((unsigned long long*)a.no_cols, (unsigned long long)c0);
    atomicAdd((unsigned long long*)(a.no_cols + 1), (unsigned long long)c1);
  }
}

template <int KIND>
cudaError_t launch_box(BoxArgs a, cudaStream_t s) {
  constexpr size_t step_sip = KIND == BOX_GOLOVIN ? 16 : (KIND == BOX_KGRID ? 20 : 44);
  constexpr size_t scr_sip = KIND == BOX_GOLOVIN ? 8 : (KIND == BOX_KGRID ? 12 : 20);
  constexpr int most = KIND == BOX_ECOL ? LACMO_ECOL_BOX_MAX_SIPS : LACMO_BOX_MAX_SIPS;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  static std::atomic<int> sms_of[64];   // SMs, once the kernels' attributes are set
  int sms = dev < 64 ? sms_of[dev].load() : 0;
  if (sms <= 0) {
    e = cudaFuncSetAttribute(k_box_step<KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)(most * step_sip + 4 * BOX_CAND));
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(k_box_screen<KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)(most * scr_sip));
    if (e != cudaSuccess) return e;
    e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    if (dev < 64) sms_of[dev].store(sms);
  }
  const int64_t P = (int64_t)a.n * (a.n - 1) / 2;
  a.limit = a.n;
  a.screened = 0;
  a.count = nullptr; a.cand = nullptr; a.f = nullptr; a.bin = nullptr; a.erow = nullptr;
  a.dtdv_f = (float)a.dtdv;
  Scratch mem(s);
  if (P > BOX_SELF) {
    const size_t rows = KIND == BOX_GOLOVIN ? 0 : (size_t)a.nb;
    const size_t per = KIND == BOX_GOLOVIN ? 0 : 20;
    const size_t bytes = 256 + 4 * BOX_CAND + per * (size_t)a.n + 4 * rows;
    char* const scratch = (char*)mem.get(bytes);
    if (scratch) {   // without, the one CTA runs the diagonals
      a.count = (uint32_t*)scratch;
      a.cand = (uint32_t*)(scratch + 256);
      if (KIND != BOX_GOLOVIN) {
        a.f = (float4*)(scratch + 256 + 4 * BOX_CAND);
        a.bin = (int32_t*)(a.f + a.n);
        a.erow = (float*)(a.bin + a.n);
      }
      a.screened = 1;
    }
  }
  if (a.screened) {
    if (KIND == BOX_GOLOVIN) {
      e = cudaMemsetAsync(a.count, 0, 4, s);
    } else {
      const int64_t work = a.n > 32 * a.nb ? a.n : 32 * a.nb;
      const int64_t blocks = (work + 127) / 128;
      k_box_prep<<<(unsigned)(blocks < 8 * sms ? blocks : 8 * sms), 128, 0, s>>>(a, KIND);
      note_launches(1);
      e = cudaGetLastError();
    }
    if (e == cudaSuccess) {
      // two blocks an SM, a warp at least four windows
      const int64_t want = (P + 64 * 4 * (SCREEN_THREADS / 32) - 1) / (64 * 4 * (SCREEN_THREADS / 32));
      k_box_screen<KIND><<<(unsigned)(want < 2 * sms ? want : 2 * sms), SCREEN_THREADS,
                           scr_sip * (size_t)a.n, s>>>(a);
      note_launches(1);
      e = cudaGetLastError();
    }
  }
  if (e == cudaSuccess) {
    k_box_step<KIND><<<1, BOX_THREADS, step_sip * (size_t)a.n + 4 * BOX_CAND, s>>>(a);
    note_launches(1);
    e = cudaGetLastError();
  }
  return e;
}

BoxArgs box_args(double* xis, double* m, int64_t n, double dtdv, int64_t* no_cols,
                 const double* rnd, uint64_t seed, uint64_t step) {
  BoxArgs a = {};
  a.X = xis; a.M = m; a.n = (int)n; a.dtdv = dtdv; a.no_cols = no_cols;
  a.rnd = rnd; a.seed = seed; a.step = step;
  a.nb = 0; a.lo = 0.0; a.bl = 1.0;
  return a;
}

}  // namespace

cudaError_t launch_golovin(double* xis, double* m, int64_t n, double dtdv, int64_t* no_cols,
                           const double* rnd, uint64_t seed, uint64_t step, cudaStream_t s) {
  return launch_box<BOX_GOLOVIN>(box_args(xis, m, n, dtdv, no_cols, rnd, seed, step), s);
}
cudaError_t launch_kgrid_box(double* xis, double* m, int64_t n, double dtdv, const double* K,
                             int64_t nb, double lo, double bl, int64_t* no_cols, const double* rnd,
                             uint64_t seed, uint64_t step, cudaStream_t s) {
  BoxArgs a = box_args(xis, m, n, dtdv, no_cols, rnd, seed, step);
  a.K = K; a.nb = nb; a.lo = lo; a.bl = bl;
  return launch_box<BOX_KGRID>(a, s);
}
cudaError_t launch_ecol_box(double* xis, double* m, double* R, const double* vel,
                            const double* rho, int64_t n, double dtdv, const double* E, int64_t nb,
                            double lo, double bl, int64_t* no_cols, const double* rnd,
                            uint64_t seed, uint64_t step, cudaStream_t s) {
  BoxArgs a = box_args(xis, m, n, dtdv, no_cols, rnd, seed, step);
  a.R = R; a.V = vel; a.Rho = rho; a.K = E; a.nb = nb; a.lo = lo; a.bl = bl;
  return launch_box<BOX_ECOL>(a, s);
}

namespace {
// collision/kernel.py:107-167 Beard (1976) terminal velocity (R in um)
__device__ double beard_velocity(double R) {
  const double rho_w = 1.0E3, rho_a = 1.225, visc = 1.818E-5, sigma = 73.0E-3;
  const double g = 9.80665, drho = rho_w - rho_a;
  if (R < 10.0) {
    const double l0 = 6.62E-2;
    const double C1 = drho * g / (4.5 * visc);
    const double C_sc = 1.0 + 1.257 * l0 / R;
    return C1 * C_sc * R * R * 1.0E-12;
  } else if (R < 535.0) {
    const double N_Da = 32.0E-18 * R * R * R * rho_a * drho * g / (3.0 * visc * visc);
    double Y = log(N_Da);
    const double p1[7] = {-0.327815e-5, 0.855176e-4, -0.578878e-3, -0.987059e-3,
                          -0.153193e-2, 0.992696, -0.318657e1};
    double r = p1[0] * Y + p1[1];
    for (int k = 2; k < 7; ++k) r = r * Y + p1[k];
    const double l0 = 6.62E-2;
    const double C_sc = 1.0 + 1.257 * l0 / R;
    return visc * C_sc * exp(r) / (rho_a * R * 2.0E-6);
  } else if (R < 3500.0) {
    const double N_Bo = 16.0E-12 * R * R * drho * g / (3.0 * sigma);
    const double v4 = (visc * visc) * (visc * visc);
    const double N_P16 = pow(sigma * sigma * sigma * rho_a * rho_a / (v4 * drho * g), 1.0 / 6.0);
    const double Y = log(N_Bo * N_P16);
    const double p2[6] = {0.238449e-2, -0.542819e-1, 0.475294, -0.204914e1, 0.523778e1,
                          -0.500015e1};
    double r = p2[0] * Y + p2[1];
    for (int k = 2; k < 6; ++k) r = r * Y + p2[k];
    return visc * N_P16 * exp(r) / (rho_a * R * 2.0E-6);
  }
  return 9.04929248;
}
__global__ void k_beard(double* vel, const double* R, int64_t n) {
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n;
       k += (int64_t)gridDim.x * blockDim.x)
    vel[k] = beard_velocity(R[k]);
}
__global__ void k_radius_bin(const double* m, const double* rho, int64_t n, double lo, double bl,
                             int64_t nb, double* R, int64_t* k) {
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n;
       q += (int64_t)gridDim.x * blockDim.x) {
    const double r = col_radius(m[q], rho[q]);
    R[q] = r;
    if (k) k[q] = col_bin(r, lo, bl, nb);
  }
}

inline int nblk(int64_t n, int t) {
  const int64_t b = (n + t - 1) / t;
  return (int)(b < 1 ? 1 : (b < 152 * 32 ? b : 152 * 32));
}
}  // namespace

cudaError_t launch_beard(double* vel, const double* R, int64_t n, cudaStream_t s) {
  k_beard<<<nblk(n, 128), 128, 0, s>>>(vel, R, n); note_launches(1);
  return cudaGetLastError();
}
cudaError_t launch_radius_bin(const double* m, const double* rho, int64_t n, double lo, double bl,
                              int64_t nb, double* R, int64_t* k, cudaStream_t s) {
  k_radius_bin<<<nblk(n, 128), 128, 0, s>>>(m, rho, n, lo, bl, nb, R, k); note_launches(1);
  return cudaGetLastError();
}

}  // namespace lacmo
