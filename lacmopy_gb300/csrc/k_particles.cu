// Particle, grid and cell-binning kernels of the SIP hot path (FP64).
//
// k_particles fuses one whole particle sub-step of the reference
// (integration.py:944-1091): T_p from the cell, radius / mass fraction /
// density, the implicit Newton condensation (integration.py:728-940), the
// implicit drag update with the staggered bilinear wind interpolation
// (integration.py:632-719, grid.py:257-323), the Euler position update with
// periodic x, capped z and ground removal (integration.py:552-630) and the
// cell re-index (integration.py:509-550).  It reads each SIP attribute once
// and writes it once; grid data come from small L2-resident arrays.
//
// Sums the reference accumulates in ascending SIP ID (the per-cell condensed
// mass delta_m_l, integration.py:916-936, and water_removed, :620-628) are integer
// sums of every bit of their terms here (acc_add64, which states the range), brought
// to FP64 at the end: independent of the order, so a step gives the same bits run to
// run and batched or not, within the rounding of the reference's sequential sums,
// and no sub-step needs its SIPs sorted.
#include <cuda_runtime.h>

#include <atomic>

#include "lacmo_ff.cuh"
#include "lacmo_internal.cuh"
#include "lacmo_math64.cuh"
#include "lacmo_physics.cuh"

namespace lacmo {

static inline int nblocks(int64_t n, int t, int cap = 152 * 32) {
  int64_t b = (n + t - 1) / t;
  if (b < 1) b = 1;
  return (int)(b < cap ? b : cap);
}

// ---------------------------------------------------------------------------
__global__ void k_cells_import(const int64_t* __restrict__ cells, const uint8_t* __restrict__ act,
                               int32_t* __restrict__ cell, int64_t n, int64_t nz) {
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n;
       k += (int64_t)gridDim.x * blockDim.x) {
    int64_t i = cells[k], j = cells[n + k];
    cell[k] = act[k] ? (int32_t)(i * nz + j) : (int32_t)(-1 - i);
  }
}

__global__ void k_cells_export(const int32_t* __restrict__ cell, const double* __restrict__ pos,
                               double* __restrict__ rel, int64_t* __restrict__ cells,
                               uint8_t* __restrict__ act, int64_t n, int64_t nz, double x_min,
                               double z_min, double dx, double dz) {
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n;
       k += (int64_t)gridDim.x * blockDim.x) {
    int32_t c = cell[k];
    if (c >= 0) {
      int64_t i = c / nz, j = c - (c / nz) * nz;
      cells[k] = i; cells[n + k] = j; act[k] = 1;
      rel[k] = (pos[k] - x_min) / dx - (double)i;
      rel[n + k] = (pos[n + k] - z_min) / dz - (double)j;
    } else {
      cells[k] = -1 - (int64_t)c; cells[n + k] = -1; act[k] = 0;
    }
  }
}

// per-cell terms of the mass rate for the next sub-step; their FP32 copies in
// the cell records (cell_records) feed the mixed-precision kernel without
// double->float conversions there
// the mixed path's terms and record of a cell
__device__ __forceinline__ void write_mixed(double* aux, int64_t c, int64_t C, double T, double S,
                                            double sigw, double rhow, double lap0, double lbp0,
                                            double c1, double c2, double mu, double rho_f) {
  double* const am = mixed_aux(aux, C);
  am[c] = sigw; am[C + c] = rhow; am[2 * C + c] = lap0; am[3 * C + c] = lbp0;
  am[4 * C + c] = c1; am[5 * C + c] = c2;
  float4* af = cell_records(aux, C) + CELL_REC * c;
  af[0] = make_float4((float)T, (float)(S - 1.0), (float)sigw, (float)rhow);
  af[1] = make_float4((float)lap0, (float)lbp0, (float)c1, (float)c2);
  af[2] = make_float4((float)mu, (float)rho_f, 0.0f, 0.0f);
}
// the FP64 path's
__device__ __forceinline__ void write_fp64(double* aux, int64_t c, int64_t C, double T, double S,
                                           double L_v, double mu, double rho_f,
                                           const CellTerms& t) {
  aux[c] = t.sigw; aux[C + c] = t.rhow; aux[2 * C + c] = t.lap0; aux[3 * C + c] = t.lbp0;
  aux[4 * C + c] = t.c1; aux[5 * C + c] = t.c2;
  write_rec64(cell_rec64(aux, C) + 2 * c, T, S, L_v, mu, rho_f, t);
}

__global__ void k_cell_aux(const __grid_constant__ MRef mr) {
  const Member& mb = mr.get();
  const int64_t C = mb.g.nx * mb.g.nz;
  const double *gsf = mb.g.scalar_fields, *gmp = mb.g.mat_prop;
  double* aux = mb.w.aux;
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < C;
       c += (int64_t)gridDim.x * blockDim.x)
  {
    const double T = gsf[c], p = gsf[C + c], S = gsf[6 * C + c], e_s = gsf[7 * C + c],
                 K = gmp[c], D_v = gmp[C + c], L_v = gmp[2 * C + c], mu = gmp[5 * C + c],
                 rho_f = gmp[6 * C + c];
    const CellAmb a = make_cell_amb(T, p, S, e_s, L_v, K, D_v);
    write_mixed(aux, c, C, a.T, a.S, a.sigw, a.rhow, a.lap0, a.lbp0, a.c1, a.c2, mu, rho_f);
    write_fp64(aux, c, C, T, S, L_v, mu, rho_f, cell_terms64(T, p, e_s, L_v, K, D_v));
  }
}

// ---------------------------------------------------------------------------
// binning: histogram (arrival rank) -> scan -> scatter -> order by ID
// The arrival rank of a SIP in cell c, for the lanes that come here together: one
// atomic for a run of neighbouring lanes with the same cell (SIPs in memory order
// start out cell by cell; the half-step move of 64 members, 51.9 million SIPs,
// 1204 us with an atomic each, 895 us now; k_histogram over 720,000 SIPs 35 and
// 7 us).
__device__ __forceinline__ int32_t rank_in(int32_t* counts, int32_t c) {
  const unsigned here = __activemask();
  const int lane = threadIdx.x & 31;
  const unsigned below = here & ((1u << lane) - 1u);
  const int32_t prev = __shfl_sync(here, c, below ? 31 - __clz(below) : lane);
  const unsigned heads = __ballot_sync(here, !below || prev != c);
  if (heads == here) return atomicAdd(counts + c, 1);   // no two alike (raining states)
  const unsigned upto = (2u << lane) - 1u;
  const int head = 31 - __clz(heads & upto);
  const unsigned after = heads & ~upto;
  const unsigned run = here & ~((1u << head) - 1u) & (after ? (after & -after) - 1u : ~0u);
  int32_t base = 0;
  if (lane == head) base = atomicAdd(counts + c, __popc(run));
  return __shfl_sync(here, base, head) + __popc(run & below);
}
__global__ void k_histogram(const __grid_constant__ MRef mr) {
  const Member& mb = mr.get();
  const int32_t* __restrict__ cell = mb.sp.cell;
  const int64_t n = mb.sp.n;
  int32_t *counts = mb.w.counts, *rank = mb.w.rank;
  const int64_t C = mb.g.nx * mb.g.nz;
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n;
       k += (int64_t)gridDim.x * blockDim.x) {
    int32_t c = cell[k];
    if (c < 0) continue;
    if (c < C) rank[k] = rank_in(counts, c);
    else atomicOr(mb.w.flags, LACMO_FLAG_CELL_RANGE);   // left out of the binning
  }
}

// Exclusive sums of a and b over the block's 1024 threads; the block's sums come
// back in ta, tb.  w: shared memory, free again after the caller's next barrier.
__device__ __forceinline__ void block_exclusive(int32_t& a, int64_t& b, int32_t& ta, int64_t& tb,
                                                int32_t (*wa)[33], int64_t (*wb)[33]) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int32_t x = a;
  int64_t y = b;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int32_t u = __shfl_up_sync(0xffffffffu, x, off);
    const int64_t v = __shfl_up_sync(0xffffffffu, y, off);
    if (lane >= off) { x += u; y += v; }
  }
  if (lane == 31) { (*wa)[wid] = x; (*wb)[wid] = y; }
  __syncthreads();
  // every warp sums the warps' totals up
  int32_t p = (*wa)[lane];
  int64_t q = (*wb)[lane];
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int32_t u = __shfl_up_sync(0xffffffffu, p, off);
    const int64_t v = __shfl_up_sync(0xffffffffu, q, off);
    if (lane >= off) { p += u; q += v; }
  }
  ta = __shfl_sync(0xffffffffu, p, 31);
  tb = __shfl_sync(0xffffffffu, q, 31);
  const int32_t p0 = __shfl_sync(0xffffffffu, p, wid > 0 ? wid - 1 : 0);
  const int64_t q0 = __shfl_sync(0xffffffffu, q, wid > 0 ? wid - 1 : 0);
  a = x - a + (wid ? p0 : 0);
  b = y - b + (wid ? q0 : 0);
}
// Single block: the exclusive scans of the SIP counts (slots) and pair counts
// (draws), and the collision work order: cells by descending SIP count (a counting
// sort on min(count, 1023); the order inside a size class is arbitrary).  Waits
// for barriers, loads and atomics, so a tile of 1024 cells takes one barrier, its
// counts are there before, and a warp whose cells are of one class takes their
// places with one atomic (120 cells: 5.7 us with scans through shared memory and
// strided chunks, 3.3 us now; 5625 cells: 15.6 and 9.8 us).
__global__ void __launch_bounds__(1024) k_scan(const __grid_constant__ MRef mr) {
  const Member& mb = mr.get();
  int32_t *counts = mb.w.counts, *start = mb.w.start, *order = mb.w.cell_order;
  int64_t *draw_off = mb.w.draw_off, *total_pairs = mb.w.total_pairs;
  const int64_t C = mb.g.nx * mb.g.nz;
  __shared__ int32_t s_hist[1024];
  __shared__ int32_t s_a[2][33];
  __shared__ int64_t s_b[2][33];
  const int t = threadIdx.x, lane = t & 31;
  s_hist[t] = 0;
  __syncthreads();
  auto size_class = [](int32_t m) { return 1023 - (m < 1023 ? m : 1023); };
  int32_t os = 0;
  int64_t op = 0;
  int32_t next = t < C ? counts[t] : 0;
  for (int64_t base = 0, tile = 0; base < C; base += 1024, ++tile) {
    const int64_t c = base + t;
    const int32_t m = next;
    next = c + 1024 < C ? counts[c + 1024] : 0;
    // one atomic for a warp of one class (fresh states), else one per cell
    const int key = c < C ? size_class(m) : -1;
    if (__all_sync(0xffffffffu, key == __shfl_sync(0xffffffffu, key, 0))) {
      if (lane == 0 && key >= 0) atomicAdd(&s_hist[key], 32);
    } else if (key >= 0) {
      atomicAdd(&s_hist[key], 1);
    }
    int32_t a = m, ta;
    int64_t b = (int64_t)m * (m - 1) / 2, tb;
    block_exclusive(a, b, ta, tb, &s_a[tile & 1], &s_b[tile & 1]);
    if (c < C) {
      start[c] = os + a;
      draw_off[c] = op + b;
    }
    os += ta;
    op += tb;
  }
  if (t == 0) { start[C] = os; draw_off[C] = op; *total_pairs = op; }
  __syncthreads();
  int32_t first = s_hist[t], ta;
  int64_t z = 0, tb;
  block_exclusive(first, z, ta, tb, &s_a[0], &s_b[0]);
  s_hist[t] = first;
  __syncthreads();
  for (int64_t base = 0; base < C; base += 1024) {
    const int64_t c = base + t;
    const int key = c < C ? size_class(counts[c]) : -1;
    if (c < C) counts[c] = 0;
    if (__all_sync(0xffffffffu, key == __shfl_sync(0xffffffffu, key, 0))) {
      int at = 0;
      if (lane == 0 && key >= 0) at = atomicAdd(&s_hist[key], 32);
      at = __shfl_sync(0xffffffffu, at, 0);
      if (key >= 0) order[at + lane] = (int32_t)c;
    } else if (key >= 0) {
      order[atomicAdd(&s_hist[key], 1)] = (int32_t)c;
    }
  }
}

__global__ void k_scatter(const __grid_constant__ MRef mr) {
  const Member& mb = mr.get();
  const int32_t* __restrict__ cell = mb.sp.cell;
  const int32_t* __restrict__ rank = mb.w.rank;
  const int32_t* __restrict__ start = mb.w.start;
  int32_t* perm = mb.w.perm;
  const int64_t n = mb.sp.n, C = mb.g.nx * mb.g.nz;
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n;
       k += (int64_t)gridDim.x * blockDim.x) {
    int32_t c = cell[k];
    if (c >= 0 && c < C) perm[start[c] + rank[k]] = (int32_t)k;
  }
}

// Bitonic sort of 32 * PER keys held by a warp, key[u] = element lane * PER + u,
// ascending: compare-exchange stages of distance j >= PER between lanes
// (shuffles), of smaller distance within a lane's registers.
template <int PER>
__device__ __forceinline__ void warp_bitonic(int32_t (&key)[PER], int lane) {
  constexpr int N = 32 * PER;
#pragma unroll
  for (int k = 2; k <= N; k <<= 1) {
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1) {
      if (j >= PER) {
#pragma unroll
        for (int u = 0; u < PER; ++u) {
          const int e = lane * PER + u;
          const int32_t other = __shfl_xor_sync(0xffffffffu, key[u], j / PER);
          const bool take_min = ((e & k) == 0) == ((e & j) == 0);
          key[u] = take_min ? min(key[u], other) : max(key[u], other);
        }
      } else {
#pragma unroll
        for (int u = 0; u < PER; ++u) {
          if (u & j) continue;
          const bool up = ((lane * PER + u) & k) == 0;
          const int32_t x = key[u], y = key[u ^ j];
          key[u] = up ? min(x, y) : max(x, y);
          key[u ^ j] = up ? max(x, y) : min(x, y);
        }
      }
    }
  }
}
// the L <= 32 * PER slots of one cell sorted by SIP ID in the warp's registers
template <int PER>
__device__ __forceinline__ void sort_cell_ids(int32_t* perm, int32_t b, int L, int lane) {
  int32_t key[PER];
#pragma unroll
  for (int u = 0; u < PER; ++u) {
    const int e = lane * PER + u;
    key[u] = e < L ? perm[b + e] : 0x7fffffff;
  }
  warp_bitonic<PER>(key, lane);
#pragma unroll
  for (int u = 0; u < PER; ++u) {
    const int e = lane * PER + u;
    if (e < L) perm[b + e] = key[u];
  }
}

// Number of keys of the sorted run a[0..len) that are below x (IDs are
// unique, so keys of the other run never tie with x).
__device__ __forceinline__ int32_t count_below(const int32_t* a, int32_t len, int32_t x) {
  int32_t lo = 0, hi = len;
  while (lo < hi) {
    const int32_t mid = (lo + hi) >> 1;
    if (a[mid] < x) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// one warp per cell: order the cell's slots by ascending SIP ID.  Up to 256
// slots: a bitonic sort in registers.  Larger cells: runs of 256 sorted in
// registers, then merged pairwise, each key placed at its rank in the merged
// run (its index in its own run plus a binary search in the other), ping-pong
// between perm and the rank array (free after the scatter); O(L log L).
constexpr int ORDER_SMEM = 256;
__global__ void __launch_bounds__(256) k_order(const __grid_constant__ MRef mr) {
  const Member& mb = mr.get();
  const int32_t* __restrict__ start = mb.w.start;
  int32_t *perm = mb.w.perm, *scratch = mb.w.rank;
  const int64_t C = mb.g.nx * mb.g.nz;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int64_t c = blockIdx.x * 8LL + wid; c < C; c += (int64_t)gridDim.x * 8) {
    const int32_t b = start[c], L = start[c + 1] - b;
    if (L <= 1) continue;
    if (L <= ORDER_SMEM) {
      if (L <= 64) sort_cell_ids<2>(perm, b, L, lane);
      else if (L <= 128) sort_cell_ids<4>(perm, b, L, lane);
      else sort_cell_ids<8>(perm, b, L, lane);
      __syncwarp();
      continue;
    }
    for (int32_t r0 = 0; r0 < L; r0 += ORDER_SMEM) {
      const int32_t len = L - r0 < ORDER_SMEM ? L - r0 : ORDER_SMEM;
      sort_cell_ids<8>(perm, b + r0, len, lane);
    }
    __syncwarp();
    int32_t* src = perm + b;
    int32_t* dst = scratch + b;
    for (int32_t width = ORDER_SMEM; width < L; width <<= 1) {
      for (int32_t lo = 0; lo < L; lo += 2 * width) {
        const int32_t mid = lo + width < L ? lo + width : L;
        const int32_t hi = lo + 2 * width < L ? lo + 2 * width : L;
        const int32_t *A = src + lo, *Bv = src + mid;
        const int32_t la = mid - lo, lb = hi - mid;
        for (int32_t q = lane; q < la; q += 32) dst[lo + q + count_below(Bv, lb, A[q])] = A[q];
        for (int32_t q = lane; q < lb; q += 32) dst[lo + q + count_below(A, la, Bv[q])] = Bv[q];
      }
      __syncwarp();
      int32_t* t = src; src = dst; dst = t;
    }
    if (src != perm + b)
      for (int32_t q = lane; q < L; q += 32) perm[b + q] = src[q];
    __syncwarp();
  }
}

// ---- exact sums of FP64 values as integers in units of 2^-64 (fg): four words
// of b bits each, each summed by a 64-bit integer atomic (executed by L2, in any
// order).  b = acc_bits(n) leaves a word room for one value from every SIP of the
// member, so no word wraps: |sum of n parts below 2^b| < 2^62.  A value keeps all
// its bits from 2^-12 fg up; below that it is rounded to 2^-64 fg.  What lies
// beyond the four words (2^104 fg for up to 2^20 SIPs, 2^60 fg for 2^31),
// infinities and NaN go to a plain FP64 sum (over).
constexpr int ACC64_WORDS = 4, ACC64_UNIT = 64;
__device__ __forceinline__ int acc_bits(int64_t n) {
  const int log_n = n > 1 ? 64 - __clzll(n - 1) : 0;   // n <= 2^log_n
  return log_n < 20 ? 42 : 62 - log_n;
}
__device__ __forceinline__ void acc_add64(long long* acc, int bits, double* over, double v) {
  const uint64_t u = (uint64_t)__double_as_longlong(v);
  int s = (int)((u >> 52) & 0x7ffu) - (1075 - ACC64_UNIT);   // v 2^64 = m 2^s
  if (s > ACC64_WORDS * bits - 53) {
    atomicAdd(over, v);
    return;
  }
  if (s < -53) return;   // rounds to zero
  uint64_t m = (u & 0x000fffffffffffffull) | 0x0010000000000000ull;
  if (s < 0) {
    m = (m + (1ull << (-s - 1))) >> (-s);
    s = 0;
  }
  // m 2^s from word k on: 53 bits reach into at most three words
  const int k = (s >= bits) + (s >= 2 * bits) + (s >= 3 * bits);
  s -= k * bits;
  const uint64_t mask = (1ull << bits) - 1;
  uint64_t p0 = (m << s) & mask;
  m >>= bits - s;
  uint64_t p1 = m & mask, p2 = m >> bits;
  if (u >> 63) { p0 = 0 - p0; p1 = 0 - p1; p2 = 0 - p2; }
  unsigned long long* const w = (unsigned long long*)acc + k;
  if (p0) atomicAdd(w, (unsigned long long)p0);
  if (p1) atomicAdd(w + 1, (unsigned long long)p1);
  if (p2) atomicAdd(w + 2, (unsigned long long)p2);
}
// The sum, within 0.8 of its last place: the words' carries taken up so that each
// holds at most half of 2^b, then from the top down; the sums are exact up to 53
// bits, and from the first one rounded on a word adds a quarter of a last place
// at most.
__device__ __forceinline__ double acc_value64(longlong2 a, longlong2 b, int bits) {
  const long long half = 1ll << (bits - 1);
  long long c = (a.x + half) >> bits;
  const long long w0 = a.x - (c << bits);
  a.y += c;
  c = (a.y + half) >> bits;
  const long long w1 = a.y - (c << bits);
  b.x += c;
  c = (b.x + half) >> bits;
  const long long w2 = b.x - (c << bits), w3 = b.y + c;
  const double base = __longlong_as_double((long long)(1023 + bits) << 52);
  double v = (double)w1;
  if (w2 | w3) v = fma(fma((double)w3, base, (double)w2), base, v);
  return fma(v, base, (double)w0) * 0x1p-64;
}
__device__ __forceinline__ double acc_read64(const long long* acc, int bits) {
  const longlong2* const p = (const longlong2*)acc;
  return acc_value64(p[0], p[1], bits);
}
__device__ __forceinline__ void acc_clear64(long long* acc) {
  longlong2* const p = (longlong2*)acc;
  p[0] = p[1] = make_longlong2(0, 0);
}

// ---------------------------------------------------------------------------
struct PArgs {
  double *pos, *vel, *m_w, *rel, *T_p;
  const double *m_s, *xi;
  int32_t* cell;
  const double *gsf, *gmp, *aux, *gv;
  int64_t n, nx, nz;
  double x_min, x_max, z_min, z_cap, dx, dz;
  double dt_sub, dt_pos, g_set;
  int no_iter, sol, write_Tp;
  int32_t *counts, *rank;
  long long *acc64, *wr64;      // FP64: per-cell and water sums (acc_add64)
  double* accx;                 // FP64: values beyond their range
  int acc_bits;                 // FP64: bits of the sums' words
  // mixed precision: SIPs whose Newton repeats in FP64 (k_newton_fallback),
  // queued in scratch that mixed sub-steps leave unused
  int32_t *fb_count, *fb_done, *fb_id, *fb_c;
  double* fb_mw;
  uint32_t* flags;
  // mixed precision
  double* acc;                  // [C] per-cell sums of dm * xi, int64 units of 2^-4 fg
  int hist;                     // count SIPs per new cell for a following binning
  unsigned long long* nfb;      // SIPs whose Newton fell back to FP64
  const float4* crec;           // [C][CELL_REC] FP32 cell records (cell_records)
  double inv_dx, inv_dz;
  float inv_dxf, inv_dzf, dt_subf, dtg_f, dt_posf;
  float x_minf, x_maxf, z_minf, z_capf;
  double* water_removed;
};

// per-call scalars of a particle sub-step (common to all members)
struct PCall {
  double dt_sub, dt_pos, g_set;
  int no_iter, sol, write_Tp, hist;
  float dt_subf, dtg_f, dt_posf;
};
struct PK {
  MRef m;
  PCall c;
};

__device__ __forceinline__ PArgs make_pargs(const Member& mb, const PCall& c) {
  PArgs a;
  const lacmo_sips_t& sp = mb.sp;
  const lacmo_grid_t& g = mb.g;
  const Ws& w = mb.w;
  a.pos = sp.pos; a.vel = sp.vel; a.m_w = sp.m_w; a.rel = sp.rel_pos; a.T_p = sp.T_p;
  a.m_s = sp.m_s; a.xi = sp.xi; a.cell = sp.cell;
  a.gsf = g.scalar_fields; a.gmp = g.mat_prop; a.aux = w.aux; a.gv = g.velocity;
  a.n = sp.n; a.nx = g.nx; a.nz = g.nz;
  a.x_min = g.x_min; a.x_max = g.x_max; a.z_min = g.z_min; a.z_cap = mb.z_cap;
  a.dx = g.dx; a.dz = g.dz;
  a.dt_sub = c.dt_sub; a.dt_pos = c.dt_pos; a.g_set = c.g_set;
  a.no_iter = c.no_iter; a.sol = c.sol; a.write_Tp = c.write_Tp;
  a.counts = w.counts; a.rank = w.rank; a.flags = w.flags;
  a.acc64 = w.acc64; a.wr64 = w.wr64; a.accx = w.accx; a.acc_bits = acc_bits(sp.n);
  a.fb_count = w.fb_count; a.fb_done = w.fb_done; a.fb_id = w.rm_id; a.fb_c = w.colk;
  a.fb_mw = w.rm_val;
  a.acc = w.div; a.hist = c.hist; a.nfb = w.nfb;
  a.crec = cell_records(w.aux, g.nx * g.nz);
  a.inv_dx = mb.inv_dx; a.inv_dz = mb.inv_dz;
  a.inv_dxf = mb.inv_dxf; a.inv_dzf = mb.inv_dzf;
  a.dt_subf = c.dt_subf; a.dtg_f = c.dtg_f; a.dt_posf = c.dt_posf;
  a.x_minf = mb.x_minf; a.x_maxf = mb.x_maxf; a.z_minf = mb.z_minf; a.z_capf = mb.z_capf;
  a.water_removed = sp.water_removed;
  return a;
}


// The wind corners the FP32 interpolation of grid.py:257-323 can read in cell
// (i, j), in float4 3..5 of the cell's record (float4 6 holds i, j and
// whether j is the bottom or top row): U[a][b] = u at (i + a,
// j - 1 + b), a < 2, b < 3, and V[a][b] = w at (i - 1 + a, j + b), a < 3,
// b < 2, as (U00 U01 U02 U10) (U11 U12 V00 V01) (V10 V11 V20 V21); indices
// below zero wrap like the reference's (the periodic column i = -1 is column
// nx; row j - 1 = -1 is never read).
__global__ void k_wind_table(const __grid_constant__ MRef mr) {
  const Member& mb = mr.get();
  const double* in = mb.g.velocity;
  const int64_t nx = mb.g.nx, nz = mb.g.nz, C = nx * nz;
  float4* rec = cell_records(mb.w.aux, C);
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < C;
       c += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = c / nz, j = c - i * nz;
    auto at = [&](int comp, int64_t ii, int64_t jj) {
      if (ii < 0) ii += nx + 1;
      if (jj < 0) jj += nz + 1;
      return (float)in[((int64_t)comp * (nx + 1) + ii) * (nz + 1) + jj];
    };
    float4* out = rec + CELL_REC * c;
    out[3] = make_float4(at(0, i, j - 1), at(0, i, j), at(0, i, j + 1), at(0, i + 1, j - 1));
    out[4] = make_float4(at(0, i + 1, j), at(0, i + 1, j + 1), at(1, i - 1, j), at(1, i - 1, j + 1));
    out[5] = make_float4(at(1, i, j), at(1, i, j + 1), at(1, i + 1, j), at(1, i + 1, j + 1));
    out[6] = make_float4((float)i, (float)j, j == 0 ? 1.0f : 0.0f, j == nz - 1 ? 1.0f : 0.0f);
  }
}

// grid.py:257-323 in FP32 from a cell's wind corners (k_wind_table); wx, wy
// are the position in the cell in units of the cell size, jlo / jhi mark the
// bottom and top rows of cells
__device__ __forceinline__ void interp_wind(const float4 w0, const float4 w1, const float4 w2,
                                            bool jlo, bool jhi, float wx, float wy, float& u,
                                            float& v) {
  if ((jlo && wy <= 0.5f) || (jhi && wy >= 0.5f)) {
    u = wx * w1.x + (1 - wx) * w0.y;
  } else if (wy > 0.5f) {
    const float b = wy - 0.5f;
    u = wx * (b * w1.y + (1 - b) * w1.x) + (1 - wx) * (b * w0.z + (1 - b) * w0.y);
  } else {
    const float b = wy + 0.5f;
    u = wx * (b * w1.x + (1 - b) * w0.w) + (1 - wx) * (b * w0.y + (1 - b) * w0.x);
  }
  if (wx > 0.5f) {
    const float a = wx - 0.5f;
    v = a * (wy * w2.w + (1 - wy) * w2.z) + (1 - a) * (wy * w2.y + (1 - wy) * w2.x);
  } else {
    const float a = wx + 0.5f;
    v = a * (wy * w2.y + (1 - wy) * w2.x) + (1 - a) * (wy * w1.w + (1 - wy) * w1.z);
  }
}

// The records of the FP64 kernel from the grid's arrays as they are now: the
// thermodynamic terms (the cell update rewrites them every sub-step), and the wind
// (grid.py:257-323): the values the bilinear interpolation starts from and the
// differences between its corners (indices below zero wrap as in k_wind_table).
// known: the cell's six terms are the stored ones (no mixed-precision step came
// after they were written), which leaves out most of the chain of FP64 operations.
__global__ void k_records64(const __grid_constant__ MRef mr, int known) {
  const Member& mb = mr.get();
  const double *gsf = mb.g.scalar_fields, *gmp = mb.g.mat_prop;
  const double* in = mb.g.velocity;
  const int64_t nx = mb.g.nx, nz = mb.g.nz, C = nx * nz;
  WindFF* rec = (WindFF*)cell_rec64(mb.w.aux, C);
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < C;
       c += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = c / nz, j = c - i * nz;
    auto at = [&](int comp, int64_t ii, int64_t jj) {
      if (ii < 0) ii += nx + 1;
      if (jj < 0) jj += nz + 1;
      return in[((int64_t)comp * (nx + 1) + ii) * (nz + 1) + jj];
    };
    WindFF w;
    w.U0[0] = at(0, i, j - 1); w.U0[1] = at(0, i, j);
    for (int b = 0; b < 3; ++b) w.dxU[b] = at(0, i + 1, j - 1 + b) - at(0, i, j - 1 + b);
    for (int b = 0; b < 2; ++b) w.dyU[b] = at(0, i, j + b) - at(0, i, j - 1 + b);
    w.V0[0] = at(1, i - 1, j); w.V0[1] = at(1, i, j);
    for (int a = 0; a < 3; ++a) w.dyV[a] = at(1, i - 1 + a, j + 1) - at(1, i - 1 + a, j);
    for (int a = 0; a < 2; ++a) w.dxV[a] = at(1, i + a, j) - at(1, i - 1 + a, j);
    w.i = (int32_t)i; w.j = (int32_t)j;
    w.edge = (j == 0 ? 1 : 0) | (j == nz - 1 ? 2 : 0);
    w.pad = 0;
    rec[2 * c + 1] = w;
    const double T = gsf[c], S = gsf[6 * C + c], L_v = gmp[2 * C + c], mu = gmp[5 * C + c],
                 rho_f = gmp[6 * C + c];
    if (known) {
      const double* const a = mb.w.aux + c;
      const CellTerms t{a[0], a[C], a[2 * C], a[3 * C], a[4 * C], a[5 * C]};
      write_rec64(cell_rec64(mb.w.aux, C) + 2 * c, T, S, L_v, mu, rho_f, t);
    } else {
      write_fp64(mb.w.aux, c, C, T, S, L_v, mu, rho_f,
                 cell_terms64(T, gsf[C + c], gsf[7 * C + c], L_v, gmp[c], gmp[C + c]));
    }
  }
}
// the sum of the water removed at the ground into water_removed; one thread
__device__ __forceinline__ void take_water(const Member& mb) {
  long long* const wr = mb.w.wr64;
  if (wr[0] | wr[1] | wr[2] | wr[3]) {
    mb.sp.water_removed[0] += acc_read64(wr, acc_bits(mb.sp.n));
    acc_clear64(wr);
  }
}
// where no cell update follows: the water removed is taken, the cells' sums are
// dropped
__global__ void k_clear_acc64(const __grid_constant__ MRef mr) {
  const Member& mb = mr.get();
  const int64_t C = mb.g.nx * mb.g.nz;
  if (blockIdx.x == 0 && threadIdx.x == 0) take_water(mb);
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < C;
       c += (int64_t)gridDim.x * blockDim.x) {
    acc_clear64(mb.w.acc64 + ACC64_WORDS * c);
    mb.w.accx[c] = 0.0;
  }
}

// Rare paths of the FP64 kernel, out of line.
// near or past a boundary: periodic x (integration.py:577-583), capped z
// (:585-589), and whether the SIP reached the ground (:606)
struct Edges {
  double x_max, z_cap, z_min;
};
__device__ __noinline__ int particle_edges(Edges e, double x, double z, double* xo, double* zo) {
  x = py_mod(x, e.x_max);
  z = np_min(z, e.z_cap);
  *xo = x; *zo = z;
  return z <= e.z_min ? 1 : 0;
}
__device__ __noinline__ int floor_div(double x, double d) {
  const double q = floor(x / d);
  return q > 2.0e9 ? 2000000000 : (q < -2.0e9 ? -2000000000 : (q == q ? (int)q : -1));
}
// the Newton of SIPs outside the two-float form's bounds: newton_fast, for
// masses beyond FP32 and NaN newton_full
__device__ __noinline__ double particle_newton64(const PArgs& a, int32_t c, double mw, double ms) {
  const int64_t C = a.nx * a.nz;
  CellAmb amb;
  amb.T = a.gsf[c]; amb.p = a.gsf[C + c]; amb.S = a.gsf[6 * C + c]; amb.e_s = a.gsf[7 * C + c];
  amb.K = a.gmp[c]; amb.D_v = a.gmp[C + c]; amb.L_v = a.gmp[2 * C + c];
  amb.sigw = a.aux[c]; amb.rhow = a.aux[C + c]; amb.lap0 = a.aux[2 * C + c];
  amb.lbp0 = a.aux[3 * C + c]; amb.c1 = a.aux[4 * C + c]; amb.c2 = a.aux[5 * C + c];
  if (ff_mass_ok(mw) && ff_mass_ok(ms))
    return newton_fast(a.sol, a.dt_sub, a.no_iter, mw, ms, cell_fast(a.sol, amb), 1.0) - mw;
  const double m_p = mw + ms;
  const double w_s = ms / m_p;
  const double rho = (a.sol == SOL_AS) ? density_AS_solution_rw(w_s, amb.rhow)
                                       : density_NaCl_solution(w_s, amb.T);
  const double R = radius_from_mass(m_p, rho);
  const double sig = (a.sol == SOL_AS) ? surface_tension_AS_sw(w_s, amb.sigw)
                                       : surface_tension_NaCl_sw(w_s, amb.sigw);
  return newton_full(a.sol, a.dt_sub, a.no_iter, mw, ms, w_s, R, amb.T, rho, sig, amb, nullptr);
}
// the drag update of integration.py:699-718 in FP64 throughout, for drops
// whose velocity does not follow the air (k dt below 8, radii above some 30 um)
// or with a Reynolds correction
__device__ __noinline__ void particle_drag64(const PArgs& a, int32_t c, double mw, double ms,
                                             double uf, double wf, double* u, double* w) {
  const int64_t C = a.nx * a.nz;
  const double m_p = mw + ms;
  const double rho = density_AS_solution_rw(ms / m_p, a.aux[C + c]);
  const double R = radius_from_mass(m_p, rho);
  const double mu_f = a.gmp[5 * C + c], rho_f = a.gmp[6 * C + c];
  const double d0 = uf - *u, d1 = wf - *w;
  const double vel_dev = sqrt(d0 * d0 + d1 * d1);
  const double Re_p = 2.0E-6 * rho_f * R * vel_dev / mu_f;
  double k_dt = 4.5E12 * a.dt_sub * mu_f / (rho * R * R);
  if (Re_p > 0.5) {
    if (Re_p < 1000.0) k_dt *= (1 + 0.15 * pow(Re_p, 0.687));
    else k_dt *= 0.0183333333333 * Re_p;
  }
  *u = (*u + k_dt * uf) / (1.0 + k_dt);
  *w = (*w + k_dt * wf - a.dt_sub * a.g_set) / (1.0 + k_dt);
}
// a SIP removed earlier: its position moves on, its relative position keeps
// the per-call division of integration.py:548-549
__device__ __noinline__ void particle_inactive(const PArgs& a, int64_t k, int32_t c) {
  const int64_t i = -1 - (int64_t)c;
  const double x = a.pos[k] + a.dt_pos * a.vel[k];
  const double z = a.pos[a.n + k] + a.dt_pos * a.vel[a.n + k];
  a.pos[k] = py_mod(x, a.x_max);
  a.pos[a.n + k] = np_min(z, a.z_cap);
  a.rel[k] = a.rel[k] / a.dx - (double)i;
  a.rel[a.n + k] = a.rel[a.n + k] / a.dz - (-1.0);
}
// a SIP reaching the ground (integration.py:606-630); returns its new z
__device__ __noinline__ double particle_removed(const PArgs& a, int64_t k, int32_t c, double x,
                                                double z, double mw) {
  const int64_t i = (int64_t)c / a.nz, j = (int64_t)c - i * a.nz;
  acc_add64(a.wr64, a.acc_bits, a.water_removed, a.xi[k] * mw);
  const double rel_x = (x - a.x_min) / a.dx - (double)i;
  const double rel_z = (z - a.z_min) / a.dz - (double)j;
  // the re-index of this call leaves the old relative position divided by the
  // cell size (integration.py:548-549)
  a.rel[k] = rel_x / a.dx - (double)i;
  a.rel[a.n + k] = rel_z / a.dz - (-1.0);
  return a.z_min - 0.01 * a.dz;
}

// The FP64 sub-step.  In plain FP64 this kernel was bound by the FP64 pipe: some
// 670 FP64 instructions per SIP at 2 lanes an SM and clock, 478 us per launch
// over 360,000 SIPs.  The Newton and the drag now run in two-float arithmetic
// around the FP64 operations that decide the result's rounding (lacmo_ff.cuh;
// about 65 a SIP are left, and some 3700 FP32 and integer instructions): 85 us once
// few SIPs need plain FP64, 95 us averaged over 20 sub-steps from a state out of
// equilibrium.
// New cell indices come from the FP32 position where it is clear of the cell's
// edges, boundaries likewise.
// SIPs that need plain FP64 for the Newton (a step of more than an eighth of
// the mass, a radius below 5 nm, no solute) or the drag (drops above some 30 um) wait
// in the block's queue until its other SIPs are done: a few of them in every warp
// would hold all warps on the FP64 pipe, gathered they fill a few warps (a
// raining state of 545,000 SIPs, 1.3% of them large drops, averaged the same way:
// 291 us in place, 217 us gathered, 144 us with newton_fast and no more blocks than
// are resident, 135 us when the queue's second pass does only what is left of a SIP;
// 732 us in plain FP64).  Which of these ways a SIP takes follows from its own state
// and gives the same bits in place and from the queue.
__device__ __forceinline__ double i2d_int(int i) {   // i >= 0
  return i < (1 << 24) ? f2d_int((float)i) : (double)i;
}
constexpr int PQ = 1024;   // queue slots; a SIP beyond them is done in place
template <bool PHYS, bool FULL>
__global__ void __launch_bounds__(128) k_particles(const __grid_constant__ PK x) {
  __shared__ PArgs s_a;
  __shared__ int32_t s_q[PHYS ? PQ : 1];
  __shared__ int s_n;
  if (threadIdx.x == 0) {
    s_a = make_pargs(x.m.get(), x.c);
    s_n = 0;
  }
  __syncthreads();
  const PArgs& a = s_a;
  const int64_t C = a.nx * a.nz;
  const int nx = (int)a.nx, nz = (int)a.nz;
  const CellFF* const rec = cell_rec64((double*)a.aux, C);
  // FP32 positions are within 2^-23 of the domain: margins around boundaries
  // (m) and cell edges (cells) inside which FP64 decides
  const float ext = fmaxf(fmaxf(fabsf(a.x_maxf), fabsf(a.z_capf)), fabsf(a.z_minf));
  const float mpos = fmaxf(1e-3f, ext * 0x1p-20f);
  const float mcell = fmaxf(1e-4f, fmaxf((float)nx, (float)nz) * 0x1p-20f);
  // pass 0: the block's SIPs; pass 1: its queue
#pragma unroll 1
  for (int pass = 0; pass < (PHYS ? 2 : 1); ++pass) {
    if (pass) __syncthreads();
    const int64_t stride = pass ? blockDim.x : (int64_t)gridDim.x * blockDim.x;
    const int64_t end = pass ? min(s_n, PQ) : a.n;
#pragma unroll 1
    for (int64_t q = pass ? threadIdx.x : blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < end;
         q += stride) {
      // a queue entry: SIP, and in the sign bit whether its Newton is still to do
      // (else its new mass is stored and only the drag is left)
      const int32_t e = pass ? s_q[q] : 0;
      const bool redo = e < 0;
      const int64_t k = pass ? (int64_t)(e & 0x7fffffff) : q;
      const int32_t c = a.cell[k];
      if (c < 0) {
        if (PHYS && a.write_Tp) a.T_p[k] = __ldg(a.gsf + (int64_t)(-1 - c) * nz + nz - 1);
        particle_inactive(a, k, c);
        continue;
      }
      const double x0 = a.pos[k], z0 = a.pos[a.n + k];
      double u = a.vel[k], w = a.vel[a.n + k];
      double mw = PHYS ? a.m_w[k] : 0.0;
      if (PHYS) {
        const double ms = a.m_s[k];
        const WindFF* const wr = (const WindFF*)(rec + 2 * (int64_t)c + 1);
        CellFF cf;
        {
          const float4* src = (const float4*)(rec + 2 * (int64_t)c);
          float4* dst = (float4*)&cf;
#pragma unroll
          for (int e = 0; e < 6; ++e) dst[e] = __ldg(src + e);
        }
        double m = mw, dm = 0.0;
        if (pass == 0) {
          // masses outside the two-float range (pure water) gain nothing from the
          // queue where they fill the warp
          bool ok = ff_mass_ok(mw) && ff_mass_ok(ms);
          const bool gather = __any_sync(__activemask(), ok) != 0;
          if (ok) {
            m = newton_ff<false, FULL>(a.sol, a.no_iter, mw, ms, cf,
                                       d2ff(LC_FOUR_PI * 1.0E12 * a.dt_sub), 1.0, &ok);
            dm = m - mw;   // a step below m / 8: mw + dm is m
          }
          if (!ok) {
            const int at = gather ? atomicAdd(&s_n, 1) : PQ;
            if (at < PQ) {
              s_q[at] = (int32_t)((uint32_t)k | 0x80000000u);
              continue;
            }
            dm = particle_newton64(a, c, mw, ms);
            m = mw + dm;
          }
        } else if (redo) {
          dm = particle_newton64(a, c, mw, ms);
          m = mw + dm;
        }
        if (pass == 0 || redo)
          acc_add64(a.acc64 + ACC64_WORDS * (int64_t)c, a.acc_bits, a.accx + c, dm * a.xi[k]);
        // integration.py:699-718 with the radius of ammonium sulfate whatever the
        // solute (:1075): the wind at the SIP
        const int4 wi = __ldg((const int4*)&wr->i);
        // (no FP64 instruction for an origin at 0 or for an index)
        double xo = x0, zo = z0;
        if (__double_as_longlong(a.x_min) << 1) xo = x0 - a.x_min;
        if (__double_as_longlong(a.z_min) << 1) zo = z0 - a.z_min;
        const double rx = fma(-i2d_int(wi.x), a.dx, xo) * a.inv_dx;
        const double rz = fma(-i2d_int(wi.y), a.dz, zo) * a.inv_dz;
        const double* const wd = (const double*)wr;
        auto ld = [&](int at) { return __ldg(wd + at); };
        // compared with 0.5 by their bits (an FP32 copy would take the wrong piece
        // next to it)
        const long long half = 0x3fe0000000000000ll;
        const long long bx = __double_as_longlong(rx), bz = __double_as_longlong(rz);
        double uf, wf;
        {
          // rows of u: b0 = 0 below the cell's middle (row j - 1), 1 above; the
          // bottom and top rows are linear in x at their outer half
          const bool lin = ((wi.z & 1) && bz <= half) || ((wi.z & 2) && bz >= half);
          const int b0 = (lin || bz > half) ? 1 : 0;
          const double dx0 = ld(2 + b0);
          uf = fma(rx, dx0, ld(b0));
          if (!lin)
            uf = fma(rz + (b0 ? -0.5 : 0.5), fma(rx, ld(3 + b0) - dx0, ld(5 + b0)), uf);
          const int a0 = bx > half ? 1 : 0;
          const double dy0 = ld(9 + a0);
          wf = fma(rx + (a0 ? -0.5 : 0.5), fma(rz, ld(10 + a0) - dy0, ld(12 + a0)),
                   fma(rz, dy0, ld(7 + a0)));
        }
        const double du = uf - u, dw = wf - w;
        const ff mpf = d2ff(m + ms);
        const ff wfr = ff_mul(d2ff(ms), ff_rcp(mpf));
        ff pr = ff_horner(FFC(LC_PAR_RHO_AS_1), FFC(LC_PAR_RHO_AS_0), wfr);
        pr = ff_horner(FFC(LC_PAR_RHO_AS_2), pr, wfr);
        const ff ipr = ff_rcp(ff_one_plus(ff_mul(pr, wfr)));
        const ff xr = ff_mul(ff_mul(cf.cx, mpf), ipr);
        const ff z = ff_icbrt(xr);   // 1 / R
        const ff kd = ff_mul(ff_mul(ff_mul(d2ff(4.5E12 * a.dt_sub), cf.mr), ipr), ff_mul(z, z));
        const ff duf = d2ff(du), dwf = d2ff(dw + a.dt_sub * a.g_set);
        const float dwh = d2f_int(dw);
        const float Re = 2.0E-6f * cf.rm * f_sqrt(duf.h * duf.h + dwh * dwh) * f_rcp(z.h);
        if (Re < 0.499f && kd.h > 8.0f && ff_mass_ok(m + ms)) {
          // (u + k uf) / (1 + k) = uf - (uf - u) / (1 + k)
          const ff inv = ff_rcp(ff_add(kd, 1.0f));
          u = uf - ff2d_of<FULL>(ff_mul(duf, inv));
          w = wf - ff2d_of<FULL>(ff_mul(dwf, inv));
        } else {
          if (pass == 0) {
            const int at = atomicAdd(&s_n, 1);
            if (at < PQ) {
              a.m_w[k] = m;
              s_q[at] = (int32_t)k;
              continue;
            }
          }
          particle_drag64(a, c, m, ms, uf, wf, &u, &w);
        }
        mw = m;
        if (a.write_Tp) a.T_p[k] = __ldg(a.gsf + c);
      }
      // integration.py:552-630
      double xn = x0 + a.dt_pos * u, zn = z0 + a.dt_pos * w;
      float px = d2f_int(xn), pz = d2f_int(zn);
      bool removed = false;
      if (!(px > mpos && px < a.x_maxf - mpos && pz < a.z_capf - mpos && pz > a.z_minf + mpos)) {
        removed = particle_edges(Edges{a.x_max, a.z_cap, a.z_min}, xn, zn, &xn, &zn) != 0;
        px = d2f_int(xn); pz = d2f_int(zn);
      }
      int32_t newc;
      if (removed) {
        zn = particle_removed(a, k, c, x0, z0, PHYS ? mw : a.m_w[k]);
        u = 0.0; w = 0.0;
        newc = -1 - (int32_t)(c / nz);
      } else {
        const float qx = px * a.inv_dxf, qz = pz * a.inv_dzf;
        int ci = __float2int_rd(qx), cj = __float2int_rd(qz);
        const float fx = qx - floorf(qx), fz = qz - floorf(qz);
        if (!(fx > mcell && fx < 1.0f - mcell)) ci = floor_div(xn, a.dx);
        if (!(fz > mcell && fz < 1.0f - mcell)) cj = floor_div(zn, a.dz);
        if (ci >= nx || ci < 0 || cj >= nz || cj < 0) {
          atomicOr(a.flags, LACMO_FLAG_CELL_CLAMPED);
          ci = ci < 0 ? 0 : (ci >= nx ? nx - 1 : ci);
          cj = cj < 0 ? 0 : (cj >= nz ? nz - 1 : cj);
        }
        newc = ci * nz + cj;
        if (a.hist) a.rank[k] = rank_in(a.counts, newc);
      }
      a.pos[k] = xn; a.pos[a.n + k] = zn;
      if (PHYS || removed) { a.vel[k] = u; a.vel[a.n + k] = w; }
      if (PHYS) a.m_w[k] = mw;
      a.cell[k] = newc;
    }
  }
}

// ---------------------------------------------------------------------------
// integration.py:402-484 for one cell (and update_material_properties :359),
// and the cell's terms and records for the next sub-step (aux may be null)
__device__ __forceinline__ void grid_cell_update(double* gsf, double* gmp, double* aux, int64_t c,
                                                 int64_t C, double p_ref, double p_ref_inv,
                                                 double dTh, double drv, double dml, double V) {
  double Th = gsf[2 * C + c], r_v = gsf[4 * C + c];
  const double rho_d = gsf[3 * C + c];
  cell_step64(&Th, &r_v, rho_d, gsf[8 * C + c], gmp[2 * C + c], dTh, drv, dml, V, p_ref_inv);
  const CellState a = cell_state64(Th, r_v, rho_d, p_ref, p_ref_inv);
  gsf[c] = a.T; gsf[C + c] = a.p; gsf[2 * C + c] = Th; gsf[4 * C + c] = r_v;
  gsf[6 * C + c] = a.S; gsf[7 * C + c] = a.e_s;
  gmp[c] = a.K; gmp[C + c] = a.D_v; gmp[2 * C + c] = a.L_v;
  gmp[4 * C + c] = LC_C_PD * (1 + 0.897 * r_v); gmp[5 * C + c] = a.mu; gmp[6 * C + c] = a.rho_f;
  gmp[3 * C + c] = a.t.sigw;
  if (aux) {
    write_mixed(aux, c, C, a.T, a.S, a.t.sigw, a.t.rhow, a.t.lap0, a.t.lbp0, a.t.c1, a.t.c2, a.mu,
                a.rho_f);
    write_fp64(aux, c, C, a.T, a.S, a.L_v, a.mu, a.rho_f, a.t);
  }
}

// grid_cell_update by four lanes of a warp for each cell (role 0 to 3), bit for
// bit.  in: a cell to be written.
__device__ __forceinline__ void grid_cell_update_x4(double* gsf, double* gmp, double* aux,
                                                    int64_t c, int64_t C, double p_ref,
                                                    double p_ref_inv, double dTh, double drv,
                                                    double dml, double V, bool in) {
  const int role = threadIdx.x & 3;
  double Th = gsf[2 * C + c], r_v = gsf[4 * C + c];
  const double rho_d = gsf[3 * C + c];
  cell_step64(&Th, &r_v, rho_d, gsf[8 * C + c], gmp[2 * C + c], dTh, drv, dml, V, p_ref_inv);
  double irho, kelvin;
  const CellState a = cell_state64_x4(Th, r_v, rho_d, p_ref, p_ref_inv, &irho, &kelvin);
  if (!in) return;
  if (role == 0) {
    gsf[c] = a.T; gsf[C + c] = a.p; gsf[2 * C + c] = Th; gsf[4 * C + c] = r_v;
    gsf[6 * C + c] = a.S; gsf[7 * C + c] = a.e_s;
    write_mixed(aux, c, C, a.T, a.S, a.t.sigw, a.t.rhow, a.t.lap0, a.t.lbp0, a.t.c1, a.t.c2, a.mu,
                a.rho_f);
  } else if (role == 1) {
    gmp[c] = a.K; gmp[C + c] = a.D_v; gmp[2 * C + c] = a.L_v; gmp[3 * C + c] = a.t.sigw;
    gmp[4 * C + c] = LC_C_PD * (1 + 0.897 * r_v); gmp[5 * C + c] = a.mu; gmp[6 * C + c] = a.rho_f;
  } else if (role == 2) {
    aux[c] = a.t.sigw; aux[C + c] = a.t.rhow; aux[2 * C + c] = a.t.lap0;
    aux[3 * C + c] = a.t.lbp0; aux[4 * C + c] = a.t.c1; aux[5 * C + c] = a.t.c2;
  } else {
    write_rec64(cell_rec64(aux, C) + 2 * c, a.T, a.S, a.L_v, a.mu, a.rho_f, a.t, irho, kelvin);
  }
}

// Four lanes per cell: delta_m_l from the cell's exact sum of dm*xi
// (integration.py:916-936; then zeroed), the grid update of the cell and its
// terms for the next sub-step; the first thread adds the water removed at the
// ground.  Bound by the latency of a cell's chain (120 cells: 13.8 us with one
// thread per cell, 10.5 us now; 5625 cells: 14.3 and 12.7 us).
__global__ void __launch_bounds__(32) k_cell_update(const __grid_constant__ MRef mr,
                                                     int grid_update) {
  const Member& mb = mr.get();
  double *delta_m_l = mb.g.delta_m_l, *gsf = mb.g.scalar_fields, *gmp = mb.g.mat_prop,
         *aux = mb.w.aux;
  const double *dTh = mb.w.dTh, *drv = mb.w.drv;
  const int64_t C = mb.g.nx * mb.g.nz;
  const double p_ref = mb.g.p_ref, p_ref_inv = mb.g.p_ref_inv, V = mb.g.volume_cell;
  const int bits = acc_bits(mb.sp.n);
  if (blockIdx.x == 0 && threadIdx.x == 0) take_water(mb);
  __syncwarp();
  const int64_t cells = (int64_t)gridDim.x * 8;
  for (int64_t c0 = (int64_t)blockIdx.x * 8; c0 < C; c0 += cells) {
    int64_t c = c0 + (threadIdx.x >> 2);
    const bool in = c < C, first = in && (threadIdx.x & 3) == 0;
    if (!in) c = C - 1;
    long long* const acc = mb.w.acc64 + ACC64_WORDS * c;
    double sum = acc_read64(acc, bits);
    const double x = mb.w.accx[c];
    if (x != 0.0) sum += x;   // NaN too
    const double dml = sum * 1.0E-18;
    __syncwarp();   // all lanes have read the sums
    if (first) {
      acc_clear64(acc);
      if (x != 0.0) mb.w.accx[c] = 0.0;
      delta_m_l[c] = dml;
    }
    if (grid_update)
      grid_cell_update_x4(gsf, gmp, aux, c, C, p_ref, p_ref_inv, dTh[c], drv[c], dml, V, in);
  }
}

// ---------------------------------------------------------------------------
// Mixed precision particle sub-step.  GB300 issues FP64 arithmetic, FP64
// compares and double<->float conversions on a pipe that is 64x narrower than
// the FP32 one, so this kernel keeps the FP64 pipe for the three state
// updates x += dx, z += dz, m_w += dm and does everything else in FP32 or in
// integer units:
//  * double -> float rounding (to nearest even) and float -> double are done
//    on the IEEE bit patterns with integer instructions (d2f_int / f2d_int);
//  * comparisons of non-negative doubles compare their bit patterns;
//  * the new cell index comes from the FP32 position with a certified margin
//    (1e-4 of a cell) around cell edges, inside which FP64 decides;
//  * the per-cell sums of dm * xi are exact integer sums (acc_add), which L2
//    executes, independent of their order.
// The Newton condensation and the drag update run in FP32 (lacmo_physics.cuh)
// with the FP64 Newton for SIPs near the critical radius.  water_removed takes
// the SIPs reaching the ground with FP64 atomics, in arbitrary order.
// Rare FP64 paths stay out of line (__noinline__) so that the common path
// issues no FP64 instruction, not even predicated off.
// removed SIP: only the relative position keeps its per-call division
__device__ __noinline__ void mixed_inactive_rel(double* rel, int64_t n, double dx, double dz,
                                                int64_t k, int i) {
  rel[k] = rel[k] / dx - (double)i;
  rel[n + k] = rel[n + k] / dz - (-1.0);
}
// near the critical radius: FP64 residual and Newton step
struct NewtonFP64 {
  const double *gsf, *gmp, *aux;
  int64_t C;
  double dt_sub;
  int sol, no_iter;
  unsigned long long* nfb;
};
// FAST: newton_fast (k_newton_fallback: 24 -> 16 us a launch, its latency); the
// particle kernel, which calls it for a rare SIP leaving the domain, keeps
// newton_full: the larger callee cost its main path 8% through the registers
template <bool FAST>
__device__ __noinline__ double mixed_newton_fp64(NewtonFP64 a, int32_t c, double mw, double ms) {
  const int64_t C = a.C;
  const double T_p = __ldg(a.gsf + c);   // the cell temperature
  CellAmb amb;
  amb.T = T_p; amb.p = __ldg(a.gsf + C + c); amb.S = __ldg(a.gsf + 6 * C + c);
  amb.e_s = __ldg(a.gsf + 7 * C + c); amb.K = __ldg(a.gmp + c);
  amb.D_v = __ldg(a.gmp + C + c); amb.L_v = __ldg(a.gmp + 2 * C + c);
  amb.sigw = __ldg(a.aux + c); amb.rhow = __ldg(a.aux + C + c);
  amb.lap0 = __ldg(a.aux + 2 * C + c); amb.lbp0 = __ldg(a.aux + 3 * C + c);
  amb.c1 = __ldg(a.aux + 4 * C + c); amb.c2 = __ldg(a.aux + 5 * C + c);
  atomicAdd(a.nfb, 1ull);
  if (FAST && ff_mass_ok(mw) && ff_mass_ok(ms))
    return newton_fast(a.sol, a.dt_sub, a.no_iter, mw, ms, cell_fast(a.sol, amb), 1.0) - mw;
  const double m_p = mw + ms;
  const double w_s = ms / m_p;
  const double rho64 = (a.sol == SOL_AS) ? density_AS_solution_rw(w_s, amb.rhow)
                                         : density_NaCl_solution(w_s, T_p);
  const double R64 = radius_from_mass(m_p, rho64);
  const double sig64 = (a.sol == SOL_AS) ? surface_tension_AS_sw(w_s, amb.sigw)
                                         : surface_tension_NaCl_sw(w_s, amb.sigw);
  return newton_full(a.sol, a.dt_sub, a.no_iter, mw, ms, w_s, R64, T_p, rho64, sig64, amb,
                     nullptr);
}
// the FP64 position update near or past a boundary: periodic x
// (integration.py:577-583), capped z (:585-589), and whether the SIP reached
// the ground (:606); bit 0 of the result: below z_min
struct EdgeIn { double x, z, dx, dz, x_max, z_cap, z_min; int wrap, cap; };
__device__ __noinline__ int mixed_edges(EdgeIn e, double* xo, double* zo) {
  double x = e.x, z = e.z;
  if (e.wrap) x = py_mod(x, e.x_max);
  if (e.cap) z = np_min(z, e.z_cap);
  *xo = x; *zo = z;
  return z <= e.z_min ? 1 : 0;
}
__device__ __noinline__ int mixed_floor_div(double x, double d) { return (int)floor(x / d); }
// SIP reaching the ground (integration.py:606-630)
struct GroundGeo {
  double* rel;
  double* water_removed;
  int64_t n;
  double x_min, z_min, dx, dz;
};
__device__ __noinline__ double mixed_remove(GroundGeo a, int64_t k, int i, int j, double x0,
                                            double z0, double xik, double mw) {
  atomicAdd(a.water_removed, xik * mw);   // FP64, any order
  const double rel_x = (x0 - a.x_min) / a.dx - (double)i;
  const double rel_z = (z0 - a.z_min) / a.dz - (double)j;
  a.rel[k] = rel_x / a.dx - (double)i;
  a.rel[a.n + k] = rel_z / a.dz - (-1.0);
  return a.z_min - 0.01 * a.dz;
}

// ---- bulk copies into shared memory (cp.async.bulk + mbarrier) ----
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared.b64 [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared.b64 _, [%0], %1;\n" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// global -> shared, completion counted in bytes on the mbarrier; the SIP
// state streams through once per sub-step (L2 evict-first policy) so that
// the per-cell records the kernel gathers stay in L2
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes,
                                         uint64_t* bar, uint64_t pol) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint"
      " [%0], [%1], %2, [%3], %4;\n" ::"r"(smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar)), "l"(pol)
      : "memory");
}
__device__ __forceinline__ uint64_t l2_evict_first_policy() {
  uint64_t pol;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;\n" : "=l"(pol));
  return pol;
}
__device__ __forceinline__ void prefetch_l1(const void* p) {
  asm volatile("prefetch.global.L1 [%0];\n" ::"l"(p));
}
// Mixed precision: the per-cell sums of dm * xi (FP32 products) are exact
// integer sums in units of 2^-4 fg, so their order does not matter and a
// step gives the same bits run to run and batched or not.  v 2^4 rounded to
// the nearest integer (halves away from zero) from the FP32 bits, without a
// conversion instruction; |v| up to 2^58 fg (a cell's per-sub-step total
// stays below 2^59 / 2^4 fg = 36 kg); beyond, the value is clamped and
// LACMO_FLAG_ACC_RANGE raised.
constexpr double ACC_UNIT = 0.0625;   // fg per integer unit
__device__ __forceinline__ long long fix_of(float v, uint32_t* flags) {
  const uint32_t b = __float_as_uint(v);
  const int e = (int)((b >> 23) & 0xffu);
  if (e == 0) return 0;   // zero or below 2^-126
  const uint64_t m = (uint64_t)((b & 0x7fffffu) | 0x800000u);
  const int sh = e - 146;   // v 2^4 = m 2^(e - 150 + 4)
  uint64_t mag;
  if (sh >= 35 || e == 0xff) {
    atomicOr(flags, LACMO_FLAG_ACC_RANGE);
    mag = 1ull << 58;
  } else if (sh >= 0) {
    mag = m << sh;
  } else if (sh > -26) {
    mag = (m + (1ull << (-sh - 1))) >> (-sh);
  } else {
    mag = 0;
  }
  return (b >> 31) ? -(long long)mag : (long long)mag;
}
__device__ __forceinline__ void acc_add(double* acc, int64_t c, float v, uint32_t* flags) {
  atomicAdd((unsigned long long*)(acc + c), (unsigned long long)fix_of(v, flags));
}

// an mbarrier wait never spins without bound: after this many polls (each
// try_wait suspends the thread for a while) the kernel gives up and raises
// LACMO_FLAG_SYNC_TIMEOUT
constexpr uint32_t MBAR_POLL_LIMIT = 1u << 22;

// Tiles of PM_TILE consecutive SIPs move HBM -> shared memory as bulk copies,
// one per attribute, issued by one thread two tiles ahead (three stages).
// Each attribute's slot has room for a window that starts at the 16-byte
// boundary below the tile's first element (the rows z and w start 8 bytes off
// a boundary when n is odd).  When a tile's data lands, every thread
// prefetches the cell record of its SIP in that tile into L1, one tile
// before it is used.  Tiles a bulk copy cannot take (the last ones of a
// member, or arrays not 16-byte aligned) are loaded by the threads.
#ifndef LACMO_PM_THREADS
#define LACMO_PM_THREADS 128
#endif
constexpr int PM_THREADS = LACMO_PM_THREADS;
constexpr int PM_TILE = PM_THREADS;
constexpr int PM_STAGES = 3;
enum { PF_X, PF_Z, PF_U, PF_W, PF_MW, PF_MS, PF_XI, PF_N };
struct PmStage {
  double f[PF_N][PM_TILE + 2];
  int32_t c[PM_TILE + 4];
};

template <bool PHYS>
struct PmTiles {
  // the rows z and w (second rows of pos and vel) start 8 bytes off a 16-byte
  // boundary when n is odd: their slots then hold the window from 8 bytes
  // below the tile's first element, and the data starts at slot index zoff
  int zoff;
  bool bulk;   // arrays aligned for bulk copies
  __device__ __forceinline__ void init(const PArgs& a) {
    uintptr_t al = (uintptr_t)a.pos | (uintptr_t)a.vel | (uintptr_t)a.cell;
    if (PHYS) al |= (uintptr_t)a.m_w | (uintptr_t)a.m_s | (uintptr_t)a.xi;
    bulk = al % 16 == 0;
    zoff = bulk ? (int)(a.n & 1) : 0;
  }
  // tile k0 by bulk copy: aligned arrays, and every window inside its array
  // (the window of a second row reaches 8 bytes past the tile's end)
  __device__ __forceinline__ bool by_bulk(const PArgs& a, int64_t k0) const {
    return bulk && k0 + PM_TILE + 2 <= a.n;
  }
  __device__ __forceinline__ void issue(const PArgs& a, int64_t k0, PmStage& s, uint64_t* bar,
                                        uint64_t pol) const {
    const uint32_t zb = PM_TILE * 8 + 16 * zoff;   // bytes of a second-row window
    mbar_expect_tx(bar, PM_TILE * 4 + (PHYS ? 5 : 2) * PM_TILE * 8 + 2 * zb);
    bulk_g2s(&s.f[PF_X][0], a.pos + k0, PM_TILE * 8, bar, pol);
    bulk_g2s(&s.f[PF_Z][0], a.pos + a.n + k0 - zoff, zb, bar, pol);
    bulk_g2s(&s.f[PF_U][0], a.vel + k0, PM_TILE * 8, bar, pol);
    bulk_g2s(&s.f[PF_W][0], a.vel + a.n + k0 - zoff, zb, bar, pol);
    if (PHYS) {
      bulk_g2s(&s.f[PF_MW][0], a.m_w + k0, PM_TILE * 8, bar, pol);
      bulk_g2s(&s.f[PF_MS][0], a.m_s + k0, PM_TILE * 8, bar, pol);
      bulk_g2s(&s.f[PF_XI][0], a.xi + k0, PM_TILE * 8, bar, pol);
    }
    bulk_g2s(&s.c[0], a.cell + k0, PM_TILE * 4, bar, pol);
  }
  // the slot of thread t's SIP in the stage
  __device__ __forceinline__ double get(const PmStage& s, int f, int t) const {
    return s.f[f][(f == PF_Z || f == PF_W) ? zoff + t : t];
  }
  // the threads' own loads of a tile (same slots)
  __device__ __forceinline__ void load(const PArgs& a, int64_t k, PmStage& s, int t) const {
    if (k >= a.n) return;
    s.f[PF_X][t] = __ldcs(a.pos + k);
    s.f[PF_Z][zoff + t] = __ldcs(a.pos + a.n + k);
    s.f[PF_U][t] = __ldcs(a.vel + k);
    s.f[PF_W][zoff + t] = __ldcs(a.vel + a.n + k);
    if (PHYS) {
      s.f[PF_MW][t] = __ldcs(a.m_w + k);
      s.f[PF_MS][t] = __ldcs(a.m_s + k);
      s.f[PF_XI][t] = __ldcs(a.xi + k);
    }
    s.c[t] = __ldcs(a.cell + k);
  }
};

// MINB: resident blocks per SM the register budget is set for (the
// TUNE_PARTICLE_BLOCKS knob picks the instance)
template <bool PHYS, int MINB>
__global__ void __launch_bounds__(PM_THREADS, MINB) k_particles_mixed(const __grid_constant__ PK x) {
  // the member's arguments, once per block in shared memory: threads read
  // them on use instead of holding some 60 registers of pointers and sizes
  __shared__ PArgs s_a;
  extern __shared__ __align__(128) unsigned char pm_smem[];
  PmStage* st = (PmStage*)pm_smem;
  __shared__ __align__(8) uint64_t s_bar[PM_STAGES];
  const int t = threadIdx.x;
  if (t == 0) {
    s_a = make_pargs(x.m.get(), x.c);
    for (int q = 0; q < PM_STAGES; ++q) mbar_init(&s_bar[q], 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
  }
  __syncthreads();
  const PArgs& a = s_a;
  const int C = (int)(a.nx * a.nz);
  const int nz = (int)a.nz;
  PmTiles<PHYS> tl;
  tl.init(a);
  // SIP indices fit in 32 bits (n < 2^31)
  const int ntiles = (int)((a.n + PM_TILE - 1) / PM_TILE);
  const int G = gridDim.x;
  const int first = blockIdx.x;
  const int my_tiles = first < ntiles ? (ntiles - first + G - 1) / G : 0;
  // prologue: tiles 0 and 1 of this block in flight
  if (t == 0) {
    const uint64_t pol = l2_evict_first_policy();
    for (int i = 0; i < 2 && i < my_tiles; ++i) {
      const int k0 = (first + i * G) * PM_TILE;
      if (tl.by_bulk(a, k0)) tl.issue(a, k0, st[i], &s_bar[i], pol);
    }
  }
  bool tout = false;   // an mbarrier wait of this thread ran out of polls
  int i = 0;
  for (; i < my_tiles; ++i) {
    const int k0 = (first + i * G) * PM_TILE;
    const int sg = i % PM_STAGES;
    // every thread is done with tile i - 1's stage; all stop together when a
    // wait ran out
    if (i > 0 && __syncthreads_or(tout)) break;
    if (t == 0 && i + 2 < my_tiles) {
      const int k2 = (first + (i + 2) * G) * PM_TILE;
      const int s2 = (i + 2) % PM_STAGES;
      if (tl.by_bulk(a, k2)) {
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        tl.issue(a, k2, st[s2], &s_bar[s2], l2_evict_first_policy());
      }
    }
    // this tile's data (the first tile's, else waited for one tile ago), and
    // the next tile's: its cell records go to L1 now
    for (int w = (i == 0 ? 0 : 1); w <= 1; ++w) {
      const int iw = i + w;
      if (iw >= my_tiles) break;
      const int kw = (first + iw * G) * PM_TILE;
      if (!tl.by_bulk(a, kw)) continue;
      const int sw = iw % PM_STAGES;
      const uint32_t parity = (uint32_t)((iw / PM_STAGES) & 1);
      uint32_t polls = 0;
      while (!mbar_try_wait(&s_bar[sw], parity)) {
        if (++polls >= MBAR_POLL_LIMIT) { tout = true; break; }
      }
      if (PHYS && w == 1 && !tout) {
        const int32_t cn = st[sw].c[t];
        if (cn >= 0) prefetch_l1(a.crec + CELL_REC * (int64_t)cn);
      }
    }
    if (tout) continue;   // this tile's data cannot be trusted
    PmStage& S = st[sg];
    const int k = k0 + t;
    if (!tl.by_bulk(a, k0)) tl.load(a, k, S, t);
    if (k >= a.n) continue;
    const int32_t c = S.c[t];
    if (c < 0) {
      const int i_ = -1 - c;
      if (a.write_Tp) a.T_p[k] = __ldg(a.gsf + (int64_t)i_ * nz + nz - 1);
      mixed_inactive_rel(a.rel, a.n, a.dx, a.dz, k, i_);
      continue;
    }
    if (a.write_Tp) a.T_p[k] = __ldg(a.gsf + c);
    float un, wn2, d = 0.0f, xf, zf;
    int fb_slot = -1;   // queue slot of a SIP whose Newton repeats in FP64
    const float4* rec = a.crec + CELL_REC * (int64_t)c;
    if (PHYS) {
      const float4 q0 = __ldg(rec), q1 = __ldg(rec + 1);
      CellAmbF af;
      af.T = q0.x; af.S_m1 = q0.y; af.sigw = q0.z; af.rhow = q0.w;
      af.lap0 = q1.x; af.lbp0 = q1.y; af.c1 = q1.z; af.c2 = q1.w;
      const float msf = d2f_int(tl.get(S, PF_MS, t)), mwf = d2f_int(tl.get(S, PF_MW, t));
      const float mpf = mwf + msf;
      const float wsf = msf * f_rcp(mpf);
      const float rho = (a.sol == SOL_AS)
                            ? af.rhow * ((((float)LC_PAR_RHO_AS_0 * wsf + (float)LC_PAR_RHO_AS_1) *
                                              wsf + (float)LC_PAR_RHO_AS_2) * wsf +
                                         (float)LC_PAR_RHO_AS_3)
                            : (float)LC_PAR_SOL_DENS_NACL_0 + (float)LC_PAR_SOL_DENS_NACL_1 * wsf +
                                  (float)LC_PAR_SOL_DENS_NACL_2 * af.T +
                                  (float)LC_PAR_SOL_DENS_NACL_3 * wsf * wsf +
                                  (float)LC_PAR_SOL_DENS_NACL_4 * wsf * af.T +
                                  (float)LC_PAR_SOL_DENS_NACL_5 * af.T * af.T;
      const float R = f_cbrt((float)LC_FOUR_PI_OVER_THREE_INV * mpf * f_rcp(rho));
      const float sig = af.sigw * (1.0f + (a.sol == SOL_AS ? (float)LC_PAR_SIGMA_AS
                                                            : (float)LC_PAR_SIGMA_NACL) *
                                               wsf * f_rcp(1.f - wsf));
      // efflorescence floor m_s (1/0.78 - 1) as an increment, in FP32
      const float d_effl = msf * (float)(LC_W_S_MAX_AS_INV - 1.0) - mwf;
      const bool ok = newton_mixed_f(a.sol, a.dt_subf, a.no_iter, mwf, msf, wsf, R, af.T, rho,
                                     sig, af, d_effl, &d);
      if (ok) {
        // per-cell exact sum of dm * xi (executed by L2)
        acc_add(a.acc, c, d * d2f_int(tl.get(S, PF_XI, t)), a.flags);
      } else {
        // near the critical radius the Newton repeats in FP64, in full warps
        // in k_newton_fallback: queue the SIP with its mass before the
        // sub-step; drag and motion go on with the FP32 increment
        fb_slot = atomicAdd(a.fb_count, 1);
        a.fb_id[fb_slot] = (int32_t)k;
        a.fb_c[fb_slot] = c;
        a.fb_mw[fb_slot] = tl.get(S, PF_MW, t);
      }
      // drag (integration.py:699-718) in FP32 with the ammonium-sulfate radius
      const float mpn = (mwf + d) + msf;
      const float wn = msf * f_rcp(mpn);
      const float rhon = af.rhow * ((((float)LC_PAR_RHO_AS_0 * wn + (float)LC_PAR_RHO_AS_1) * wn +
                                     (float)LC_PAR_RHO_AS_2) * wn + (float)LC_PAR_RHO_AS_3);
      const float Rn = f_cbrt((float)LC_FOUR_PI_OVER_THREE_INV * mpn * f_rcp(rhon));
      const float4 cij = __ldg(rec + 6);   // (i, j, j == 0, j == nz - 1)
      xf = d2f_int(tl.get(S, PF_X, t));
      zf = d2f_int(tl.get(S, PF_Z, t));
      const float rxf = (xf - a.x_minf) * a.inv_dxf - cij.x;
      const float rzf = (zf - a.z_minf) * a.inv_dzf - cij.y;
      float uf, wf;
      interp_wind(__ldg(rec + 3), __ldg(rec + 4), __ldg(rec + 5), cij.z != 0.0f, cij.w != 0.0f,
                  rxf, rzf, uf, wf);
      const float2 q2 = __ldg((const float2*)(rec + 2));
      const float mu_f = q2.x, rho_f = q2.y;
      const float uo = d2f_int(tl.get(S, PF_U, t)), wo = d2f_int(tl.get(S, PF_W, t));
      const float d0 = uf - uo, d1 = wf - wo;
      const float vel_dev = f_sqrt(d0 * d0 + d1 * d1);
      const float inv_mu = f_rcp(mu_f);
      const float Re_p = 2.0E-6f * rho_f * Rn * vel_dev * inv_mu;
      float k_dt = 4.5E12f * a.dt_subf * mu_f * f_rcp(rhon * Rn * Rn);
      if (Re_p > 0.5f) {
        if (Re_p < 1000.0f) k_dt *= (1.f + 0.15f * f_pow(Re_p, 0.687f));
        else k_dt *= 0.0183333333333f * Re_p;
      }
      const float inv = f_rcp(1.0f + k_dt);
      un = (uo + k_dt * uf) * inv;
      wn2 = (wo + k_dt * wf - a.dtg_f) * inv;
    } else {
      // the half-step move of integration.py:1474-1481: positions only
      un = d2f_int(tl.get(S, PF_U, t));
      wn2 = d2f_int(tl.get(S, PF_W, t));
      xf = d2f_int(tl.get(S, PF_X, t));
      zf = d2f_int(tl.get(S, PF_Z, t));
    }
    // position (integration.py:552-630)
    const double x0 = tl.get(S, PF_X, t), z0 = tl.get(S, PF_Z, t);
    const float xf0 = xf, zf0 = zf;
    const float dxf = a.dt_posf * un, dzf = a.dt_posf * wn2;
    double xn = x0 + f2d_int(dxf);
    double zn = z0 + f2d_int(dzf);
    const float xnf = xf0 + dxf, znf = zf0 + dzf;
    double u = f2d_int(un), w = f2d_int(wn2);
    // periodic x / capped z / ground: exact FP64 only when near or past a
    // boundary
    const int wrap = !(xnf > 1e-3f && xnf < a.x_maxf - 1e-3f);
    const int cap = !(znf < a.z_capf - 1e-3f);
    const int low = !(znf > a.z_minf + 1e-3f);
    int edge = 0;
    if (wrap | cap | low)
      edge = mixed_edges(EdgeIn{xn, zn, a.dx, a.dz, a.x_max, a.z_cap, a.z_min, wrap, cap}, &xn,
                         &zn);
    int32_t newc;
    bool removed = false;
    if (low && (edge & 1)) {
      const int i_ = c / nz, j_ = c - i_ * nz;
      const double xik = PHYS ? tl.get(S, PF_XI, t) : a.xi[k];
      double mw = PHYS ? tl.get(S, PF_MW, t) + f2d_int(d) : a.m_w[k];
      if (PHYS && fb_slot >= 0) {
        // a queued SIP leaving the domain: its FP64 Newton here, for the
        // water it takes along
        const double mw0 = tl.get(S, PF_MW, t);
        const double dm = mixed_newton_fp64<false>(NewtonFP64{a.gsf, a.gmp, mixed_aux((double*)a.aux, C), (int64_t)C, a.dt_sub,
                                                       a.sol, a.no_iter, a.nfb},
                                            c, mw0, tl.get(S, PF_MS, t));
        mw = mw0 + dm;
        acc_add(a.acc, c, d2f_int(dm) * d2f_int(xik), a.flags);
        a.fb_id[fb_slot] = -1;
      }
      if (PHYS) __stcs(a.m_w + k, mw);
      zn = mixed_remove(GroundGeo{a.rel, a.water_removed, a.n, a.x_min, a.z_min, a.dx, a.dz}, k,
                        i_, j_, x0, z0, xik, mw);
      u = 0.0; w = 0.0;
      removed = true;
      newc = (int32_t)(-1 - i_);
    } else {
      // the new cell from the FP32 position, FP64 when within 1e-4 of an edge
      const float px = wrap ? d2f_int(xn) : xnf, pz = cap ? d2f_int(zn) : znf;
      const float qx = px * a.inv_dxf, qz = pz * a.inv_dzf;
      int ci = __float2int_rd(qx), cj = __float2int_rd(qz);
      const float fx = qx - floorf(qx), fz = qz - floorf(qz);
      if (!(fx > 1e-4f && fx < 0.9999f)) ci = mixed_floor_div(xn, a.dx);
      if (!(fz > 1e-4f && fz < 0.9999f)) cj = mixed_floor_div(zn, a.dz);
      if (ci >= a.nx || ci < 0 || cj >= nz || cj < 0) {
        atomicOr(a.flags, LACMO_FLAG_CELL_CLAMPED);
        ci = ci < 0 ? 0 : (ci >= a.nx ? (int)a.nx - 1 : ci);
        cj = cj < 0 ? 0 : (cj >= nz ? nz - 1 : cj);
      }
      newc = (int32_t)(ci * nz + cj);
      if (a.hist) a.rank[k] = rank_in(a.counts, newc);
      if (PHYS) __stcs(a.m_w + k, tl.get(S, PF_MW, t) + f2d_int(d));
    }
    // streaming stores (evict first)
    __stcs(a.pos + k, xn); __stcs(a.pos + a.n + k, zn);
    if (PHYS || removed) { __stcs(a.vel + k, u); __stcs(a.vel + a.n + k, w); }
    __stcs(a.cell + k, newc);
  }
  if (__syncthreads_or(tout)) {
    // a wait ran out: flag it, and wait (again bounded) for the copies this
    // block may still have in flight before the block's shared memory goes
    if (t == 0) {
      atomicOr(a.flags, LACMO_FLAG_SYNC_TIMEOUT);
      for (int j = i; j < i + 2 && j < my_tiles; ++j) {
        if (!tl.by_bulk(a, (first + j * G) * PM_TILE)) continue;
        const int sj = (int)(j % PM_STAGES);
        for (uint32_t p = 0; p < MBAR_POLL_LIMIT; ++p)
          if (mbar_try_wait(&s_bar[sj], (uint32_t)((j / PM_STAGES) & 1))) break;
      }
    }
  }
}
constexpr size_t PM_SMEM = (size_t)PM_STAGES * sizeof(PmStage);

// The FP64 Newton of the SIPs a mixed sub-step queued (near the critical
// radius), one SIP per thread: the mass and the per-cell sum as the inline
// FP64 path gives them; the last block empties the queue.
__global__ void __launch_bounds__(128) k_newton_fallback(const __grid_constant__ PK x) {
  __shared__ PArgs s_a;
  if (threadIdx.x == 0) s_a = make_pargs(x.m.get(), x.c);
  __syncthreads();
  const PArgs& a = s_a;
  const int cnt = *(volatile int32_t*)a.fb_count;
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < cnt; q += gridDim.x * blockDim.x) {
    const int32_t k = a.fb_id[q];
    if (k < 0) continue;   // handled where it left the domain
    const int32_t c = a.fb_c[q];
    const double mw0 = a.fb_mw[q];
    const double dm = mixed_newton_fp64<true>(NewtonFP64{a.gsf, a.gmp,
                                                         mixed_aux((double*)a.aux, a.nx * a.nz),
                                                         a.nx * a.nz, a.dt_sub,
                                                   a.sol, a.no_iter, a.nfb},
                                        c, mw0, a.m_s[k]);
    a.m_w[k] = mw0 + dm;
    acc_add(a.acc, c, d2f_int(dm) * d2f_int(a.xi[k]), a.flags);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(a.fb_done, 1) == (int)gridDim.x - 1) {
      *a.fb_count = 0;
      *a.fb_done = 0;
    }
  }
}

// Mixed precision: the grid update of one cell (integration.py:402-484,
// update_material_properties :359-400) in FP64 with exp/log in place of pow,
// pow(x, y) = exp(y log x) to a few 1e-15 relative, and the chained powers of
// the Exner function folded into one log; then the per-cell Newton terms
// (FP64 and the FP32 table) from the same values.
__device__ __forceinline__ void grid_cell_update_mixed(double* gsf, double* gmp, double* aux,
                                                       int64_t c, int64_t C, double p_ref,
                                                       double p_ref_inv, double dTh, double drv,
                                                       double dml, double V) {
  double Th = gsf[2 * C + c];
  const double rho_d = gsf[3 * C + c];
  double r_v = gsf[4 * C + c];
  const double mdi = gsf[8 * C + c];
  const double L_v0 = gmp[2 * C + c];
  Th += dTh;
  r_v += drv - dml * mdi;
  const double ToT = exp(LC_KAPPA_FACTOR2 * log(p_ref_inv * LC_R_D * rho_d * Th));
  Th += ToT * (L_v0 * dml) / (LC_C_PD * rho_d * V * (1.0 + r_v * LC_HEAT_FACTOR_R_V));
  const double L2 = log(rho_d * Th * LC_R_D * p_ref_inv);
  const double pdr = exp(LC_KAPPA_FACTOR * L2);
  const double T = Th * exp((LC_KAPPA_FACTOR * LC_KAPPA_AIR_DRY) * L2);
  const double p = pdr * p_ref * (1 + r_v / LC_EPSILON_GC);
  const double e_s = 2.53E11 * exp(-5420.0 / T);
  const double S = rho_d * r_v * T * LC_R_V / e_s;
  const double K = 4.1868E-3 * (5.69 + 0.017 * (T - 273.15));
  const double D_v = 4.01218E-5 * exp(1.94 * log(T)) / p;
  const double L_v = 1.0E3 * (2500.82 - 2.358 * (T - 273.0));
  const double tau = 1 - T / 647.096;
  const double sigw = 0.2358 * exp(1.256 * log(tau)) * (1 - 0.625 * tau);
  const double mu = 1.458E-6 * T * sqrt(T) / (T + 110.4);
  const double rho_f = rho_d * (1.0 + r_v);
  gsf[c] = T; gsf[C + c] = p; gsf[2 * C + c] = Th; gsf[4 * C + c] = r_v;
  gsf[6 * C + c] = S; gsf[7 * C + c] = e_s;
  gmp[c] = K; gmp[C + c] = D_v; gmp[2 * C + c] = L_v; gmp[3 * C + c] = sigw;
  gmp[4 * C + c] = LC_C_PD * (1 + 0.897 * r_v); gmp[5 * C + c] = mu; gmp[6 * C + c] = rho_f;
  // the terms of make_cell_amb (lacmo_physics.cuh) from the values above
  const double rhow = density_water(T);
  const double lap0 = (LC_C_ALPHA_1 + LC_C_ALPHA_2 * (T - LC_T_ALPHA_0)) * K / p;
  const double lbp0 = LC_C_BETA_1 * (1.0 + LC_C_BETA_2 * (T - LC_T_ALPHA_0)) * D_v;
  const double c1 = L_v * L_v / (LC_R_V * K * T * T);
  const double c2 = LC_R_V * T / (D_v * e_s);
  double* const am = mixed_aux(aux, C);
  am[c] = sigw; am[C + c] = rhow; am[2 * C + c] = lap0; am[3 * C + c] = lbp0;
  am[4 * C + c] = c1; am[5 * C + c] = c2;
  float4* af = cell_records(aux, C) + CELL_REC * c;
  af[0] = make_float4((float)T, (float)(S - 1.0), (float)sigw, (float)rhow);
  af[1] = make_float4((float)lap0, (float)lbp0, (float)c1, (float)c2);
  af[2] = make_float4((float)mu, (float)rho_f, 0.0f, 0.0f);
}

// mixed precision: the grid sub-step from the per-cell exact sums (then zeroed)
__global__ void k_grid_acc(const __grid_constant__ MRef mr) {
  const Member& mb = mr.get();
  double *acc = mb.w.div, *delta_m_l = mb.g.delta_m_l, *gsf = mb.g.scalar_fields,
         *gmp = mb.g.mat_prop, *aux = mb.w.aux;
  const double *dTh = mb.w.dTh, *drv = mb.w.drv;
  const int64_t C = mb.g.nx * mb.g.nz;
  const double p_ref = mb.g.p_ref, p_ref_inv = mb.g.p_ref_inv, V = mb.g.volume_cell;
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < C;
       c += (int64_t)gridDim.x * blockDim.x) {
    long long* acc_i = (long long*)acc;
    const double dml = (double)acc_i[c] * ACC_UNIT * 1.0E-18;
    acc_i[c] = 0;
    delta_m_l[c] = dml;
    grid_cell_update_mixed(gsf, gmp, aux, c, C, p_ref, p_ref_inv, dTh[c], drv[c], dml, V);
  }
}

__global__ void k_grid_only(double* gsf, double* gmp, double* aux, const double* dTh,
                            const double* drv, const double* dml, int64_t C, double p_ref,
                            double p_ref_inv, double V) {
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < C;
       c += (int64_t)gridDim.x * blockDim.x) {
    grid_cell_update(gsf, gmp, aux, c, C, p_ref, p_ref_inv, dTh[c], drv[c], dml[c], V);
  }
}

// grid.py:370-412 (ascending-ID fold per cell)
__global__ void __launch_bounds__(256) k_r_l(const __grid_constant__ MRef mr) {
  const Member& mb = mr.get();
  const int32_t* __restrict__ start = mb.w.start;
  const int32_t* __restrict__ perm = mb.w.perm;
  const double* __restrict__ m_w = mb.sp.m_w;
  const double* __restrict__ xi = mb.sp.xi;
  double* gsf = mb.g.scalar_fields;
  const int64_t C = mb.g.nx * mb.g.nz;
  const int lane = threadIdx.x & 31;
  for (int64_t c = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; c < C;
       c += ((int64_t)gridDim.x * blockDim.x) >> 5) {
    const int32_t b = start[c], e = start[c + 1];
    double acc = 0.0;
    for (int32_t base = b; base < e; base += 32) {
      const int32_t idx = base + lane;
      double v = 0.0;
      if (idx < e) { int32_t id = perm[idx]; v = m_w[id] * xi[id]; }
      const int m = (e - base) < 32 ? (e - base) : 32;
      for (int q = 0; q < m; ++q) acc += __shfl_sync(0xffffffffu, v, q);
    }
    if (lane == 0) gsf[5 * C + c] = acc * (1.0E-18 * gsf[8 * C + c]);
  }
}

// ---------------------------------------------------------------------------
// integration.py:80-148 limiter and face flux (Hundsdorfer et al. 1995)
__device__ __forceinline__ double limiter_arg(double a0, double a1, double a2) {
  const double r = (fabs(a1 - a2) > 1.0E-8 * fabs(a0 - a1)) ? (a0 - a1) / (a1 - a2)
                                                             : (a0 - a1) * 1.0E8 * np_sign(a1 - a2);
  const double K = __dmul_rn(1.0 + 2.0 * r, LC_ONE_THIRD);
  return np_max(0.0, fmin(2.0 * r, fmin(K, 2.0)));
}
// the field at a face, from the limiter of the upwind side only
__device__ __forceinline__ double face_value(double u, double am2, double am1, double a0,
                                             double ap1) {
  const bool pos = u >= 0.0;
  const double o = pos ? a0 : am1, p = pos ? am1 : a0, q = pos ? am2 : ap1;
  return __fma_rn(0.5 * limiter_arg(o, p, q), p - q, p);
}
// i in [-2, N + 1], wrapped (bc 0) or clamped
__device__ __forceinline__ int bc_idx(int i, int N, int bc) {
  if (bc == 0) return N == 1 ? 0 : (i < 0 ? i + N : (i >= N ? i - N : i));
  return i < 0 ? 0 : (i > N - 1 ? N - 1 : i);
}
// integration.py:150-287, divergence of field * flux in cell (i, j): the part of
// the faces across x (dir 0) or z (dir 1).  Roundings are written out, and fuse
// forms the difference of the two fluxes with one (r_v across x): the mixed path
// rounds cell terms to FP32, where an increment's last bit shows.
__device__ __forceinline__ double divergence_part(const double* f, const double* flux, int nx,
                                                  int nz, int i, int j, int dir, double d, int bc,
                                                  bool fuse) {
  const int N = dir ? nz : nx, at = dir ? j : i;
  const int64_t step = dir ? 1 : nz, fstep = dir ? 1 : nz + 1;
  const double* const g = f + (dir ? (int64_t)i * nz : j);
  const double* const u = flux + (dir ? (int64_t)(nx + 1) * (nz + 1) : 0) + (int64_t)i * (nz + 1) + j;
  double v[5];
#pragma unroll
  for (int e = 0; e < 5; ++e) v[e] = g[bc_idx(at + e - 2, N, bc) * step];
  const double u0 = u[0], u1 = u[fstep];
  const double f0 = face_value(u0, v[0], v[1], v[2], v[3]);
  const double f1 = face_value(u1, v[1], v[2], v[3], v[4]);
  double F0 = __dmul_rn(u0, f0), F1 = __dmul_rn(u1, f1);
  if (bc == 1 && at == 0) F0 = 0.0;
  if (bc == 1 && at + 1 == N) F1 = 0.0;
  if (fuse) return __fma_rn(u1, f1, -F0) / d;
  return __dsub_rn(F1, F0) / d;
}

__global__ void k_divergence(const double* f, const double* flux, int64_t nx, int64_t nz, double dx,
                             double dz, int bcx, int bcz, double* out) {
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < nx * nz;
       c += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = c / nz, j = c - i * nz;
    out[c] = divergence_part(f, flux, (int)nx, (int)nz, (int)i, (int)j, 0, dx, bcx, false) +
             divergence_part(f, flux, (int)nx, (int)nz, (int)i, (int)j, 1, dz, bcz, false);
  }
}

// integration.py:325-354; the column sum runs over x in order like NumPy's
// axis-0 reduction of a C-ordered array
__global__ void k_relaxation(const double* f, int64_t nx, int64_t nz, const double* prof,
                             const double* trel, double dt, double* out) {
  for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < nz;
       j += (int64_t)gridDim.x * blockDim.x) {
    double s = f[j];
    for (int64_t i = 1; i < nx; ++i) s += f[i * nz + j];
    out[j] = dt * (prof[j] - s / (double)nx) / trel[j];
  }
}

// both relaxation terms of a sub-step in one launch: r_v into out[0:nz],
// Theta into out[nz:2nz] (integration.py:325-354)
__global__ void k_relaxation2(const __grid_constant__ MRef mr, const double* prof_rv,
                              const double* prof_th, const double* trel, double dt) {
  const Member& mb = mr.get();
  const double* gsf = mb.g.scalar_fields;
  const int64_t nx = mb.g.nx, nz = mb.g.nz;
  double* out = mb.w.relax;
  if (mb.prof_rv) { prof_rv = mb.prof_rv; prof_th = mb.prof_th; trel = mb.t_relax; }
  const int64_t C = nx * nz;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < 2 * nz;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t j = t < nz ? t : t - nz;
    const double* f = gsf + (t < nz ? 4 : 2) * C;
    const double* prof = t < nz ? prof_rv : prof_th;
    double s = f[j];
#pragma unroll 8
    for (int64_t i = 1; i < nx; ++i) s += f[i * nz + j];
    out[t] = dt * (prof[j] - s / (double)nx) / trel[j];
  }
}

// integration.py:1483-1508 (factor 1) and 1536-1561 (factor 2, minus the
// previous increment): advective + relaxation increments per sub-step.  Bound
// by the chain of FP64 operations of a face (and, with many members, by the FP64
// pipe): four lanes per cell, r_v and Theta across x and across z, two faces each
// (5625 cells: 21.0 us with one thread per cell and both limiters of every
// face, 5.9 us now; 64 members of 5625 cells: 303 and 163 us).
__global__ void k_advection(const __grid_constant__ MRef mr, double dt_sub, int relax_on,
                            int second) {
  const Member& mb = mr.get();
  const double *gsf = mb.g.scalar_fields, *flux = mb.g.mass_flux_air_dry, *relax = mb.w.relax;
  const int nx = (int)mb.g.nx, nz = (int)mb.g.nz;
  const double dx = mb.g.dx, dz = mb.g.dz;
  const int64_t C = (int64_t)nx * nz;
  const int role = threadIdx.x & 3, th = role & 1, dir = role >> 1;
  double* const out = th ? mb.w.dTh : mb.w.drv;
  const int64_t cells = (int64_t)gridDim.x * blockDim.x >> 2;
  for (int64_t c0 = (int64_t)blockIdx.x * blockDim.x >> 2; c0 < C; c0 += cells) {
    int64_t c = c0 + (threadIdx.x >> 2);
    const bool in = c < C;
    if (!in) c = C - 1;
    const int i = (int)(c / nz), j = (int)(c - (int64_t)i * nz);
    const double part = divergence_part(gsf + (th ? 2 : 4) * C, flux, nx, nz, i, j, dir,
                                        dir ? dz : dx, dir, !dir && !th);
    const double div = part + __shfl_xor_sync(0xffffffffu, part, 2);
    if (dir || !in) continue;
    const double rdi = gsf[9 * C + c];
    double a;
    const double w = -dt_sub * div, w2 = -2.0 * dt_sub * div;
    if (!second) {
      a = __dmul_rn(w, rdi);
      if (relax_on) a = __dadd_rn(a, relax[th * nz + j]);
    } else {
      a = __fma_rn(w2, rdi, -out[c]);
      if (relax_on) a = __fma_rn(2., relax[th * nz + j], a);
    }
    out[c] = a;
  }
}

// ---------------------------------------------------------------------------
// elementwise microphysics (unit parity entry points)
__global__ void k_mass_rate(int sol, int64_t n, InPtrs in, double* g, double* dg) {
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n;
       k += (int64_t)gridDim.x * blockDim.x) {
    CellAmb a = make_cell_amb(in.p[6][k], in.p[7][k], in.p[8][k], in.p[9][k], in.p[10][k], in.p[11][k], in.p[12][k]);
    a.sigw = surface_tension_water(in.p[4][k]);
    a.rhow = density_water(in.p[4][k]);
    mass_rate_and_derivative(sol, in.p[0][k], in.p[1][k], in.p[2][k], in.p[3][k], in.p[4][k], in.p[5][k],
                             in.p[13][k], a, g[k], dg[k]);
  }
}
__global__ void k_newton(int sol, int64_t n, double dt_sub, int no_iter, InPtrs in, double* dm,
                         double* g0) {
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n;
       k += (int64_t)gridDim.x * blockDim.x) {
    CellAmb a = make_cell_amb(in.p[6][k], in.p[7][k], in.p[8][k], in.p[9][k], in.p[10][k], in.p[11][k], in.p[12][k]);
    a.sigw = surface_tension_water(in.p[4][k]);
    a.rhow = density_water(in.p[4][k]);
    dm[k] = newton_full(sol, dt_sub, no_iter, in.p[0][k], in.p[1][k], in.p[2][k], in.p[3][k], in.p[4][k],
                        in.p[5][k], in.p[13][k], a, g0 + k);
  }
}
__global__ void k_interp(const int32_t* cell, const double* rel, const double* gvp, int64_t n,
                         int64_t nx, int64_t nz, double* out) {
  const GridVel gv{gvp, nx, nz};
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n;
       k += (int64_t)gridDim.x * blockDim.x) {
    int32_t c = cell[k];
    double u = 0.0, v = 0.0;
    if (c >= 0) {
      int64_t i = c / nz, j = c - (c / nz) * nz;
      gv.interp(i, j, rel[k], rel[n + k], u, v);
    }
    out[k] = u; out[n + k] = v;
  }
}

// ---------------------------------------------------------------------------
cudaError_t launch_cells_import(const int64_t* cells, const uint8_t* act, int32_t* cell, int64_t n,
                                int64_t nx, int64_t nz, cudaStream_t s) {
  (void)nx;
  k_cells_import<<<nblocks(n, 256), 256, 0, s>>>(cells, act, cell, n, nz); note_launches(1);
  return cudaGetLastError();
}
cudaError_t launch_cells_export(const int32_t* cell, const double* pos, double* rel, int64_t* cells,
                                uint8_t* act, int64_t n, int64_t nx, int64_t nz, double x_min,
                                double z_min, double dx, double dz, cudaStream_t s) {
  (void)nx;
  k_cells_export<<<nblocks(n, 256), 256, 0, s>>>(cell, pos, rel, cells, act, n, nz, x_min, z_min,
                                                 dx, dz); note_launches(1);
  return cudaGetLastError();
}
static inline dim3 grid2(int64_t per_member, int t, int M, int cap = 152 * 32) {
  return dim3((unsigned)nblocks(per_member, t, cap), (unsigned)M);
}
static PCall pcall(const lacmo_params_t& p, double dt_sub, double dt_pos, bool write_Tp,
                   bool hist) {
  PCall c;
  c.dt_sub = dt_sub; c.dt_pos = dt_pos; c.g_set = p.g_set;
  c.no_iter = p.no_iter_impl_mass; c.sol = p.solute; c.write_Tp = write_Tp ? 1 : 0;
  c.hist = hist ? 1 : 0;
  c.dt_subf = (float)dt_sub; c.dtg_f = (float)(dt_sub * p.g_set); c.dt_posf = (float)dt_pos;
  return c;
}
cudaError_t launch_cell_aux(const Bt& B, cudaStream_t s) {
  k_cell_aux<<<grid2(B.nx * B.nz, 32, B.M), 32, 0, s>>>(B.ref()); note_launches(1);
  // the wind parts of the cell records too, for sub-steps run before a full step
  k_wind_table<<<grid2(B.nx * B.nz, 256, B.M), 256, 0, s>>>(B.ref()); note_launches(1);
  return launch_records64(B, false, s);
}
cudaError_t launch_records64(const Bt& B, bool known, cudaStream_t s) {
  k_records64<<<grid2(B.nx * B.nz, 32, B.M), 32, 0, s>>>(B.ref(), known ? 1 : 0); note_launches(1);
  return cudaGetLastError();
}
cudaError_t launch_clear_acc64(const Bt& B, cudaStream_t s) {
  k_clear_acc64<<<grid2(B.nx * B.nz, 128, B.M), 128, 0, s>>>(B.ref()); note_launches(1);
  return cudaGetLastError();
}
__global__ void k_set_i64(int64_t* p, int64_t v) { *p = v; }
cudaError_t launch_set_i64(int64_t* p, int64_t v, cudaStream_t s) {
  k_set_i64<<<1, 1, 0, s>>>(p, v); note_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_histogram(const Bt& B, cudaStream_t s) {
  k_histogram<<<grid2(B.n_max, 256, B.M), 256, 0, s>>>(B.ref()); note_launches(1);
  return cudaGetLastError();
}
// the binning left empty (k_scan over counts left at zero) until the next one
cudaError_t launch_empty_bin(const Bt& B, cudaStream_t s) {
  k_scan<<<dim3(1, B.M), 1024, 0, s>>>(B.ref()); note_launches(1);
  return cudaGetLastError();
}
cudaError_t launch_bin(const Bt& B, cudaStream_t s) {
  const int64_t C = B.nx * B.nz;
  k_scan<<<dim3(1, B.M), 1024, 0, s>>>(B.ref()); note_launches(1);
  k_scatter<<<grid2(B.n_max, 256, B.M), 256, 0, s>>>(B.ref()); note_launches(1);
  k_order<<<grid2(C * 32, 256, B.M, 152 * tune_value(TUNE_ORDER_CTAS)), 256, 0, s>>>(B.ref());
  note_launches(1);
  return cudaGetLastError();
}
cudaError_t launch_move(const Bt& B, double dt_pos, bool hist, cudaStream_t s) {
  lacmo_params_t p = {};
  PK x{B.ref(), pcall(p, 0.0, dt_pos, false, hist)};
  k_particles<false, false><<<grid2(B.n_max, 128, B.M, 152 * 16), 128, 0, s>>>(x); note_launches(1);
  return cudaGetLastError();
}
// No more blocks than are resident at once: a block's queue holds its place until
// the few SIPs in it are done, some 15 us (360,000 SIPs: 128 us a launch with up to
// 2432 blocks, 114 us with the 608 that are resident; 545,000 SIPs, 1.3% of them
// large drops: 198 and 153 us).  States that fill the GPU more than once over
// are bound by the FP64 pipe and take FULL (the two above: 107 and 144 us); smaller
// ones wait for one SIP's chain, which FULL lengthens (1920 SIPs: 23.6 us without,
// 23.9 us with it).  The queue's second pass doing only what is left of a SIP
// took all of these to 95, 135 and 19 us.
cudaError_t launch_particles(const Bt& B, const lacmo_params_t& p, double dt_sub,
                             double dt_sub_pos, bool write_Tp, bool hist, cudaStream_t s) {
  PK x{B.ref(), pcall(p, dt_sub, dt_sub_pos, write_Tp, hist)};
  static std::atomic<int> cached[64];
  int res = 0;
  cudaError_t e = resident_blocks((const void*)k_particles<true, true>, 128, 0, cached, &res);
  if (e != cudaSuccess) return e;
  const int cap = res / B.M > 0 ? res / B.M : 1;
  const dim3 grid = grid2(B.n_max, 128, B.M, cap);
  if (B.n_max > 128 * (int64_t)cap) k_particles<true, true><<<grid, 128, 0, s>>>(x);
  else k_particles<true, false><<<grid, 128, 0, s>>>(x);
  note_launches(1);
  return cudaGetLastError();
}
// Resident-sized grid for the pipelined mixed kernel: each thread walks many
// SIPs so the one-ahead staging hides the loads of all but the first.
template <bool PHYS, int MINB>
static cudaError_t mixed_launch(const Bt& B, const PK& x, cudaStream_t s) {
  static std::atomic<int> cached[64];
  int res = 0;
  cudaError_t e = resident_blocks((const void*)k_particles_mixed<PHYS, MINB>, PM_THREADS, PM_SMEM,
                                  cached, &res);
  if (e != cudaSuccess) return e;
  // resident-sized grid: each warp walks many tiles through the staging
  // pipeline; small states take one block per tile (more blocks in flight
  // hide the latency better)
  int64_t bx = res / B.M;
  const int64_t need = (B.n_max + PM_THREADS - 1) / PM_THREADS;
  if (bx * PM_THREADS * 8 > B.n_max) bx = need < 152 * 16 ? need : 152 * 16;
  if (bx > need) bx = need;
  if (bx < 1) bx = 1;
  k_particles_mixed<PHYS, MINB><<<dim3((unsigned)bx, (unsigned)B.M), PM_THREADS, PM_SMEM, s>>>(x);
  note_launches(1);
  return cudaGetLastError();
}
template <bool PHYS>
static cudaError_t mixed_launch_tuned(const Bt& B, const PK& x, cudaStream_t s) {
  switch (tune_value(TUNE_PARTICLE_BLOCKS)) {
    case 5: return mixed_launch<PHYS, 5>(B, x, s);
    case 8: return mixed_launch<PHYS, 8>(B, x, s);
    default: return mixed_launch<PHYS, 6>(B, x, s);
  }
}
cudaError_t launch_particles_mixed(const Bt& B, const lacmo_params_t& p, double dt_sub,
                                   double dt_sub_pos, bool write_Tp, bool hist, cudaStream_t s) {
  PK x{B.ref(), pcall(p, dt_sub, dt_sub_pos, write_Tp, hist)};
  cudaError_t e = mixed_launch_tuned<true>(B, x, s);
  if (e != cudaSuccess) return e;
  k_newton_fallback<<<dim3(64, B.M), 128, 0, s>>>(x); note_launches(1);
  return cudaGetLastError();
}
cudaError_t launch_move_mixed(const Bt& B, double dt_pos, cudaStream_t s) {
  lacmo_params_t p = {};
  PK x{B.ref(), pcall(p, 0.0, dt_pos, false, true)};
  return mixed_launch<false, 6>(B, x, s);
}
cudaError_t launch_wind_float(const Bt& B, cudaStream_t s) {
  k_wind_table<<<grid2(B.nx * B.nz, 256, B.M), 256, 0, s>>>(B.ref()); note_launches(1);
  return cudaGetLastError();
}
cudaError_t launch_grid_acc(const Bt& B, cudaStream_t s) {
  k_grid_acc<<<grid2(B.nx * B.nz, 32, B.M), 32, 0, s>>>(B.ref()); note_launches(1);
  return cudaGetLastError();
}
cudaError_t launch_cell_update(const Bt& B, bool grid_update, cudaStream_t s) {
  k_cell_update<<<grid2(4 * B.nx * B.nz, 32, B.M), 32, 0, s>>>(B.ref(), grid_update ? 1 : 0); note_launches(1);
  return cudaGetLastError();
}
cudaError_t launch_grid_only(const lacmo_grid_t& g, const double* dTh, const double* drv,
                             const double* dml, double* aux, cudaStream_t s) {
  int64_t C = g.nx * g.nz;
  k_grid_only<<<nblocks(C, 32), 32, 0, s>>>(g.scalar_fields, g.mat_prop, aux, dTh, drv, dml, C,
                                              g.p_ref, g.p_ref_inv, g.volume_cell); note_launches(1);
  return cudaGetLastError();
}
cudaError_t launch_advection(const Bt& B, const lacmo_params_t& p, bool second, cudaStream_t s) {
  const bool relax_on = p.act_relaxation && p.init_profile_r_v && p.init_profile_Theta &&
                        p.relaxation_time_profile;
  if (relax_on) {
    k_relaxation2<<<grid2(2 * B.nz, 32, B.M), 32, 0, s>>>(B.ref(), p.init_profile_r_v,
                                                           p.init_profile_Theta,
                                                           p.relaxation_time_profile, p.dt_sub); note_launches(1);
  }
  k_advection<<<grid2(4 * B.nx * B.nz, 32, B.M), 32, 0, s>>>(B.ref(), p.dt_sub, relax_on ? 1 : 0,
                                                          second ? 1 : 0); note_launches(1);
  return cudaGetLastError();
}
cudaError_t launch_divergence(const double* f, const double* flux, int64_t nx, int64_t nz,
                              double dx, double dz, int bcx, int bcz, double* out, cudaStream_t s) {
  k_divergence<<<nblocks(nx * nz, 128), 128, 0, s>>>(f, flux, nx, nz, dx, dz, bcx, bcz, out); note_launches(1);
  return cudaGetLastError();
}
cudaError_t launch_relaxation(const double* f, int64_t nx, int64_t nz, const double* prof,
                              const double* trel, double dt, double* out, cudaStream_t s) {
  k_relaxation<<<nblocks(nz, 128), 128, 0, s>>>(f, nx, nz, prof, trel, dt, out); note_launches(1);
  return cudaGetLastError();
}
cudaError_t launch_r_l_binned(const Bt& B, cudaStream_t s) {
  k_r_l<<<grid2(B.nx * B.nz * 32, 256, B.M, 152 * 16), 256, 0, s>>>(B.ref()); note_launches(1);
  return cudaGetLastError();
}
cudaError_t launch_mass_rate(int sol, int64_t n, const InPtrs& in, double* g, double* dg,
                             cudaStream_t s) {
  k_mass_rate<<<nblocks(n, 128), 128, 0, s>>>(sol, n, in, g, dg); note_launches(1);
  return cudaGetLastError();
}
cudaError_t launch_newton(int sol, int64_t n, double dt_sub, int no_iter, const InPtrs& in,
                          double* dm, double* g0, cudaStream_t s) {
  k_newton<<<nblocks(n, 128), 128, 0, s>>>(sol, n, dt_sub, no_iter, in, dm, g0); note_launches(1);
  return cudaGetLastError();
}
cudaError_t launch_interp(const int32_t* cell, const double* rel, const double* gv, int64_t n,
                          int64_t nx, int64_t nz, double* out, cudaStream_t s) {
  k_interp<<<nblocks(n, 128), 128, 0, s>>>(cell, rel, gv, n, nx, nz, out); note_launches(1);
  return cudaGetLastError();
}

}  // namespace lacmo
