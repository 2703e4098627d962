/*
 * oddeven_cols.cuh -- the odd-even smoother for 9 to 64 states, no more
 * observation rows than states: one thread block per work item, one thread per
 * matrix column, the column's rows in registers.  Included by oddeven.cu.
 *
 * The block-per-item kernels of oddeven_cta.cuh keep their panels in global
 * scratch: every reflector reads each column twice and writes it once through
 * L1, behind a block-wide reduction.  Here a reflector costs two barriers, its
 * vector is read from shared memory by every column at once, and the columns
 * stay in registers for the whole reduction.  At n = 12 the FP64 pipe is then
 * what bounds it (1,800 warp instructions a pair at 19 cycles an SM each); at a
 * few items a level it is the chain of 2 n reflectors, 50 us.  Measured, ms,
 * pairs / back-substitution / weighing, before and now:
 *   16 tracks of 64 to 4,000 steps, n = 12  FP64   7.2 2.0 1.5    2.2 1.1 0.7
 *   2,000 steps, n = 48                     FP64   22.7 8.4 1.6   10.8 6.3 2.3
 *                                           df     16.6 9.9 1.0   4.8 4.5 1.1
 *   4,000 steps, n = 64, states             FP32   8.9 1.0 1.5    3.9 0.4 2.1
 * (the weighing now includes the triangularization).
 *
 * Structure.  Every observation block is upper trapezoidal: the weighing
 * triangularizes it at level 0, stage C from there on.  So each reduction is a
 * trapezoid of m rows on top of a block of rows below.  Reflector k < m takes
 * the top row k and all rows below; from k = m on the top is used up, and the
 * pivot row is the first row below: the rows move up by one, and a zero row
 * joins at the end.  What is left below are the rows that the reduction leaves
 * over.  A top row is needed at its own step only, so it is read then and
 * written then, and only the rows below take registers.
 */
#pragma once

namespace cols {
using ctak::CArgs;
using ctak::RawA;
using columns::back_subst;
using columns::load_end;
using columns::load_rows;
using lanes::inv_root;
using lanes::recip;
using lanes::Refl;
using lanes::reflector;

/* Stage C beside stage B (4 n + 2 columns), or after it where the registers
 * want fewer warps (3 n + 1 columns): a scheduler has 16,384 registers, so
 * nine warps (n = 64) would get 168 each, seven get 255.                     */
template <int NP>
__host__ __device__ constexpr bool merged() { return NP <= 48; }
template <int NP>
__host__ __device__ constexpr int threads() { return ((merged<NP>() ? 4 * NP + 2 : 3 * NP + 1) + 31) / 32 * 32; }
/* the weighing's 3 n + 2 columns, the back-substitution's 3 n + 1 */
template <int NP>
__host__ __device__ constexpr int threads3() { return (3 * NP + 2 + 31) / 32 * 32; }
/* blocks per SM that the registers are budgeted for: a column's rows and about
 * 40 more, without spills                                                   */
template <typename T, int NP>
__host__ __device__ constexpr int blocks()
{
  return sizeof(T) == 8 ? (NP <= 12 ? 8 : NP <= 16 ? 6 : NP <= 24 ? 4 : NP <= 40 ? 2 : 1)
                        : (NP <= 12 ? 12 : NP <= 16 ? 8 : NP <= 24 ? 5 : NP <= 32 ? 4 : 2);
}
template <typename T, int NP>
__host__ __device__ constexpr int blocks3()
{
  return sizeof(T) == 8 ? (NP <= 12 ? 8 : NP <= 16 ? 8 : NP <= 24 ? 5 : NP <= 32 ? 3 : NP <= 56 ? 2 : 1)
                        : (NP <= 12 ? 12 : NP <= 16 ? 12 : NP <= 24 ? 6 : 4);
}

/* the fewest states an instantiation is used for; rows below it need no test
 * (a test every few rows keeps the reads of x from running ahead)             */
template <int NP>
__host__ __device__ constexpr int least() { return NP <= 16 ? NP - 3 : NP <= 24 ? 17 : NP <= 32 ? 25 : NP <= 48 ? 33 : 49; }

template <typename T, int NP>
struct QrShared {
  T x[2][2][NP];       /* [step parity][panel]: the pivot column's rows below */
  T amb[2][2], inv[2][2]; /* its reflector (amb = 0: none) */
};

/* In FP64 a warp without a live column waits, instead of forming products for
 * nothing on the pipe that bounds the kernel: 64 tracks of 100 steps, n = 33,
 * pairs 17.6 -> 14.7 ms, n = 64 63.4 -> 55.4.  Up to 16 states there are two or
 * three warps, and on the FP32 pipe the others hide it: the test costs 1 to 3 %
 * more than it saves.                                                        */
template <typename T, int NP>
__host__ __device__ constexpr bool skips() { return std::is_same<T, double>::value && NP >= 24; }
/* One step of a reduction for a thread whose column has the rows b below and
 * tk on top; panel: 0, or 1 for a second panel reduced at the same time; live:
 * the column takes part; pivot: it is the step's pivot.  Returns the top entry
 * after the step.                                                            */
template <typename T, int NP>
__device__ __forceinline__ T step(QrShared<T, NP>& sm, int k, int panel, bool live, bool pivot, int n, T tk, T (&b)[NP])
{
  const int buf = k & 1;
  T* x = sm.x[buf][panel];
  if (live && pivot)
#pragma unroll
    for (int i = 0; i < NP; ++i) x[i] = b[i];
  __syncthreads();
  T dot = T(0);
  if (!skips<T, NP>() || live) {
    T d0 = T(0), d1 = T(0);
#pragma unroll
    for (int i = 0; i < NP; i += 4)
      if (i < least<NP>() || i < n) { /* rows past n are zero; the same in every thread */
        d0 = fma(x[i], b[i], d0);
        d1 = fma(x[i + 1], b[i + 1], d1);
        d0 = fma(x[i + 2], b[i + 2], d0);
        d1 = fma(x[i + 3], b[i + 3], d1);
      }
    dot = d0 + d1;
  }
  /* the pivot's own product is the tail: its warp alone forms the reflector (a
     fifth to a third of the FP64 instructions, were every warp to do it) */
  if (live && pivot) {
    Refl<T> r;
    r.beta = tk;
    r.amb = r.inv = T(0);
    if (dot != T(0)) r = reflector(tk, dot);
    sm.amb[buf][panel] = r.amb;
    sm.inv[buf][panel] = r.inv;
    tk = r.beta;
  }
  __syncthreads();
  const T amb = sm.amb[buf][panel], inv = sm.inv[buf][panel];
  if (!live || pivot || amb == T(0)) return tk;
  const T d = fma(amb, tk, dot) * inv;
#pragma unroll
  for (int i = 0; i < NP; i += 4)
    if (i < least<NP>() || i < n) {
#pragma unroll
      for (int u = 0; u < 4; ++u) b[i + u] = fma(-d, x[i + u], b[i + u]);
    }
  return fma(-d, amb, tk);
}

/* the rows below move up: the first becomes the top entry */
template <typename T, int NP>
__device__ __forceinline__ T shift(T (&b)[NP])
{
  const T t = b[0];
#pragma unroll
  for (int i = 0; i + 1 < NP; ++i) b[i] = b[i + 1];
  b[NP - 1] = T(0);
  return t;
}

/* A reduction of up to two panels at once: this thread's column is number c of
 * its panel, with m top rows (load(k) reads the top entry, zero past the
 * panel's content) and `steps` reflectors; store(k, v) takes the results.
 * all: the largest `steps` of the block's panels.  Top entries are read a step
 * ahead.  Every thread of the block calls it.                               */
template <typename T, int NP, class LD, class ST>
__device__ __forceinline__ void reduce(QrShared<T, NP>& sm, int panel, bool act, int c, int n, int m, int steps, int all,
                                       T (&b)[NP], LD load, ST store)
{
  T next = act && m > 0 ? load(0) : T(0);
#pragma unroll 1
  for (int k = 0; k < all; ++k) {
    const bool on = act && k < steps;
    T tk = next;
    if (on && k >= m) tk = shift<T, NP>(b);
    next = act && k + 1 < m ? load(k + 1) : T(0);
    /* what a pivot column holds below its own row is not read any more */
    tk = step<T, NP>(sm, k, panel, on && c >= k, c == k, n, tk, b);
    if (on) store(k, tk);
  }
}

/* ---------------------------------------------------------------------------
 * level 0: weighing, and the triangularization of [W G | W o].
 * Threads 0..2n: columns of [H | -F | c]; threads 2n+1..3n+1: columns of [G | o].
 * ------------------------------------------------------------------------ */
/* Lower Cholesky factor of the n x n matrix in L (column-major, ld NP + 1) by one
 * warp, row i on lane i, in registers, the reciprocals of the diagonal in d;
 * *bad is set for a pivot that is not positive (replaced by 1)               */
template <typename T>
__device__ __forceinline__ T bcast(T v, int src) { return __shfl_sync(0xffffffffu, v, src); }
template <>
__device__ __forceinline__ ukg_df::dd bcast<ukg_df::dd>(ukg_df::dd v, int src)
{
  return ukg_df::dd(__shfl_sync(0xffffffffu, v.hi, src), __shfl_sync(0xffffffffu, v.lo, src));
}
template <typename T, int NP>
__device__ __forceinline__ void cholesky_warp(T* L, T* d, int n, int* bad)
{
  constexpr int LD = NP + 1;
  const int lane = threadIdx.x & 31;
  T r[NP]; /* row `lane`, rotated: entry j + k at k in round j */
#pragma unroll
  for (int k = 0; k < NP; ++k) r[k] = lane < n && k <= lane ? L[k * LD + lane] : T(0);
#pragma unroll 1
  for (int j = 0; j < n; ++j) {
    const T s = bcast(r[0], j);
    const bool pd = s > T(0);
    const T v = pd ? inv_root(s) : T(1);
    const T lj = r[0] * v;
    if (lane == j) {
      d[j] = v;
      if (!pd) *bad = 1;
    }
    if (lane > j && lane < n) L[j * LD + lane] = lj;
#pragma unroll
    for (int k = 0; k + 1 < NP; k += 4)
      if (j + 1 + k < n) /* the same in every lane */
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (k + u + 1 < NP) r[k + u] = fma(-lj, bcast(lj, (j + 1 + k + u) & 31), r[k + u + 1]);
  }
}

template <typename T, int NP>
__global__ void __launch_bounds__(threads3<NP>(), blocks3<T, NP>()) weigh_cols(CArgs<T> a, RawA raw)
{
  constexpr int LD = NP + 1, NT = threads3<NP>();
  __shared__ QrShared<T, NP> sm;
  extern __shared__ __align__(16) unsigned char dyn[];
  T* Lk = (T*)dyn;            /* K's factor, column-major */
  T* Lc = Lk + NP * LD;       /* C's */
  T* dk = Lc + NP * LD;       /* reciprocal diagonals (or the weights of 'w') */
  T* dc = dk + NP;
  T* Gs = dc + NP;            /* [W G | W o], column by column */
  __shared__ int bad;
  const int n = a.n, mm = raw.mmax, tid = threadIdx.x;
  const int64_t g = blockIdx.x, nn = (int64_t)n * n;
  const int t = find_track(a.track_start, a.ntracks, g);
  const int64_t q = a.ct.slot[t] + (g - a.track_start[t]);
  const bool evol = g > a.track_start[t];
  int m = raw.obs_rows[g];
  int flag = 0;
  if (m < 0 || m > mm) {
    m = 0;
    flag |= 4;
  }
  const char kt = raw.K_type[g], ct = raw.C_type[g];
  if (evol && !cta::valid_cov_type(kt)) flag |= 4;
  if (m > 0 && !cta::valid_cov_type(ct)) flag |= 4;
  auto fetch = [&](char type, const double* cov, int ld, int rows, T* L, T* d) {
    if (type == 'w') {
      for (int i = tid; i < rows; i += NT) d[i] = ukg_df::narrow<T>(cov[i]);
      return;
    }
    for (int j = tid >> 5; j < rows; j += NT / 32)
      for (int i = tid & 31; i < rows; i += 32) {
        const T v = ukg_df::narrow<T>(cov[(int64_t)j * ld + i]);
        L[j * LD + i] = v;
        if (i == j && (type == 'U' || type == 'F')) {
          d[j] = T(1) / v;
          if (v == T(0)) flag |= 1;
        }
      }
  };
  if (tid == 0) bad = 0;
  if (evol) fetch(kt, raw.K + g * nn, n, n, Lk, dk);
  if (m > 0) fetch(ct, raw.C + g * (int64_t)mm * mm, mm, m, Lc, dc);
  __syncthreads();
  { /* K's factor in the first warp, C's in the second */
    const bool second = tid >= 32;
    if (tid < 64 && (second ? m > 0 && ct == 'C' : evol && kt == 'C'))
      cholesky_warp<T, NP>(second ? Lc : Lk, second ? dc : dk, second ? m : n, &bad);
    __syncthreads();
  }
  if (tid == 0) a.ce.m[q] = m;
  if (tid == 0 && bad) flag |= 1;
  if (flag) atomicOr(a.flag, flag);
  __syncthreads();
  const bool ev = tid <= 2 * n, ob = !ev && tid <= 3 * n + 1;
  const int c = ev ? tid : tid - (2 * n + 1);
  const int rows = ev ? n : m;
  const char type = ev ? kt : ct;
  const T* L = ev ? Lk : Lc;
  const T* d = ev ? dk : dc;
  const double* src = ev ? (c < n ? raw.H + g * nn + (int64_t)c * n
                                  : c < 2 * n ? raw.F + g * nn + (int64_t)(c - n) * n : raw.c + g * n)
                         : (c < n ? raw.G + g * (int64_t)mm * n + (int64_t)c * mm : raw.o + g * mm);
  T* dst = ev ? (c < n ? &a.ce.H.at(c * n, q) : c < 2 * n ? &a.ce.F.at((c - n) * n, q) : &a.ce.c.at(0, q))
              : Gs + c * NP;
  const bool neg = ev && c >= n && c < 2 * n;
  if (ev ? evol : ob && m > 0) {
    T b[NP];
    if (type == 'W') {
#pragma unroll
      for (int i = 0; i < NP; ++i) b[i] = T(0);
#pragma unroll 1
      for (int k = 0; k < rows; ++k) {
        T v = ukg_df::narrow<T>(src[k]);
        if (neg) v = -v;
#pragma unroll
        for (int i = 0; i < NP; ++i)
          if (i < rows) b[i] = fma(L[k * LD + i], v, b[i]);
      }
#pragma unroll
      for (int i = 0; i < NP; ++i)
        if (i < rows) dst[i] = b[i];
    } else {
#pragma unroll
      for (int i = 0; i < NP; ++i) {
        b[i] = T(0);
        if (i < rows) b[i] = ukg_df::narrow<T>(src[i]);
        if (neg) b[i] = -b[i];
      }
      const bool low = type == 'C' || type == 'U' || type == 'F';
#pragma unroll 1
      for (int j = 0; j < rows; ++j) { /* forward substitution; the rows move up as they are done */
        const T v = low || type == 'w' ? b[0] * d[j] : b[0];
        dst[j] = v;
        const T* Lj = L + j * LD + j + 1;
#pragma unroll
        for (int i = 0; i < NP; i += 4)
          if (j + 1 + i < rows) 
#pragma unroll
            for (int u = 0; u < 4; ++u)
              if (i + u + 1 < NP) b[i + u] = j + 1 + i + u >= rows ? T(0) : low ? fma(-v, Lj[i + u], b[i + u + 1]) : b[i + u + 1];
      }
    }
  }
  if (m == 0) return; /* the whole block */
  __syncthreads();
  /* R of [W G | W o]: all steps take their pivot from the rows below */
  T b[NP];
  const bool act = tid <= n;
  load_rows<T, NP>(Gs + tid * NP, m, act, b);
  const int steps = m < n ? m : n;
  T* out = tid < n ? &a.ce.G.at(tid * a.mx, q) : &a.ce.o.at(0, q);
  reduce<T, NP>(sm, 0, act, tid, m, 0, steps, steps, b, [](int) { return T(0); },
                [&](int k, T v) { out[k] = tid < n && k > tid ? T(0) : v; });
}
/* Above 32 states ctak::weigh_cta weighs: a block a step here is one or two an
 * SM, whose chain of n pivots and n reflectors nothing hides (6,400 steps, n = 49,
 * m = 24: 14.2 ms, double-float 11.6; apart 7.2 and 4.3).
 * Then the observations alone are triangularized.                            */
template <int NP>
__host__ __device__ constexpr int tri_threads() { return (NP + 1 + 31) / 32 * 32; }
template <typename T, int NP>
__global__ void __launch_bounds__(tri_threads<NP>(), sizeof(T) == 8 ? (NP <= 48 ? 6 : 4) : (NP <= 48 ? 8 : 5))
    triangularize(CArgs<T> a)
{
  __shared__ QrShared<T, NP> sm;
  const int n = a.n, tid = threadIdx.x;
  const int64_t g = blockIdx.x;
  const int t = find_track(a.track_start, a.ntracks, g);
  const int64_t q = a.ct.slot[t] + (g - a.track_start[t]);
  const int m = a.ce.m[q], steps = m < n ? m : n;
  const bool act = tid <= n;
  T* col = tid < n ? &a.ce.G.at(tid * a.mx, q) : &a.ce.o.at(0, q);
  T b[NP];
  load_rows<T, NP>(col, m, act, b);
  reduce<T, NP>(sm, 0, act, tid, n, 0, steps, steps, b, [](int) { return T(0); },
                [&](int k, T v) { col[k] = tid < n && k > tid ? T(0) : v; });
}
template <typename T, int NP>
constexpr size_t weigh_smem() { return (size_t)(2 * NP * (NP + 1) + 2 * NP + (NP + 1) * NP) * sizeof(T); }

/* ---------------------------------------------------------------------------
 * forward elimination of one pair: stage A on threads 0..2n (pivots, right-hand
 * side, H_{j+1}); stage B on 0..3n (the same with Y~, then F_j) while stage C
 * runs on 3n+1..4n+1.
 * ------------------------------------------------------------------------ */
template <typename T, int NP>
__global__ void __launch_bounds__(threads<NP>(), blocks<T, NP>()) pair_cols(CArgs<T> a)
{
  __shared__ QrShared<T, NP> sm;
  extern __shared__ __align__(16) unsigned char dyn[];
  const int n = a.n, mx = a.mx, tid = threadIdx.x;
  const int ldt = 2 * n + 1;
  T* Tp = (T*)dyn;             /* stage A's top rows: [R~ | rhs~ | Y~], n x (2n+1) */
  T* Hs = Tp + n * ldt;        /* [H~ | o~], column by column (n rows each, m_j in use) */
  const auto& C = a.ce;
  const auto& Nx = a.ne;
  const auto& Rr = a.cr;
  const int64_t item = blockIdx.x;
  const int t = find_track(a.ct.pair, a.ntracks, item);
  const int64_t p = item - a.ct.pair[t];
  const int64_t sj = a.ct.slot[t] + 2 * p, sj1 = sj + 1;
  const int64_t sn = a.nt.slot[t] + p, se = a.ct.solve[t] + p;
  const int mj = C.m[sj], mj1 = C.m[sj1];
  T b[NP];
  /* stage A */
  {
    const bool act = tid <= 2 * n;
    const T* bot = tid < n ? &C.F.at(tid * n, sj1) : tid == n ? &C.c.at(0, sj1) : &C.H.at((tid - n - 1) * n, sj1);
    load_rows<T, NP>(bot, n, act, b);
    const T* top = tid < n ? &C.G.at(tid * mx, sj) : &C.o.at(0, sj);
    reduce<T, NP>(sm, 0, act, tid, n, mj, n, n, b,
                  [&](int k) { return tid > n || (tid < n && k > tid) ? T(0) : top[k]; },
                  [&](int k, T v) { Tp[k * ldt + tid] = v; });
    if (tid >= n && tid <= 2 * n) {
      T* h = Hs + (tid == n ? n : tid - n - 1) * n;
#pragma unroll
      for (int i = 0; i < NP; ++i)
        if (i < mj) h[i] = b[i];
    }
    __syncthreads();
  }
  /* stages B and C */
  constexpr bool kMerged = merged<NP>();
  const int nC = mj + mj1 < n ? mj + mj1 : n;
  const bool isC = kMerged && tid > 3 * n, act = tid <= (kMerged ? 4 * n + 1 : 3 * n) && (isC || p > 0);
  const int c = isC ? tid - (3 * n + 1) : tid;
  if (!kMerged) { /* stage C first, on threads 0..n */
    load_rows<T, NP>(Hs + (tid <= n ? tid : 0) * n, mj, tid <= n, b);
    const T* top = tid < n ? &C.G.at(tid * mx, sj1) : &C.o.at(0, sj1);
    T* out = tid < n ? &Nx.G.at(tid * mx, sn) : &Nx.o.at(0, sn);
    reduce<T, NP>(sm, 0, tid <= n, tid, n, mj1, nC, nC, b, [&](int k) { return tid < n && k > tid ? T(0) : top[k]; },
                  [&](int k, T v) { out[k] = tid < n && k > tid ? T(0) : v; });
    __syncthreads(); /* the buffers of the last steps are free */
  }
  if (isC) load_rows<T, NP>(Hs + (c <= n ? c : 0) * n, mj, act, b);
  else
    load_rows<T, NP>(c < n ? &C.H.at(c * n, sj) : c == n ? &C.c.at(0, sj) : &C.F.at((c > 2 * n ? c - 2 * n - 1 : 0) * n, sj),
                     n, act && (c <= n || c > 2 * n), b);
  const T* top = isC ? (c < n ? &C.G.at(c * mx, sj1) : &C.o.at(0, sj1)) : Tp + c;
  T* out = isC ? (c < n ? &Nx.G.at(c * mx, sn) : &Nx.o.at(0, sn))
               : c < n ? &Rr.R.at(c * n, se) : c == n ? &Rr.rhs.at(0, se)
               : c <= 2 * n ? &Rr.Y.at((c - n - 1) * n, se) : &Rr.Ft.at((c - 2 * n - 1) * n, se);
  const bool zero_below = c < n; /* R~ and G are triangular: their lower entries hold reflectors, or nothing */
  reduce<T, NP>(sm, isC ? 1 : 0, act, c, n, isC ? mj1 : n, isC ? nC : n, p > 0 ? n : kMerged ? nC : 0, b,
                [&](int k) {
                  if (zero_below && k > c) return T(0);
                  return isC ? top[k] : c > 2 * n ? T(0) : top[k * ldt];
                },
                [&](int k, T v) { out[k] = zero_below && k > c ? T(0) : v; });
  if (tid == 0) Nx.m[sn] = nC;
  if (p == 0) { /* no stage B: the record is stage A's */
    if (tid <= 3 * n)
      for (int k = 0; k < n; ++k) out[k] = c > 2 * n || (c < n && k > c) ? T(0) : Tp[k * ldt + c];
    return;
  }
  if (tid >= n && tid <= 3 * n) { /* the rows left over: the next level's evolution */
    T* dst = c == n ? &Nx.c.at(0, sn) : c <= 2 * n ? &Nx.H.at((c - n - 1) * n, sn) : &Nx.F.at((c - 2 * n - 1) * n, sn);
#pragma unroll
    for (int i = 0; i < NP; ++i)
      if (i < n) dst[i] = b[i];
  }
}
template <typename T>
size_t pair_smem(int n) { return (size_t)(n * (2 * n + 1) + (n + 1) * n) * sizeof(T); }

/* ---------------------------------------------------------------------------
 * odd-length tracks: the single last step and its fix-up, or the base case
 * ------------------------------------------------------------------------ */
template <typename T, int NP>
__global__ void __launch_bounds__(threads<NP>(), blocks<T, NP>()) tail_cols(CArgs<T> a)
{
  __shared__ QrShared<T, NP> sm;
  extern __shared__ __align__(16) unsigned char dyn[];
  const int n = a.n, mx = a.mx, tid = threadIdx.x;
  constexpr int NT = threads<NP>();
  T* Z = (T*)dyn; /* rows left over, column by column; or the base factor */
  T* dv = Z + (n + 1) * n;
  T* Ri = dv + n;
  const auto& C = a.ce;
  const auto& Nx = a.ne;
  const auto& Rr = a.cr;
  const int t = (int)a.ct.tail[blockIdx.x];
  const int64_t L = a.ct.L[t], sb = a.ct.slot[t];
  if (L == 1) { /* base case: x = R^{-1} o, S = R^{-1} R^{-T} */
    const int64_t os = orig_step(a.track_start, a.level, t, 0);
    double* x = a.state + os * n;
    double* S = a.cov ? a.cov + os * (int64_t)n * n : nullptr;
    if (C.m[sb] < n) {
      for (int i = tid; i < n; i += NT) x[i] = NAN;
      if (S)
        for (int e = tid; e < n * n; e += NT) S[e] = NAN;
      if (tid == 0) atomicOr(a.flag, 2);
      return;
    }
    for (int e = tid; e < n * n; e += NT) {
      const int q = e / n, r = e - q * n;
      const T v = r <= q ? C.G.at(q * mx + r, sb) : T(0);
      Z[e] = v;
      if (r == q) {
        dv[q] = recip(v);
        if (v == T(0)) atomicOr(a.flag, 2);
      }
      if (a.baseR.p) a.baseR.at(e, t) = v;
    }
    __syncthreads();
    T b[NP];
    if (tid == n) load_end<T, NP>(&C.o.at(0, sb), n, true, b);
    else
#pragma unroll
      for (int i = 0; i < NP; ++i) b[i] = tid < n && i - NP + n == tid ? T(1) : T(0);
    if (tid == n || (tid < n && S))
      back_subst<T, NP>(Z, dv, n, b, [&](int j, T v) {
        if (tid == n) x[j] = ukg_df::widen(v);
        else Ri[tid * n + j] = v;
      });
    if (!S) return;
    __syncthreads();
    for (int e = tid; e < n * n; e += NT) {
      const int q = e / n, r = e - q * n;
      if (r < q) continue;
      T s = T(0);
      for (int k = r; k < n; ++k) s = fma(Ri[k * n + r], Ri[k * n + q], s);
      const double v = ukg_df::widen(s);
      S[q * n + r] = v;
      S[r * n + q] = v;
    }
    return;
  }
  const int64_t s = sb + L - 1, es = a.ct.solve[t] + (L - 1) / 2, sn = a.nt.slot[t] + L / 2 - 1;
  const int mt = C.m[s]; /* <= n: the observation is a trapezoid already */
  T b[NP];
  { /* [R~ | o' | 0; H_s | c_s | F_s] */
    const bool act = tid <= 2 * n;
    load_rows<T, NP>(tid < n ? &C.H.at(tid * n, s) : tid == n ? &C.c.at(0, s) : &C.F.at((tid - n - 1) * n, s), n, act, b);
    const T* top = tid < n ? &C.G.at(tid * mx, s) : &C.o.at(0, s);
    T* out = tid < n ? &Rr.R.at(tid * n, es) : tid == n ? &Rr.rhs.at(0, es) : &Rr.Ft.at((tid - n - 1) * n, es);
    reduce<T, NP>(sm, 0, act, tid, n, mt, n, n, b,
                  [&](int k) { return tid > n || (tid < n && k > tid) ? T(0) : top[k]; },
                  [&](int k, T v) { out[k] = tid < n && k > tid ? T(0) : v; });
    if (tid >= n && act) {
      T* z = Z + (tid == n ? n : tid - n - 1) * n;
#pragma unroll
      for (int i = 0; i < NP; ++i)
        if (i < mt) z[i] = b[i];
    }
    for (int e = tid; e < n * n; e += NT) Rr.Y.at(e, es) = T(0);
    __syncthreads();
  }
  /* fix-up: [G~ | o; Z | o''] */
  const int gp = Nx.m[sn], nF = gp + mt < n ? gp + mt : n;
  const bool act = tid <= n;
  load_rows<T, NP>(Z + (act ? tid : 0) * n, mt, act, b);
  T* out = tid < n ? &Nx.G.at(tid * mx, sn) : &Nx.o.at(0, sn);
  reduce<T, NP>(sm, 0, act, tid, n, gp, nF, nF, b, [&](int k) { return tid < n && k > tid ? T(0) : out[k]; },
                [&](int k, T v) { out[k] = tid < n && k > tid ? T(0) : v; });
  if (tid == 0) Nx.m[sn] = nF;
}
template <typename T>
size_t tail_smem(int n) { return (size_t)((n + 1) * n + n + n * n) * sizeof(T); }

/* ---------------------------------------------------------------------------
 * back-substitution with covariances of one even step (solve_cta's formulas):
 * threads 0..2n-1 a column of W = B Sigma each, thread 2n the state,
 * threads 2n+1..3n the columns of M = I + W B^T (its lower triangle computed)
 * ------------------------------------------------------------------------ */
template <typename T, int NP>
__global__ void __launch_bounds__(threads3<NP>(), blocks3<T, NP>()) solve_cols(CArgs<T> a)
{
  extern __shared__ __align__(16) unsigned char dyn[];
  constexpr int NT = threads3<NP>();
  const int n = a.n, tid = threadIdx.x, nn = n * n;
  T* B = (T*)dyn;      /* [F~ | Y], column-major */
  T* R = B + 2 * nn;   /* column-major */
  T* W = R + nn;       /* column-major, n x 2n; then X */
  T* M = W + 2 * nn;   /* its lower triangle, column by column */
  T* dv = M + n * (n + 1) / 2;
  auto at_m = [&](int i, int c) { return c * n - c * (c - 1) / 2 + i - c; }; /* i >= c */
  const auto& Rr = a.cr;
  const int64_t item = blockIdx.x;
  const int t = find_track(a.ct.solve, a.ntracks, item);
  const int64_t j = 2 * (item - a.ct.solve[t]), L = a.ct.L[t];
  const bool hp = j > 0, hn = j + 1 < L;
  const int64_t oj = orig_step(a.track_start, a.level, t, j);
  const int64_t om = hp ? orig_step(a.track_start, a.level, t, j - 1) : 0;
  const int64_t op = hn ? orig_step(a.track_start, a.level, t, j + 1) : 0;
  const int64_t smp = hp && hn ? a.nt.slot[t] + (j + 1) / 2 : 0;
  for (int e = tid; e < nn; e += NT) {
    B[e] = hp ? Rr.Ft.at(e, item) : T(0);
    B[nn + e] = hn ? Rr.Y.at(e, item) : T(0);
    const T r = Rr.R.at(e, item);
    R[e] = r;
    if (e % (n + 1) == 0) {
      dv[e / (n + 1)] = recip(r);
      if (r == T(0)) atomicOr(a.flag, 2);
    }
  }
  __syncthreads();
  const bool isW = tid < 2 * n, isx = tid == 2 * n;
  const int q = tid < n ? tid : tid - n;
  T b[NP]; /* aligned to the end: row i at NP - n + i */
  if (isx) load_end<T, NP>(&Rr.rhs.at(0, item), n, true, b);
  else
#pragma unroll
    for (int i = 0; i < NP; ++i) b[i] = T(0);
  auto add = [&](const T* Bk, T s) {
    const T* p = Bk + n - NP;
#pragma unroll
    for (int i = 0; i < NP; i += 4)
      if (i + 3 - NP + n >= 0) {
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (i + u - NP + n >= 0) b[i + u] = fma(p[i + u], s, b[i + u]);
      }
  };
  if (isW || isx) {
    /* b += B s, four entries of s at a time, the next four on their way */
    auto run = [&](const T* Bk, auto&& at) {
      T s[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) s[u] = u < n ? at(u) : T(0);
#pragma unroll 1
      for (int k = 0; k < n; k += 4) {
        T next[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) next[u] = k + 4 + u < n ? at(k + 4 + u) : T(0);
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (k + u < n) add(Bk + (k + u) * n, s[u]);
#pragma unroll
        for (int u = 0; u < 4; ++u) s[u] = next[u];
      }
    };
    /* Sigma's column q: Smm or Smp above, Smp^T or Spp below; the negated states
       on thread 2n.  One loop for all: the sources differ by address only.   */
    const bool both = hp && hn;
    auto half = [&](const T* Bk, const double* p, bool fp64, const T* u, int us) {
      run(Bk, [&](int k) {
        T v = T(0);
        if (fp64) v = ukg_df::narrow<T>(isx ? -p[k] : p[k]);
        else if (both) v = u[(int64_t)k * us];
        return v;
      });
    };
    const T* U = a.nr.U.p + smp * a.nr.U.w;
    if (hp) half(B, isx ? a.state + om * n : a.cov + om * nn + (int64_t)q * n, tid < n || isx, U + q * n, 1);
    if (hn) half(B + nn, isx ? a.state + op * n : a.cov + op * nn + (int64_t)q * n, tid >= n, U + q, n);
  }
  if (isW) {
#pragma unroll
    for (int i = 0; i < NP; ++i)
      if (i - NP + n >= 0) W[tid * n + i - NP + n] = b[i];
  }
  __syncthreads();
  const int q0 = hp ? 0 : n, q1 = hn ? 2 * n : n;
  /* M(i, c), i >= c: columns c and n - 1 - c together have n + 1 such entries */
  for (int e = tid; e < (n + 1) / 2 * (n + 1); e += NT) {
    const int c0 = e / (n + 1), r = e - c0 * (n + 1);
    const int c = r < n - c0 ? c0 : n - 1 - c0, i = r < n - c0 ? c0 + r : r - 1;
    if (2 * c0 == n - 1 && r >= n - c0) continue; /* the middle column of an odd n */
    T s0 = T(0), s1 = T(0);
    for (int k = q0; k + 1 < q1; k += 2) {
      s0 = fma(W[k * n + i], B[k * n + c], s0);
      s1 = fma(W[(k + 1) * n + i], B[(k + 1) * n + c], s1);
    }
    if ((q1 - q0) & 1) s0 = fma(W[(q1 - 1) * n + i], B[(q1 - 1) * n + c], s0);
    T m = s0 + s1;
    if (i == c) m += T(1);
    M[at_m(i, c)] = m;
  }
  __syncthreads(); /* W is in registers: X goes there */
  const int mc = tid - (2 * n + 1);
  const bool isM = mc >= 0 && mc < n;
  T* X = W;
  if (isM)
#pragma unroll
    for (int i = 0; i < NP; ++i) {
      const int r = i - NP + n;
      b[i] = r < 0 ? T(0) : M[r >= mc ? at_m(r, mc) : at_m(mc, r)];
    }
  {
    /* one substitution for the blocks -R^{-1} W, the state and X = R^{-1} M: the
       columns differ by where they go.  cov(x_{j-1}, x_j): row q of U;
       cov(x_j, x_{j+1}): column q                                            */
    const bool isU = isW && a.level > 0 && (tid < n ? hp : hn);
    T* dst = isU ? (tid < n ? &Rr.U.at(q, a.ct.slot[t] + j) : &Rr.U.at(q * n, a.ct.slot[t] + j + 1)) : X + (isM ? mc : 0);
    const int ds = isU && tid >= n ? 1 : n; /* X transposed: row mc */
    if (isU || isx || isM)
      back_subst<T, NP>(R, dv, n, b, [&](int r, T v) {
        if (isx) a.state[oj * n + r] = ukg_df::widen(v);
        else dst[r * ds] = isU ? -v : v;
      });
  }
  __syncthreads();
  if (isM) {
    load_end<T, NP>(X + mc * n, n, true, b); /* X^T's column mc */
    double* So = a.cov + oj * nn;
    back_subst<T, NP>(R, dv, n, b, [&](int r, T v) {
      if (r >= mc) {
        const double w = ukg_df::widen(v);
        So[mc * n + r] = w;
        So[r * n + mc] = w;
      }
    });
  }
}
template <typename T>
size_t solve_smem(int n) { return (size_t)(5 * n * n + n * (n + 1) / 2 + n) * sizeof(T); }

/* the state alone, a warp per even step: lanes over the rows (row lane + 32 u) */
template <typename T, int NP>
__global__ void __launch_bounds__(128) state_cols(CArgs<T> a)
{
  constexpr int RU = (NP + 31) / 32;
  const int64_t item = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
  if (item >= a.ct.nsolve) return; /* the whole warp */
  const int lane = threadIdx.x & 31, n = a.n;
  const auto& Rr = a.cr;
  const int t = find_track(a.ct.solve, a.ntracks, item);
  const int64_t j = 2 * (item - a.ct.solve[t]), L = a.ct.L[t];
  const bool hp = j > 0, hn = j + 1 < L;
  T x[RU];
#pragma unroll
  for (int u = 0; u < RU; ++u) {
    const int r = lane + 32 * u;
    x[u] = r < n ? (a.yrhs.p ? a.yrhs.at(r, item) : Rr.rhs.at(r, item)) : T(0);
  }
  /* eight columns' reads before their use, without branches (rows and columns
     past n are the last one's, times zero or not used): left to the compiler,
     each column waited for its own (12 levels of 128 states 1.86 ms, now
     0.84)                                                                   */
  constexpr int KB = sizeof(T) * RU > 16 ? 4 : 8;
  int row[RU];
#pragma unroll
  for (int u = 0; u < RU; ++u) row[u] = lane + 32 * u < n ? lane + 32 * u : n - 1;
  auto sub = [&](const T* B, const double* s) {
#pragma unroll 1
    for (int k0 = 0; k0 < n; k0 += KB) {
      T v[KB][RU], sk[KB];
#pragma unroll
      for (int i = 0; i < KB; ++i) {
        const int k = k0 + i < n ? k0 + i : n - 1;
        sk[i] = k0 + i < n ? -ukg_df::narrow<T>(s[k]) : T(0);
#pragma unroll
        for (int u = 0; u < RU; ++u) v[i][u] = B[k * n + row[u]];
      }
#pragma unroll
      for (int i = 0; i < KB; ++i)
#pragma unroll
        for (int u = 0; u < RU; ++u) x[u] = fma(v[i][u], sk[i], x[u]);
    }
  };
  if (hp) sub(&Rr.Ft.at(0, item), a.state + orig_step(a.track_start, a.level, t, j - 1) * n);
  if (hn) sub(&Rr.Y.at(0, item), a.state + orig_step(a.track_start, a.level, t, j + 1) * n);
  const T* R = &Rr.R.at(0, item);
  bool bad = false;
  T dv[RU];
#pragma unroll
  for (int u = 0; u < RU; ++u) {
    const int r = lane + 32 * u;
    const T d = r < n ? R[r * n + r] : T(1);
    bad |= d == T(0);
    dv[u] = recip(d);
  }
#pragma unroll
  for (int w = RU - 1; w >= 0; --w)
#pragma unroll 1
    for (int c0 = 32 * w + 32 - KB; c0 >= 32 * w; c0 -= KB) {
      if (c0 >= n) continue;
      T v[KB][RU];
#pragma unroll
      for (int i = 0; i < KB; ++i)
#pragma unroll
        for (int u = 0; u <= w; ++u) v[i][u] = R[(c0 + i < n ? c0 + i : n - 1) * n + row[u]];
#pragma unroll
      for (int i = KB - 1; i >= 0; --i) {
        const int c = c0 + i;
        if (c < n) { /* the same in every lane */
          const T xc = bcast(x[w] * dv[w], c - 32 * w);
          if (lane == c - 32 * w) x[w] = xc;
#pragma unroll
          for (int u = 0; u <= w; ++u)
            if (lane + 32 * u < c) x[u] = fma(-xc, v[i][u], x[u]);
        }
      }
    }
  double* xo = a.state + orig_step(a.track_start, a.level, t, j) * n;
#pragma unroll
  for (int u = 0; u < RU; ++u)
    if (lane + 32 * u < n) xo[lane + 32 * u] = ukg_df::widen(x[u]);
  if (bad) atomicOr(a.flag, 2);
}

/* the kernels of a state dimension: the smallest instantiation that holds it */
template <typename T>
struct Kernels {
  void (*weigh)(CArgs<T>, RawA) = nullptr; /* or ctak::weigh_cta and tri */
  void (*tri)(CArgs<T>) = nullptr;
  void (*pair)(CArgs<T>) = nullptr;
  void (*tail)(CArgs<T>) = nullptr;
  void (*solve)(CArgs<T>) = nullptr;
  void (*state)(CArgs<T>) = nullptr;
  int threads = 0, weigh_threads = 0, tri_threads = 0, solve_threads = 0;
  size_t weigh_smem = 0;
};
template <typename T, int NP>
void pairs_np(Kernels<T>& k)
{
  k.pair = pair_cols<T, NP>;
  k.tail = tail_cols<T, NP>;
  k.threads = threads<NP>();
}
template <typename T, int NP>
void solve_np(Kernels<T>& k)
{
  if constexpr (sizeof(T) == 8) {
    k.solve = solve_cols<T, NP>;
    k.solve_threads = threads3<NP>();
  }
}
template <typename T, int NP>
Kernels<T> kernels_np()
{
  Kernels<T> k;
  if constexpr (NP <= 32) {
    k.weigh = weigh_cols<T, NP>;
    k.weigh_threads = threads3<NP>();
    k.weigh_smem = weigh_smem<T, NP>();
  } else {
    k.tri = triangularize<T, NP>;
    k.tri_threads = tri_threads<NP>();
  }
  pairs_np<T, NP>(k);
  solve_np<T, NP>(k);
  k.state = state_cols<T, NP>;
  return k;
}
template <typename T>
Kernels<T> kernels(int n, int mx)
{
  if (n != mx || n < 9) return Kernels<T>();
  if (n <= 12) return kernels_np<T, 12>();
  if (n <= 16) return kernels_np<T, 16>();
  if (n <= 24) return kernels_np<T, 24>();
  if (n <= 32) return kernels_np<T, 32>();
  Kernels<T> k;
  if (n <= 64) {
    k = n <= 48 ? kernels_np<T, 48>() : kernels_np<T, 64>();
    /* Registers (and shared memory) for two blocks an SM instead of one: 64
       tracks of 100 steps, n = 33, FP64, pairs 14.7 -> 10.0 ms (19.0 -> 12.8 at
       n = 40); n = 49, even steps 19.2 -> 13.0, double-float 25.5 -> 14.3.  The
       pairs of 41 states and more would spill, the even steps of 51 and more do
       not fit the shared memory twice.                                       */
    if constexpr (sizeof(T) == 8) {
      if (n <= 40) pairs_np<T, 40>(k), solve_np<T, 40>(k);
      if (n > 48 && n <= 50) solve_np<T, 56>(k);
    }
    return k;
  }
  k.state = state_cols<T, 128>; /* above, the states' back-substitution alone */
  return k;
}

}  // namespace cols
