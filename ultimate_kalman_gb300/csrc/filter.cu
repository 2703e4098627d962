/*
 * filter.cu -- filtered estimates on the device: the sequential UltimateKalman
 * filter (c/kalman_ultimate.c: evolve 140-345, observe 347-557 with its
 * estimate 508-545) run for every track of a packed problem at once
 * (kalman_gpu_filter_packed): a warp per track and three kernels up to 8 states
 * and observation rows (below), a thread block per track (filter_cta) from there
 * on.  The reference keeps the covariance as the factor R (its covariance_type
 * 'W'); here P = R^{-1} R^{-T} is written explicitly, as the smoothers write
 * theirs.
 *
 * Kept per track is the factor of the current state's information, an
 * upper-trapezoidal R (z rows, z <= n) and its right-hand side y:
 *   evolve to step i   QR, eliminating x_{i-1}, of
 *                        [ R        0     | y    ]   (z rows)
 *                        [ -V F_i   V H_i | V c_i ]   (n rows; V from K_i)
 *                      the last z rows become [R~ | y~] for x_i;
 *   observe            QR of [R~ | y~; W G_i | W o_i] (W from C_i; no rows
 *                      when the step is unobserved) -> R, y with
 *                      z = min(z + m_i, n) rows;
 *   estimate           x_{i|i} = R^{-1} y and P_{i|i} = R^{-1} R^{-T} once
 *                      z = n (NaN before, as the reference's estimate).
 * filter_cta's QR reductions, weighing and triangular solves are the CTA
 * routines of the smoothers (cta_linalg.cuh).  FP64.
 */
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <new>
#include <numeric>
#include <vector>

#include <cuda_runtime.h>

#include "cta_linalg.cuh"
#include "lanes.cuh"
#include "profiling.h"
#include "ukgpu_internal.h"

namespace {

using cta::NT;

struct FilterArgs {
  int n, mmax, ntracks;
  const int64_t* track_start; /* device */
  const double *H, *F, *c, *K, *G, *o, *C;
  const char *K_type, *C_type;
  const int32_t* obs_rows;
  double* state;
  double* cov; /* may be null */
  double* scratch;
  int64_t per_cta;
  int* flag; /* 1: an estimate was undetermined (NaN written), 4: malformed input */
};

/* per-CTA scratch: the evolve panel (z + n) x (2n + 1), the observe panel
 * (n + mmax) x (n + 1), the weighing factor rmax^2 and product tmp, R^{-1} */
int64_t filter_scratch(int n, int mmax)
{
  const int64_t rmax = n > mmax ? n : mmax;
  const int64_t evolve = 2 * (int64_t)n * (2 * n + 1);
  const int64_t observe = (int64_t)(n + mmax) * (n + 1);
  const int64_t weigh = rmax * rmax + rmax * NT;
  return evolve + observe + weigh + (int64_t)n * n + 32;
}

__global__ void __launch_bounds__(NT) filter_cta(FilterArgs a)
{
  __shared__ double red[33];
  __shared__ int zs;
  const int n = a.n, mm = a.mmax, tid = threadIdx.x;
  const int64_t nn = (int64_t)n * n;
  const int le = 2 * n + 1, lo = n + 1;
  double* E = a.scratch + (int64_t)blockIdx.x * a.per_cta; /* evolve panel, row-major, ld le */
  double* O = E + 2 * (int64_t)n * le;                      /* observe panel, row-major, ld lo */
  double* Lw = O + (int64_t)(n + mm) * lo;                   /* weighing factor */
  double* tmp = Lw + (int64_t)(n > mm ? n : mm) * (n > mm ? n : mm);
  double* Ri = tmp + (int64_t)(n > mm ? n : mm) * NT;       /* R^{-1}, row-major */
  for (int t = blockIdx.x; t < a.ntracks; t += gridDim.x) {
    const int64_t s0 = a.track_start[t], s1 = a.track_start[t + 1];
    int z = 0; /* rows of the current factor, held in O's first rows as [R | y] */
    for (int64_t s = s0; s < s1; ++s) {
      bool bad = false;
      if (s > s0) { /* evolve: [R 0 | y; -V F  V H | V c], n pivots */
        for (int e = tid; e < z * le; e += NT) {
          const int r = e / le, q = e - r * le;
          /* R's upper triangle only: the QR that made it keeps its reflectors below */
          E[e] = q < n ? (q >= r ? O[(int64_t)r * lo + q] : 0.0) : q < 2 * n ? 0.0 : O[(int64_t)r * lo + n];
        }
        double* B = E + (int64_t)z * le;
        for (int e = tid; e < n * le; e += NT) {
          const int r = e / le, q = e - r * le;
          B[e] = q < n ? -a.F[s * nn + (int64_t)q * n + r]
                       : q < 2 * n ? a.H[s * nn + (int64_t)(q - n) * n + r] : a.c[s * n + r];
        }
        __syncthreads();
        const char kt = a.K_type[s];
        if (tid == 0 && !cta::valid_cov_type(kt)) atomicOr(a.flag, 4);
        bad |= !cta::weigh_panel(kt, a.K + s * nn, n, n, B, le, le, Lw, red, tmp);
        cta::householder(E, le, z + n, n, le, red);
        /* the last z rows: [0 | R~ | y~] -> O's first z rows */
        for (int e = tid; e < z * lo; e += NT) {
          const int r = e / lo, q = e - r * lo;
          O[e] = E[(int64_t)(n + r) * le + n + q];
        }
        __syncthreads();
      }
      /* observe: [R~ | y~ (z rows); W G | W o (m rows)], n pivots */
      int m = a.obs_rows[s];
      if (m < 0 || m > mm) {
        if (tid == 0) atomicOr(a.flag, 4);
        m = 0;
      }
      if (m > 0) {
        double* B = O + (int64_t)z * lo;
        for (int e = tid; e < m * lo; e += NT) {
          const int r = e / lo, q = e - r * lo;
          B[e] = q < n ? a.G[s * (int64_t)mm * n + (int64_t)q * mm + r] : a.o[s * mm + r];
        }
        __syncthreads();
        const char ct = a.C_type[s];
        if (tid == 0 && !cta::valid_cov_type(ct)) atomicOr(a.flag, 4);
        bad |= !cta::weigh_panel(ct, a.C + s * (int64_t)mm * mm, mm, m, B, lo, lo, Lw, red, tmp);
      }
      const int rows = z + m;
      if (rows > 0) cta::householder(O, lo, rows, n, lo, red);
      z = rows < n ? rows : n; /* rows below the factor are the residual, dropped */
      if (bad && tid == 0) atomicOr(a.flag, 1);
      /* estimate */
      if (tid == 0) {
        int ok = z == n;
        for (int i = 0; ok && i < n; ++i)
          if (O[(int64_t)i * lo + i] == 0.0) ok = 0;
        zs = ok;
      }
      __syncthreads();
      double* x = a.state + s * n;
      double* P = a.cov ? a.cov + s * nn : nullptr;
      if (!zs) {
        for (int i = tid; i < n; i += NT) x[i] = NAN;
        if (P)
          for (int e = tid; e < nn; e += NT) P[e] = NAN;
        if (tid == 0) atomicOr(a.flag, 1);
        __syncthreads();
        continue;
      }
      /* x = R^{-1} y, with y copied out of the panel (the panel stays the factor) */
      double* yv = tmp;
      for (int i = tid; i < n; i += NT) yv[i] = O[(int64_t)i * lo + n];
      __syncthreads();
      cta::solve_upper_vec(O, lo, n, yv);
      for (int i = tid; i < n; i += NT) x[i] = yv[i];
      if (P) { /* P = R^{-1} R^{-T}, column-major out */
        for (int e = tid; e < nn; e += NT) Ri[e] = (e / n == e % n) ? 1.0 : 0.0;
        __syncthreads();
        cta::solve_upper_cols(O, lo, n, Ri, n, 0, n);
        for (int e = tid; e < nn; e += NT) {
          const int r = e / n, q = e - r * n;
          double sm = 0.0;
          for (int k = (r > q ? r : q); k < n; ++k) sm = fma(Ri[(int64_t)r * n + k], Ri[(int64_t)q * n + k], sm);
          P[(int64_t)q * n + r] = sm;
        }
      }
      __syncthreads();
    }
  }
}

/* ---------------------------------------------------------------------------
 * Small states (n, mmax <= 8), in three kernels.  Only the QR reductions
 * depend on the step before; weighing the equations and turning a factor into
 * an estimate do not, so they run with a thread per step over all tracks and
 * steps, and the chain that is left is two QR reductions a step:
 *   filter_weigh     V [-F | H | c] and W [G | o] of every step
 *   filter_chain     one warp per track, a panel column per lane:
 *                    evolve  [R 0 y; -VF VH Vc] -> the information on x_i
 *                    observe [that; WG Wo] -> R, y
 *   filter_estimate  x = R^{-1} y, P = R^{-1} R^{-T}, in place of the factor
 * A chain step is 2 n reflectors of about 32 FP64 instructions at n = 6, at 64
 * to 76 cycles each: 12 to 14 us, and 16 us with the shuffles between them; with
 * the weighing and the estimate inside the chain it was 42 us.  512 tracks of 50
 * to 500 steps: 21.2 ms before, 8.3 ms now.
 *
 * A round takes kc steps of nt tracks, whose weighed equations must fit the
 * workspace; the factor is carried over between rounds.  Where one round does
 * not hold all, the tracks go by length, the longest first and at most
 * 1/kMinRound of the round's steps at a time, so that the tracks still running
 * are the first of them and their rounds get longer as the others end.  (With
 * kc steps of all tracks in every round, 150,000 tracks of 2 steps and 10 of
 * 1,500 took 1,500 rounds of one step, 117 ms; all in one launch, before the
 * filter was split, 75 ms.)
 * ------------------------------------------------------------------------ */
constexpr int kWarpsPerBlock = 4;
constexpr int kSmallN = 8;
constexpr int64_t kRoundBytes = (int64_t)128 << 20; /* 140,000 steps of 6 states: about what L2 holds */
constexpr int64_t kMinRound = 4; /* steps of a round at least: 33,000 tracks of 6 states, 50 warps a scheduler */

/* entries of a step's weighed equations: columns of [-F | H | c], n rows each,
 * then columns of [G | o], mmax rows each (zero past the step's rows) */
__host__ __device__ constexpr int step_entries(int n, int mmax) { return (2 * n + 1) * n + (n + 1) * mmax; }

struct SmallArgs {
  double* weighed;  /* [nt][kc][step_entries] */
  double* factor;   /* [nt][kc][n * n] where no covariances are asked for, else null: in place of P */
  double* carry;    /* [nt][(n + 1) * n] */
  int* carry_rows;  /* [nt] */
  const int32_t* order; /* the tracks by length, or null: as they are */
  int t0, nt;           /* tracks t0 .. t0 + nt - 1 of them */
  int64_t first, kc;    /* steps first .. first + kc - 1 of each */
  bool more;            /* their next steps follow */
  __device__ __forceinline__ int track(int u) const { return order ? order[t0 + u] : t0 + u; }
};

/* Weighing of one covariance factor by one thread: the lower factor L and the
 * reciprocals d of its diagonal ('C' Cholesky, 'U'/'F' the lower triangle),
 * the matrix ('W') or the weights ('w', in d); rows <= R.                    */
template <int R>
struct ThreadWeights {
  double L[R][R], d[R]; /* L[j][i]: column j, row i */
  char type;

  __device__ __forceinline__ bool prepare(char t, const double* cov, int ld, int rows)
  {
    type = t;
    bool ok = true;
    if (t == 'w') {
#pragma unroll
      for (int i = 0; i < R; ++i) d[i] = i < rows ? cov[i] : 0.0;
      return true;
    }
#pragma unroll
    for (int j = 0; j < R; ++j)
#pragma unroll
      for (int i = 0; i < R; ++i)
        L[j][i] = i < rows && j < rows && (t == 'W' || i >= j) ? cov[(int64_t)j * ld + i] : 0.0;
    if (t == 'W') return true;
#pragma unroll
    for (int j = 0; j < R; ++j) {
      if (t == 'C') {
        double s = L[j][j];
#pragma unroll
        for (int k = 0; k < j; ++k) s = fma(-L[k][j], L[k][j], s);
        const bool pd = s > 0.0;
        if (j < rows && !pd) ok = false;
        d[j] = pd ? lanes::inv_root(s) : 1.0;
#pragma unroll
        for (int i = j + 1; i < R; ++i) {
          double x = L[j][i];
#pragma unroll
          for (int k = 0; k < j; ++k) x = fma(-L[k][i], L[k][j], x);
          L[j][i] = x * d[j];
        }
      } else {
        if (j < rows && L[j][j] == 0.0) ok = false;
        d[j] = j < rows ? lanes::recip(L[j][j]) : 1.0;
      }
    }
    return ok;
  }
  __device__ __forceinline__ void apply(double (&x)[R]) const
  {
    if (type == 'w') {
#pragma unroll
      for (int i = 0; i < R; ++i) x[i] *= d[i];
    } else if (type == 'W') {
      double y[R];
#pragma unroll
      for (int i = 0; i < R; ++i) {
        y[i] = 0.0;
#pragma unroll
        for (int k = 0; k < R; ++k) y[i] = fma(L[k][i], x[k], y[i]);
      }
#pragma unroll
      for (int i = 0; i < R; ++i) x[i] = y[i];
    } else if (type == 'C' || type == 'U' || type == 'F') {
#pragma unroll
      for (int j = 0; j < R; ++j) {
        x[j] *= d[j];
#pragma unroll
        for (int i = j + 1; i < R; ++i) x[i] = fma(-x[j], L[j][i], x[i]);
      }
    }
  }
};

template <int N, int M>
__global__ void __launch_bounds__(64) filter_weigh(FilterArgs a, SmallArgs w)
{
  const int64_t e = (int64_t)blockIdx.x * 64 + threadIdx.x;
  const int u = (int)(e / w.kc);
  if (u >= w.nt) return;
  const int t = w.track(u);
  const int64_t s0 = a.track_start[t], s = s0 + w.first + (e - u * w.kc);
  if (s >= a.track_start[t + 1]) return;
  const int mm = a.mmax;
  const int64_t nn = (int64_t)N * N;
  double* out = w.weighed + e * step_entries(N, mm);
  int flag = 0;
  if (s > s0) {
    ThreadWeights<N> V;
    const char kt = a.K_type[s];
    if (!cta::valid_cov_type(kt)) flag |= 4;
    if (!V.prepare(kt, a.K + s * nn, N, N)) flag |= 1;
#pragma unroll 1
    for (int c = 0; c <= 2 * N; ++c) {
      const double* src = c < N ? a.F + s * nn + c * N : c < 2 * N ? a.H + s * nn + (c - N) * N : a.c + s * N;
      double x[N];
#pragma unroll
      for (int i = 0; i < N; ++i) x[i] = c < N ? -src[i] : src[i];
      V.apply(x);
#pragma unroll
      for (int i = 0; i < N; ++i) out[c * N + i] = x[i];
    }
  }
  int m = a.obs_rows[s];
  if (m < 0 || m > mm) {
    flag |= 4;
    m = 0;
  }
  out += (2 * N + 1) * N;
  if (m == 0) { /* the chain reads all mmax rows */
    for (int i = 0; i < (N + 1) * mm; ++i) out[i] = 0.0;
  } else {
    ThreadWeights<M> W;
    const char ct = a.C_type[s];
    if (!cta::valid_cov_type(ct)) flag |= 4;
    if (!W.prepare(ct, a.C + s * (int64_t)mm * mm, mm, m)) flag |= 1;
#pragma unroll 1
    for (int c = 0; c <= N; ++c) {
      const double* src = c < N ? a.G + s * (int64_t)mm * N + (int64_t)c * mm : a.o + s * mm;
      double x[M];
#pragma unroll
      for (int i = 0; i < M; ++i) x[i] = i < m ? src[i] : 0.0;
      W.apply(x);
#pragma unroll
      for (int i = 0; i < M; ++i)
        if (i < mm) out[c * mm + i] = i < m ? x[i] : 0.0;
    }
  }
  if (flag) atomicOr(a.flag, flag);
}

/* The factor's z rows (all n in the usual case) are carried on lanes 0..N
 * ([R | y], zero rows past z).  The weighed evolution goes on top of them: where
 * the process noise is small its rows are the large ones, and with the factor on
 * top the information on x_i, what is left in the lower rows of the columns
 * N..2N, would be small differences of large numbers (a covariance error of
 * 1.7e-8 instead of 1.4e-15 with noise of variance 1e-14).  Zero rows of the
 * factor stay exactly zero.                                                  */
template <int N, int M>
__global__ void __launch_bounds__(32 * kWarpsPerBlock) filter_chain(FilterArgs a, SmallArgs w)
{
  const int lane = threadIdx.x & 31;
  /* tracks by length: a long one with shorter ones on an SM, whose four
     schedulers share the FP64 pipe                                         */
  const int u = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
  if (u >= w.nt) return; /* the whole warp */
  const unsigned all = 0xffffffffu;
  const int t = w.track(u), mm = a.mmax, per = step_entries(N, mm);
  const int64_t s0 = a.track_start[t] + w.first;
  const int64_t cnt = a.track_start[t + 1] - s0 < w.kc ? a.track_start[t + 1] - s0 : w.kc;
  if (cnt <= 0) return;
  double R[N]; /* this lane's column of [R | y] */
  int z = 0;
#pragma unroll
  for (int r = 0; r < N; ++r) R[r] = 0.0;
  if (w.first > 0) {
    z = w.carry_rows[u];
    if (lane <= N)
#pragma unroll
      for (int r = 0; r < N; ++r) R[r] = w.carry[((int64_t)u * (N + 1) + lane) * N + r];
  }
  const double* in = w.weighed + (int64_t)u * w.kc * per;
  const int64_t nn = (int64_t)N * N;
  double e[N], g[M]; /* the step's columns, loaded a step ahead */
  int m = 0;
  auto load = [&](int64_t q) {
    const double* p = in + q * per;
    if (lane <= 2 * N && (w.first > 0 || q > 0))
#pragma unroll
      for (int r = 0; r < N; ++r) e[r] = p[lane * N + r];
    if (lane <= N)
#pragma unroll
      for (int r = 0; r < M; ++r)
        if (r < mm) g[r] = p[(2 * N + 1) * N + lane * mm + r];
    m = a.obs_rows[s0 + q];
    if (m < 0 || m > mm) m = 0; /* reported by the weighing */
  };
#pragma unroll
  for (int r = 0; r < N; ++r) e[r] = 0.0;
#pragma unroll
  for (int r = 0; r < M; ++r) g[r] = 0.0;
  load(0);
  for (int64_t q = 0; q < cnt; ++q) {
    double tp[1][N], bt[1][N], bo[1][M];
    const int mq = m;
#pragma unroll
    for (int r = 0; r < N; ++r) {
      const double y = __shfl_sync(all, R[r], N);
      tp[0][r] = e[r];
      bt[0][r] = lane < N ? R[r] : lane == 2 * N ? y : 0.0;
    }
#pragma unroll
    for (int r = 0; r < M; ++r) bo[0][r] = g[r];
    if (q + 1 < cnt) load(q + 1);
    if (w.first + q > 0) {
      lanes::lanes_qr_full<double, N, 32, 1, N>(tp, bt, all, lane, 0, N);
#pragma unroll
      for (int r = 0; r < N; ++r) {
        const double v = __shfl_sync(all, bt[0][r], (lane + N) & 31);
        tp[0][r] = lane <= N ? v : 0.0;
      }
    } else { /* a track's first step has no evolution */
#pragma unroll
      for (int r = 0; r < N; ++r) tp[0][r] = 0.0;
    }
    /* with fewer than N rows the observation's follow them without a gap: a
       column of zeros takes no reflector, so a row past a gap might never be
       brought up                                                           */
#pragma unroll 1
    for (int d = z; d < N; ++d) {
#pragma unroll
      for (int r = 0; r + 1 < N + M; ++r)
        if (r >= z) (r < N ? tp[0][r] : bo[0][r - N]) = r + 1 < N ? tp[0][r + 1] : bo[0][r + 1 - N];
      bo[0][M - 1] = 0.0;
    }
    z = z + mq < N ? z + mq : N;
    lanes::lanes_qr_full<double, N, 32, 1, M>(tp, bo, all, lane, 0, z);
    double* Ro = a.cov ? a.cov + (s0 + q) * nn : w.factor + ((int64_t)u * w.kc + q) * nn;
#pragma unroll
    for (int r = 0; r < N; ++r) R[r] = lane <= N && r <= lane && r < z ? tp[0][r] : 0.0;
    double* out = lane < N ? Ro + lane * N : a.state + (s0 + q) * N;
    if (lane <= N)
#pragma unroll
      for (int r = 0; r < N; ++r) out[r] = R[r];
  }
  if (!w.more) return;
  if (lane <= N)
#pragma unroll
    for (int r = 0; r < N; ++r) w.carry[((int64_t)u * (N + 1) + lane) * N + r] = R[r];
  if (lane == 0) w.carry_rows[u] = z;
}

/* x = R^{-1} y and P = R^{-1} R^{-T} of a step, over the factor that the chain
 * left in the outputs; a zero on R's diagonal (fewer than n rows, or a zero
 * pivot) is an undetermined state                                           */
template <int N>
__global__ void __launch_bounds__(64) filter_estimate(FilterArgs a, SmallArgs w)
{
  const int64_t e = (int64_t)blockIdx.x * 64 + threadIdx.x;
  const int u = (int)(e / w.kc);
  if (u >= w.nt) return;
  const int t = w.track(u);
  const int64_t s = a.track_start[t] + w.first + (e - u * w.kc);
  if (s >= a.track_start[t + 1]) return;
  const int64_t nn = (int64_t)N * N;
  double* P = a.cov ? a.cov + s * nn : nullptr;
  const double* Rp = P ? P : w.factor + e * nn;
  double* x = a.state + s * N;
  double R[N][N], d[N], y[N]; /* R[j][i]: column j, row i <= j */
  bool det = true;
#pragma unroll
  for (int j = 0; j < N; ++j) {
    y[j] = x[j];
#pragma unroll
    for (int i = 0; i <= j; ++i) R[j][i] = Rp[j * N + i];
    det = det && R[j][j] != 0.0;
  }
  if (!det) {
    for (int i = 0; i < N; ++i) x[i] = NAN;
    if (P)
      for (int i = 0; i < N * N; ++i) P[i] = NAN;
    atomicOr(a.flag, 1);
    return;
  }
#pragma unroll
  for (int j = 0; j < N; ++j) d[j] = lanes::recip(R[j][j]);
#pragma unroll
  for (int j = N - 1; j >= 0; --j) {
    y[j] *= d[j];
#pragma unroll
    for (int i = 0; i < j; ++i) y[i] = fma(-y[j], R[j][i], y[i]);
  }
#pragma unroll
  for (int i = 0; i < N; ++i) x[i] = y[i];
  if (!P) return;
  /* R <- R^{-1} column by column (column j of the inverse needs R's columns up to j), last column first */
#pragma unroll
  for (int j = N - 1; j >= 0; --j) {
    double u[N];
    u[j] = d[j];
#pragma unroll
    for (int i = 0; i < j; ++i) u[i] = -R[j][i] * d[j];
#pragma unroll
    for (int k = j - 1; k >= 0; --k) {
      u[k] *= d[k];
#pragma unroll
      for (int i = 0; i < k; ++i) u[i] = fma(-u[k], R[k][i], u[i]);
    }
#pragma unroll
    for (int i = 0; i <= j; ++i) R[j][i] = u[i];
  }
#pragma unroll
  for (int j = 0; j < N; ++j)
#pragma unroll
    for (int i = j; i < N; ++i) {
      double sm = 0.0;
#pragma unroll
      for (int k = i; k < N; ++k) sm = fma(R[k][i], R[k][j], sm);
      P[j * N + i] = sm;
      P[i * N + j] = sm;
    }
}

/* the tracks, the longest first: by counting, and by comparison past 65,535 steps */
bool by_length(const int64_t* start, int ntracks, int64_t longest, std::vector<int32_t>& order)
{
  try {
    const int64_t top = std::min<int64_t>(longest, 65535);
    auto len = [&](int t) { return start[t + 1] - start[t]; };
    auto bucket = [&](int t) { return top - std::min(len(t), top); };
    std::vector<int32_t> at(top + 2, 0);
    for (int t = 0; t < ntracks; ++t) ++at[bucket(t) + 1];
    std::partial_sum(at.begin(), at.end(), at.begin());
    const int32_t longer = at[1];
    order.resize(ntracks);
    for (int t = 0; t < ntracks; ++t) order[at[bucket(t)]++] = t;
    if (longest > top) std::sort(order.begin(), order.begin() + longer, [&](int32_t x, int32_t y) { return len(x) > len(y); });
    return true;
  } catch (const std::bad_alloc&) {
    return false;
  }
}

/* The rounds of a call that one round does not hold: len(i) is the length of the
 * i-th track, the longest first, steps what a round holds; round(t0, nt, first,
 * kc, more), more: the same tracks' next steps follow.                       */
template <class LEN, class F>
void rounds(int ntracks, int64_t steps, LEN len, F round)
{
  for (int t0 = 0, nt; t0 < ntracks && len(t0) > 0; t0 += nt) {
    const int64_t longest = len(t0);
    nt = (int)std::min<int64_t>(ntracks - t0, std::max<int64_t>(1, steps / std::min(longest, kMinRound)));
    int on = nt; /* still running */
    for (int64_t first = 0, kc; first < longest; first += kc) {
      while (len(t0 + on - 1) <= first) --on;
      kc = std::min(longest - first, std::max<int64_t>(1, steps / on));
      round(t0, on, first, kc, first + kc < longest);
    }
  }
}

template <int N, int M>
void filter_small_nm(const FilterArgs& a, const SmallArgs& w, cudaStream_t st)
{
  const unsigned chain = (unsigned)((w.nt + kWarpsPerBlock - 1) / kWarpsPerBlock);
  const unsigned steps = (unsigned)((w.nt * w.kc + 63) / 64);
  UKG_LAUNCH(UKG_K_FILTER, st, (filter_weigh<N, M><<<steps, 64, 0, st>>>(a, w)));
  UKG_LAUNCH(UKG_K_FILTER, st, (filter_chain<N, M><<<chain, 32 * kWarpsPerBlock, 0, st>>>(a, w)));
  UKG_LAUNCH(UKG_K_FILTER, st, (filter_estimate<N><<<steps, 64, 0, st>>>(a, w)));
}
/* observation rows in registers: half of n, n or 8 */
template <int N>
void filter_small_n(const FilterArgs& a, const SmallArgs& w, cudaStream_t st)
{
  if (a.mmax <= (N + 1) / 2) filter_small_nm<N, (N + 1) / 2>(a, w, st);
  else if (a.mmax <= N) filter_small_nm<N, N>(a, w, st);
  else filter_small_nm<N, kSmallN>(a, w, st);
}
void filter_small(const FilterArgs& a, const SmallArgs& w, cudaStream_t st)
{
  switch (a.n) {
    case 1: filter_small_n<1>(a, w, st); break;
    case 2: filter_small_n<2>(a, w, st); break;
    case 3: filter_small_n<3>(a, w, st); break;
    case 4: filter_small_n<4>(a, w, st); break;
    case 5: filter_small_n<5>(a, w, st); break;
    case 6: filter_small_n<6>(a, w, st); break;
    case 7: filter_small_n<7>(a, w, st); break;
    default: filter_small_n<8>(a, w, st); break;
  }
}

struct Workspace {
  void* p = nullptr;
  size_t bytes = 0;
};
thread_local Workspace tl_ws;

int ensure(size_t bytes)
{
  if (tl_ws.bytes >= bytes) return 0;
  if (tl_ws.p) cudaFree(tl_ws.p);
  tl_ws.p = nullptr;
  tl_ws.bytes = 0;
  if (cudaMalloc(&tl_ws.p, bytes) != cudaSuccess) {
    cudaGetLastError();
    return ukg_set_error(KALMAN_GPU_ENOMEM, "filter workspace of %zu bytes", bytes);
  }
  tl_ws.bytes = bytes;
  return 0;
}

}  // namespace

extern "C" int64_t ukg_filter_workspace_held(void) { return (int64_t)tl_ws.bytes; }

extern "C" void ukg_release_filter_workspace(void)
{
  if (tl_ws.p) cudaFree(tl_ws.p);
  tl_ws = Workspace{};
}

extern "C" int kalman_gpu_filter_packed(uint32_t options, const kalman_gpu_problem_t* p, void* cuda_stream)
{
  ukg_clear_error();
  const bool want_cov = !(options & (1u << 16)) && p && p->covariance;
  if (int e = ukg_validate_problem(p, 0)) return e;
  if (p->location != KALMAN_GPU_DEVICE)
    return ukg_set_error(KALMAN_GPU_EINVAL, "filter: the problem's arrays must be device arrays");
  if (p->n > cta::kMaxCov || p->mmax > cta::kMaxCov)
    return ukg_set_error(KALMAN_GPU_EINVAL, "filter: state dimension %d / observation rows %d above %d", p->n,
                         p->mmax, cta::kMaxCov);
  if (p->nsteps == 0) return KALMAN_GPU_OK;
  cudaStream_t st = (cudaStream_t)cuda_stream;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int ncta = p->ntracks < sms * 4 ? p->ntracks : sms * 4;
  const int64_t per = filter_scratch(p->n, p->mmax);
  const size_t tab = ((size_t)(p->ntracks + 1) * sizeof(int64_t) + 255) / 256 * 256;
  const bool small = p->n <= kSmallN && p->mmax <= kSmallN;
  SmallArgs w;
  memset(&w, 0, sizeof(w));
  size_t scratch = (size_t)ncta * per;
  /* the rounds: of one, or of the tracks by length */
  std::vector<int32_t> order;
  auto len = [&](int i) {
    const int t = order.empty() ? i : order[i];
    return p->track_start[t + 1] - p->track_start[t];
  };
  int64_t round_steps = 0, whole = 0, carried = 0;
  const int64_t step = step_entries(p->n, p->mmax) + (want_cov ? 0 : p->n * p->n);
  const int64_t carry = (p->n + 1) * (int64_t)p->n + 1; /* and the number of rows */
  if (small) {
    const int64_t hold = kRoundBytes / ((int64_t)sizeof(double) * (step + (carry + kMinRound - 1) / kMinRound));
    int64_t longest = 0;
    bool sorted = true;
    for (int t = 0; t < p->ntracks; ++t) {
      sorted = sorted && (t == 0 || len(t) <= len(t - 1));
      longest = std::max<int64_t>(longest, len(t));
    }
    if (longest <= hold / p->ntracks) {
      whole = longest;
      round_steps = p->ntracks * longest;
    } else {
      if (!sorted && !by_length(p->track_start, p->ntracks, longest, order))
        return ukg_set_error(KALMAN_GPU_ENOMEM, "filter: the order of %d tracks", p->ntracks);
      round_steps = hold;
      rounds(p->ntracks, hold, len, [&](int, int nt, int64_t, int64_t, bool more) {
        if (more) carried = std::max<int64_t>(carried, nt);
      });
    }
    scratch = (size_t)(round_steps * step + carried * carry) + (order.size() + 1) / 2;
  }
  if (int e = ensure(tab + 256 + scratch * sizeof(double))) return e;
  char* base = (char*)tl_ws.p;
  int64_t* dts = (int64_t*)base;
  int* dflag = (int*)(base + tab);
  cudaMemcpyAsync(dts, p->track_start, (size_t)(p->ntracks + 1) * sizeof(int64_t), cudaMemcpyHostToDevice, st);
  cudaMemsetAsync(dflag, 0, sizeof(int), st);
  FilterArgs a;
  a.n = p->n;
  a.mmax = p->mmax;
  a.ntracks = p->ntracks;
  a.track_start = dts;
  a.H = p->H;
  a.F = p->F;
  a.c = p->c;
  a.K = p->K;
  a.G = p->G;
  a.o = p->o;
  a.C = p->C;
  a.K_type = p->K_type;
  a.C_type = p->C_type;
  a.obs_rows = p->obs_rows;
  a.state = p->state;
  a.cov = want_cov ? p->covariance : nullptr;
  a.scratch = (double*)(base + tab + 256);
  a.per_cta = per;
  a.flag = dflag;
  if (small) {
    w.weighed = a.scratch;
    w.carry = w.weighed + round_steps * step;
    w.carry_rows = (int*)(w.carry + carried * (carry - 1));
    if (!order.empty()) {
      int32_t* dorder = (int32_t*)(w.carry + carried * carry);
      cudaMemcpyAsync(dorder, order.data(), order.size() * sizeof(int32_t), cudaMemcpyHostToDevice, st);
      w.order = dorder;
    }
    auto round = [&](int t0, int nt, int64_t first, int64_t kc, bool more) {
      w.t0 = t0, w.nt = nt, w.first = first, w.kc = kc, w.more = more;
      w.factor = w.weighed + nt * kc * step_entries(p->n, p->mmax); /* used without covariances only */
      filter_small(a, w, st);
    };
    if (whole) round(0, p->ntracks, 0, whole, false);
    else rounds(p->ntracks, round_steps, len, round);
  } else {
    UKG_LAUNCH(UKG_K_FILTER, st, (filter_cta<<<ncta, NT, 0, st>>>(a)));
  }
  int hflag = 0;
  cudaMemcpyAsync(&hflag, dflag, sizeof(int), cudaMemcpyDeviceToHost, st);
  cudaError_t e = cudaStreamSynchronize(st);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) return ukg_set_error(KALMAN_GPU_ECUDA, "filter: %s", cudaGetErrorString(e));
  if (hflag & 4) return ukg_set_error(KALMAN_GPU_EINVAL, "filter: malformed input (observation rows or covariance types)");
  if (hflag & 1)
    return ukg_set_error(KALMAN_GPU_ESINGULAR, "filter: some steps' states are not yet determined (NaN written there)");
  return KALMAN_GPU_OK;
}
