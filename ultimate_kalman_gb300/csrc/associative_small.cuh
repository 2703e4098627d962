/*
 * associative_small.cuh -- the scans of the associative smoother for up to 8
 * states, a warp (or half of one) per combine, up to 5 states a thread where
 * there are many.  Included by associative.cu (it uses that file's FElems,
 * SElems, ScanLevel and find_track).
 *
 * A thread that combines two elements alone is a chain of some 2,700 FP64
 * instructions of 64 cycles (175 us a level, whatever its size); with a matrix
 * column per lane the chain is about 250 for the filtering operation -- both
 * of its solves on the two halves of the warp at once -- and 75 for the
 * smoothing one.  Matrices go through shared memory between the products, and
 * all of an element is read before any of the result is written, so the
 * result may replace the right operand.
 */
#pragma once

namespace asmall {

constexpr int kWarps = 4; /* warps per block: one per scheduler */

/* Elements are arrays of entries with one stride: A, Z, J, b, e (or E, L, g)
 * follow one another, so column c of [A | Z | J | b | e] is entries c N ..   */
template <int N>
__device__ __forceinline__ void load_col(const Soa& first, int c, int64_t s, double (&v)[N])
{
  const double* p = first.p + (int64_t)c * N * first.stride + s;
#pragma unroll
  for (int i = 0; i < N; ++i, p += first.stride) v[i] = *p;
}
template <int N>
__device__ __forceinline__ void store_col(const Soa& first, int c, int64_t s, const double (&v)[N])
{
  double* p = first.p + (int64_t)c * N * first.stride + s;
#pragma unroll
  for (int i = 0; i < N; ++i, p += first.stride) *p = v[i];
}

/* out <- init + M v for the column-major M (n x n) in shared memory */
template <int N>
__device__ __forceinline__ void matvec(const double* M, const double (&v)[N], double (&out)[N])
{
#pragma unroll
  for (int k = 0; k < N; ++k)
#pragma unroll
    for (int p = 0; p < N; ++p) out[p] = fma(M[k * N + p], v[k], out[p]);
}

/* Householder QR of square panels, a column per lane, the pivots on the lanes
 * base .. base + N - 1                                                       */
template <int N>
__device__ __forceinline__ void qr_square(double (&t)[N], int lane, int base)
{
#pragma unroll
  for (int k = 0; k + 1 < N; ++k) {
    const int src = base + k;
    double x[N], dot = 0.0;
    const double alpha = __shfl_sync(0xffffffffu, t[k], src);
#pragma unroll
    for (int i = k + 1; i < N; ++i) x[i] = __shfl_sync(0xffffffffu, t[i], src);
#pragma unroll
    for (int i = k + 1; i < N; ++i) dot = fma(x[i], t[i], dot);
    const double tail = __shfl_sync(0xffffffffu, dot, src);
    if (tail != 0.0) {
      const lanes::Refl<double> r = lanes::reflector(alpha, tail);
      const double d = fma(r.amb, t[k], dot) * r.inv;
      t[k] = lane == src ? r.beta : fma(-d, r.amb, t[k]);
#pragma unroll
      for (int i = k + 1; i < N; ++i) t[i] = fma(-d, x[i], t[i]);
    }
  }
}

template <int N>
struct FBuf { /* both operands, [A | Z | J | b | e] column by column; X, Y; R of the two solves, then T */
  double i[(3 * N + 2) * N], j[(3 * N + 2) * N], X[N * N], Y[N * N], R[2 * N * N];
};

/* filteringAssociativeOperation on the operands in B (see combine_filter):
 * X = Aj (I + Zi Jj)^{-1}, Y = Ai^T (I + Jj Zi)^{-1},
 * A = X Ai, b = X (bi + Zi ej) + bj, Z = X Zi Aj^T + Zj,
 * e = Y (ej - Jj bi) + ei, J = Y Jj Ai + Ji.  Run by a whole warp.           */
template <int N>
__device__ __forceinline__ bool combine_lanes(FBuf<N>& B, int lane, const FElems& O, int64_t o)
{
  constexpr int NN = N * N;
  const double *Ai = B.i, *Zi = B.i + NN, *Ji = B.i + 2 * NN, *bi = B.i + 3 * NN, *ei = bi + N;
  const double *Aj = B.j, *Zj = B.j + NN, *Jj = B.j + 2 * NN, *bj = B.j + 3 * NN, *ej = bj + N;
  const int half = lane >= 2 * N ? 1 : 0, base = half * 2 * N, c = lane - base; /* column of [pivots | rhs] */
  const bool live = lane < 4 * N, piv = live && c < N;
  const int q = c < N ? c : c < 2 * N ? c - N : 0;
  double t[N], v[N];
  { /* pivots: column q of (I + Zi Jj)^T, or of (I + Jj Zi)^T: row q of the product */
    const double *L = half ? Jj : Zi, *Rm = half ? Zi : Jj;
#pragma unroll
    for (int k = 0; k < N; ++k) v[k] = L[k * N + q];
#pragma unroll
    for (int p = 0; p < N; ++p) {
      t[p] = p == q ? 1.0 : 0.0;
#pragma unroll
      for (int k = 0; k < N; ++k) t[p] = fma(v[k], Rm[p * N + k], t[p]);
    }
    if (!piv) /* right-hand sides: column q of Aj^T, or of Ai */
#pragma unroll
      for (int p = 0; p < N; ++p) t[p] = half ? Ai[q * N + p] : Aj[p * N + q];
  }
  qr_square<N>(t, lane, base);
  double* R = B.R + half * NN;
  if (piv)
#pragma unroll
    for (int p = 0; p < N; ++p) R[q * N + p] = t[p];
  __syncwarp();
  const double dg = R[q * N + q];
  const bool bad = live && dg == 0.0;
  const double dv = lanes::recip(dg);
#pragma unroll
  for (int k = N - 1; k >= 0; --k) {
    t[k] *= __shfl_sync(0xffffffffu, dv, base + k);
#pragma unroll
    for (int p = 0; p < k; ++p) t[p] = fma(-t[k], R[k * N + p], t[p]);
  }
  if (live && !piv) { /* column q of X^T (Y^T) is row q of X (Y) */
    double* X = half ? B.Y : B.X;
#pragma unroll
    for (int p = 0; p < N; ++p) X[p * N + q] = t[p];
  }
  __syncwarp();
  /* columns of T = X Zi, A = X Ai, T2 = Jj Ai; the vectors bi + Zi ej and ej - Jj bi */
  const int g = lane < 3 * N ? lane / N : 3, cq = lane - g * N; /* g = 3: cq 0, 1 are the vectors */
  const bool vec = g == 3 && cq < 2;
  {
    const double* src = g == 0 ? Zi + cq * N : g < 3 ? Ai + cq * N : cq == 0 ? ej : bi;
    const double* init = cq == 0 ? bi : ej;
#pragma unroll
    for (int k = 0; k < N; ++k) {
      v[k] = vec || g < 3 ? src[k] : 0.0;
      if (g == 3 && cq == 1) v[k] = -v[k];
      t[k] = vec ? init[k] : 0.0;
    }
    matvec<N>(g < 2 ? B.X : g == 2 || cq == 1 ? Jj : Zi, v, t);
  }
  double* T = B.R; /* R is spent */
  if (g == 0)
#pragma unroll
    for (int p = 0; p < N; ++p) T[cq * N + p] = t[p];
  if (g == 1) store_col<N>(O.A, cq, o, t);
  __syncwarp();
  /* columns of Z = T Aj^T + Zj, J = Y T2 + Ji; b = X (.) + bj, e = Y (.) + ei */
  {
    const double* init = g == 0 ? Zj + cq * N : g == 2 ? Ji + cq * N : cq == 0 ? bj : ei;
    double out[N];
#pragma unroll
    for (int k = 0; k < N; ++k) {
      v[k] = g == 0 ? Aj[k * N + cq] : t[k];
      out[k] = g == 0 || g == 2 || vec ? init[k] : 0.0;
    }
    matvec<N>(g == 0 ? T : g == 3 && cq == 0 ? B.X : B.Y, v, out);
    /* entries of O: Z at column N + cq, J at 2 N + cq, b at 3 N, e at 3 N + 1 */
    if (g == 0 || g == 2 || vec) store_col<N>(O.A, g == 0 ? N + cq : g == 2 ? 2 * N + cq : 3 * N + cq, o, out);
  }
  return bad;
}

/* columns of element s: lanes 0..3N+1 (n = 8: 26 lanes) */
template <int N>
__device__ __forceinline__ void fetch(const FElems& X, int64_t s, int lane, double* to)
{
  if (lane < 3 * N + 2) {
    double v[N];
    load_col<N>(X.A, lane, s, v);
#pragma unroll
    for (int i = 0; i < N; ++i) to[lane * N + i] = v[i];
  }
}
template <int N>
__device__ __forceinline__ void copy(const Soa& X, int64_t s, const Soa& O, int64_t o, int col, bool on)
{
  double v[N];
  if (!on) return;
  load_col<N>(X, col, s, v);
  store_col<N>(O, col, o, v);
}

template <int N>
__global__ void __launch_bounds__(32 * kWarps) up_filter(int T, ScanLevel lv, ScanLevel nx, FElems cur, FElems nxt,
                                                         int* flag)
{
  __shared__ FBuf<N> bufs[kWarps];
  const int lane = threadIdx.x & 31;
  const int64_t item = (int64_t)blockIdx.x * kWarps + (threadIdx.x >> 5);
  if (item >= lv.nup) return; /* the whole warp */
  FBuf<N>& B = bufs[threadIdx.x >> 5];
  const int t = find_track(lv.up_items, T, item);
  const int64_t p = item - lv.up_items[t], s0 = lv.start[t] + 2 * p, o = nx.start[t] + p;
  if (2 * p + 1 >= lv.L[t]) {
    copy<N>(cur.A, s0, nxt.A, o, lane, lane < 3 * N + 2);
    return;
  }
  fetch<N>(cur, s0, lane, B.i);
  fetch<N>(cur, s0 + 1, lane, B.j);
  __syncwarp();
  if (combine_lanes<N>(B, lane, nxt, o)) atomicOr(flag, 2);
}

template <int N>
__global__ void __launch_bounds__(32 * kWarps) down_filter(int T, ScanLevel lv, ScanLevel nx, FElems cur, FElems nxt,
                                                           int* flag)
{
  __shared__ FBuf<N> bufs[kWarps];
  const int lane = threadIdx.x & 31;
  const int64_t item = (int64_t)blockIdx.x * kWarps + (threadIdx.x >> 5);
  if (item >= lv.ndown) return; /* the whole warp */
  FBuf<N>& B = bufs[threadIdx.x >> 5];
  const int t = find_track(lv.down_items, T, item);
  const int64_t p = item - lv.down_items[t], L = lv.L[t];
  if (L < 2) return; /* a one-element sequence is its own prefix */
  const int64_t s0 = lv.start[t] + 2 * p, b0 = nx.start[t] + p;
  copy<N>(nxt.A, b0, cur.A, s0 + 1, lane, 2 * p + 1 < L && lane < 3 * N + 2);
  if (p == 0) return;
  fetch<N>(nxt, b0 - 1, lane, B.i);
  fetch<N>(cur, s0, lane, B.j);
  __syncwarp();
  if (combine_lanes<N>(B, lane, cur, s0)) atomicOr(flag, 2);
}

/* ---------------------------------------------------------------------------
 * the smoothing operation (see combine_smooth): E = Ej Ei, g = Ej gi + gj,
 * L = Ej Li Ej^T + Lj.  A half-warp per combine up to 7 states: columns of
 * Ej Li on lanes 0..N-1, of Ej Ei on N..2N-1, Ej gi + gj on 2N.
 * ------------------------------------------------------------------------ */
template <int N>
struct SmoothGroup {
  static constexpr int lanes = 2 * N + 1 <= 16 ? 16 : 32, per_block = 32 * kWarps / lanes;
  struct Buf {
    double E[N * N], T[N * N];
  };
};
template <int N>
__device__ __forceinline__ void combine_smooth_lanes(typename SmoothGroup<N>::Buf& B, int lane, unsigned gm,
                                                     const SElems& Xi, int64_t i, const SElems& Xj, int64_t j,
                                                     const SElems& O, int64_t o)
{
  const bool isL = lane < N, isE = !isL && lane < 2 * N, isg = lane == 2 * N;
  double v[N], init[N], ej[N];
  /* columns of [E | L | g]: E at 0, L at N, g at 2 N */
  load_col<N>(Xi.E, isL ? N + lane : isE ? lane - N : 2 * N, i, v);
  load_col<N>(Xj.E, isL ? N + lane : 2 * N, j, init); /* Lj's column, or gj */
  load_col<N>(Xj.E, isL ? lane : 0, j, ej);
  if (isL)
#pragma unroll
    for (int p = 0; p < N; ++p) B.E[lane * N + p] = ej[p];
  __syncwarp(gm);
  double t[N];
#pragma unroll
  for (int p = 0; p < N; ++p) t[p] = isg ? init[p] : 0.0;
  matvec<N>(B.E, v, t);
  if (isL)
#pragma unroll
    for (int p = 0; p < N; ++p) B.T[lane * N + p] = t[p];
  __syncwarp(gm);
  if (isE || isg) store_col<N>(O.E, isE ? lane - N : 2 * N, o, t);
  if (!isL) return;
#pragma unroll
  for (int k = 0; k < N; ++k) v[k] = B.E[k * N + lane]; /* row `lane` of Ej */
  matvec<N>(B.T, v, init);
  store_col<N>(O.E, N + lane, o, init);
}

template <int N>
__global__ void __launch_bounds__(32 * kWarps) up_smooth(int T, ScanLevel lv, ScanLevel nx, SElems cur, SElems nxt)
{
  using G = SmoothGroup<N>;
  __shared__ typename G::Buf bufs[G::per_block];
  const int grp = threadIdx.x / G::lanes, lane = threadIdx.x % G::lanes;
  const unsigned gm = G::lanes == 32 ? 0xffffffffu : 0xffffu << (threadIdx.x & 16);
  const int64_t item = (int64_t)blockIdx.x * G::per_block + grp;
  if (item >= lv.nup) return; /* the whole group */
  const int t = find_track(lv.up_items, T, item);
  const int64_t p = item - lv.up_items[t], s0 = lv.start[t] + 2 * p, o = nx.start[t] + p;
  if (2 * p + 1 >= lv.L[t]) copy<N>(cur.E, s0, nxt.E, o, lane, lane < 2 * N + 1);
  else combine_smooth_lanes<N>(bufs[grp], lane, gm, cur, s0, cur, s0 + 1, nxt, o);
}

template <int N>
__global__ void __launch_bounds__(32 * kWarps) down_smooth(int T, ScanLevel lv, ScanLevel nx, SElems cur, SElems nxt)
{
  using G = SmoothGroup<N>;
  __shared__ typename G::Buf bufs[G::per_block];
  const int grp = threadIdx.x / G::lanes, lane = threadIdx.x % G::lanes;
  const unsigned gm = G::lanes == 32 ? 0xffffffffu : 0xffffu << (threadIdx.x & 16);
  const int64_t item = (int64_t)blockIdx.x * G::per_block + grp;
  if (item >= lv.ndown) return; /* the whole group */
  const int t = find_track(lv.down_items, T, item);
  const int64_t p = item - lv.down_items[t], L = lv.L[t];
  if (L < 2) return;
  const int64_t s0 = lv.start[t] + 2 * p, b0 = nx.start[t] + p;
  copy<N>(nxt.E, b0, cur.E, s0 + 1, lane, 2 * p + 1 < L && lane < 2 * N + 1);
  if (p > 0) combine_smooth_lanes<N>(bufs[grp], lane, gm, nxt, b0 - 1, cur, s0, cur, s0);
}

/* ---------------------------------------------------------------------------
 * The same combines by a thread each, its operations on every entry those of the
 * lanes, so that the number of items changes no bit: for levels of many items up
 * to 5 states.  A warp's instruction costs the same whether 4 N or 32 of its
 * lanes have work: 1,000 tracks of 1,000 steps, n = 1 to 5, by lanes alone 2.4,
 * 7.4, 14.7, 24.3 and 38.4 ms, now 0.9, 2.2, 5.3, 10.5 and 20.6 (a thread per
 * combine with its matrices in shared memory 1.1, 2.9, 7.9, 16.8 and 37.2).
 * From 6 states on the matrices do not fit a thread's registers.
 * ------------------------------------------------------------------------ */
constexpr int kThreads = 64;

template <int N>
__device__ __forceinline__ double at(const Soa& first, int c, int r, int64_t s)
{
  return first.p[(int64_t)(c * N + r) * first.stride + s];
}
template <int N>
__device__ __forceinline__ void load_mat(const Soa& first, int c, int64_t s, double (&M)[N][N])
{
#pragma unroll
  for (int k = 0; k < N; ++k)
#pragma unroll
    for (int r = 0; r < N; ++r) M[k][r] = at<N>(first, c + k, r, s);
}
/* out <- out + M v */
template <int N>
__device__ __forceinline__ void matvec(const double (&M)[N][N], const double (&v)[N], double (&out)[N])
{
#pragma unroll
  for (int k = 0; k < N; ++k)
#pragma unroll
    for (int p = 0; p < N; ++p) out[p] = fma(M[k][p], v[k], out[p]);
}

/* X <- B^T (I + L R)^{-1}, B in the columns X on entry; false: a zero pivot */
template <int N>
__device__ __forceinline__ bool solve_thread(const double (&L)[N][N], const double (&R)[N][N], double (&X)[N][N])
{
  double t[2 * N][N], dv[N];
#pragma unroll
  for (int q = 0; q < N; ++q)
#pragma unroll
    for (int p = 0; p < N; ++p) {
      t[q][p] = p == q ? 1.0 : 0.0;
#pragma unroll
      for (int k = 0; k < N; ++k) t[q][p] = fma(L[k][q], R[p][k], t[q][p]);
      t[N + q][p] = X[q][p];
    }
#pragma unroll
  for (int k = 0; k + 1 < N; ++k) {
    double tail = 0.0;
#pragma unroll
    for (int i = k + 1; i < N; ++i) tail = fma(t[k][i], t[k][i], tail);
    if (tail == 0.0) continue;
    const lanes::Refl<double> r = lanes::reflector(t[k][k], tail);
    t[k][k] = r.beta;
#pragma unroll
    for (int c = k + 1; c < 2 * N; ++c) {
      double d = 0.0;
#pragma unroll
      for (int i = k + 1; i < N; ++i) d = fma(t[k][i], t[c][i], d);
      d = fma(r.amb, t[c][k], d) * r.inv;
      t[c][k] = fma(-d, r.amb, t[c][k]);
#pragma unroll
      for (int i = k + 1; i < N; ++i) t[c][i] = fma(-d, t[k][i], t[c][i]);
    }
  }
  bool ok = true;
#pragma unroll
  for (int k = 0; k < N; ++k) {
    ok = ok && t[k][k] != 0.0;
    dv[k] = lanes::recip(t[k][k]);
  }
#pragma unroll
  for (int q = 0; q < N; ++q)
#pragma unroll
    for (int k = N - 1; k >= 0; --k) {
      t[N + q][k] *= dv[k];
      X[k][q] = t[N + q][k];
#pragma unroll
      for (int p = 0; p < k; ++p) t[N + q][p] = fma(-t[N + q][k], t[k][p], t[N + q][p]);
    }
  return ok;
}

/* combine_lanes' formulas; all of Xj is read before the entries it shares with
 * O are written                                                              */
template <int N>
__device__ __forceinline__ bool combine_thread(const FElems& Xi, int64_t i, const FElems& Xj, int64_t j, const FElems& O,
                                               int64_t o)
{
  double Zi[N][N], Jj[N][N], X[N][N], Y[N][N], T[N][N], v1[N], v2[N], v[N];
  load_mat<N>(Xi.A, N, i, Zi);
  load_mat<N>(Xj.A, 2 * N, j, Jj);
#pragma unroll
  for (int q = 0; q < N; ++q)
#pragma unroll
    for (int p = 0; p < N; ++p) {
      X[q][p] = at<N>(Xj.A, p, q, j); /* Aj^T */
      Y[q][p] = at<N>(Xi.A, q, p, i);
    }
  bool ok = solve_thread<N>(Zi, Jj, X);
  ok = solve_thread<N>(Jj, Zi, Y) && ok;
  /* bi + Zi ej, ej - Jj bi */
#pragma unroll
  for (int k = 0; k < N; ++k) v1[k] = at<N>(Xi.A, 3 * N, k, i), v2[k] = at<N>(Xj.A, 3 * N + 1, k, j);
#pragma unroll
  for (int k = 0; k < N; ++k) v[k] = -v1[k];
  {
    double e[N];
#pragma unroll
    for (int k = 0; k < N; ++k) e[k] = v2[k];
    matvec<N>(Zi, e, v1);
    matvec<N>(Jj, v, v2);
  }
  double bn[N], en[N];
#pragma unroll
  for (int k = 0; k < N; ++k) bn[k] = at<N>(Xj.A, 3 * N, k, j), en[k] = at<N>(Xi.A, 3 * N + 1, k, i);
  matvec<N>(X, v1, bn);
  matvec<N>(Y, v2, en);
  store_col<N>(O.A, 3 * N, o, bn);
  store_col<N>(O.A, 3 * N + 1, o, en);
  /* J = Y (Jj Ai) + Ji: Jj has been read */
#pragma unroll
  for (int q = 0; q < N; ++q) {
    double t[N], out[N];
#pragma unroll
    for (int k = 0; k < N; ++k) v[k] = at<N>(Xi.A, q, k, i), t[k] = 0.0, out[k] = at<N>(Xi.A, 2 * N + q, k, i);
    matvec<N>(Jj, v, t);
    matvec<N>(Y, t, out);
    store_col<N>(O.A, 2 * N + q, o, out);
  }
  /* Z = (X Zi) Aj^T + Zj, then A = X Ai */
#pragma unroll
  for (int q = 0; q < N; ++q) {
#pragma unroll
    for (int k = 0; k < N; ++k) T[q][k] = 0.0;
    matvec<N>(X, Zi[q], T[q]);
  }
#pragma unroll
  for (int q = 0; q < N; ++q) {
    double out[N];
#pragma unroll
    for (int k = 0; k < N; ++k) v[k] = at<N>(Xj.A, k, q, j), out[k] = at<N>(Xj.A, N + q, k, j);
    matvec<N>(T, v, out);
    store_col<N>(O.A, N + q, o, out);
  }
#pragma unroll
  for (int q = 0; q < N; ++q) {
    double out[N];
#pragma unroll
    for (int k = 0; k < N; ++k) v[k] = at<N>(Xi.A, q, k, i), out[k] = 0.0;
    matvec<N>(X, v, out);
    store_col<N>(O.A, q, o, out);
  }
  return ok;
}

template <int N>
__device__ __forceinline__ void combine_smooth_thread(const SElems& Xi, int64_t i, const SElems& Xj, int64_t j,
                                                      const SElems& O, int64_t o)
{
  double E[N][N], T[N][N], v[N], out[N];
  load_mat<N>(Xj.E, 0, j, E);
#pragma unroll
  for (int q = 0; q < N; ++q) { /* Ej Li, Ej Ei */
#pragma unroll
    for (int k = 0; k < N; ++k) v[k] = at<N>(Xi.E, N + q, k, i), T[q][k] = 0.0;
    matvec<N>(E, v, T[q]);
#pragma unroll
    for (int k = 0; k < N; ++k) v[k] = at<N>(Xi.E, q, k, i), out[k] = 0.0;
    matvec<N>(E, v, out);
    store_col<N>(O.E, q, o, out);
  }
#pragma unroll
  for (int k = 0; k < N; ++k) v[k] = at<N>(Xi.E, 2 * N, k, i), out[k] = at<N>(Xj.E, 2 * N, k, j);
  matvec<N>(E, v, out);
  store_col<N>(O.E, 2 * N, o, out);
#pragma unroll
  for (int q = 0; q < N; ++q) { /* (Ej Li) Ej^T + Lj */
#pragma unroll
    for (int k = 0; k < N; ++k) v[k] = E[k][q], out[k] = at<N>(Xj.E, N + q, k, j);
    matvec<N>(T, v, out);
    store_col<N>(O.E, N + q, o, out);
  }
}

/* columns 0 .. cols - 1 of an element */
template <int N>
__device__ __forceinline__ void copy_thread(const Soa& X, int64_t s, const Soa& O, int64_t o, int cols)
{
  for (int c = 0; c < cols; ++c) copy<N>(X, s, O, o, c, true);
}

template <int N>
__global__ void __launch_bounds__(kThreads) up_filter_thread(int T, ScanLevel lv, ScanLevel nx, FElems cur, FElems nxt,
                                                             int* flag)
{
  const int64_t item = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  if (item >= lv.nup) return;
  const int t = find_track(lv.up_items, T, item);
  const int64_t p = item - lv.up_items[t], s0 = lv.start[t] + 2 * p, o = nx.start[t] + p;
  if (2 * p + 1 >= lv.L[t]) copy_thread<N>(cur.A, s0, nxt.A, o, 3 * N + 2);
  else if (!combine_thread<N>(cur, s0, cur, s0 + 1, nxt, o)) atomicOr(flag, 2);
}
template <int N>
__global__ void __launch_bounds__(kThreads) down_filter_thread(int T, ScanLevel lv, ScanLevel nx, FElems cur, FElems nxt,
                                                               int* flag)
{
  const int64_t item = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  if (item >= lv.ndown) return;
  const int t = find_track(lv.down_items, T, item);
  const int64_t p = item - lv.down_items[t], L = lv.L[t];
  if (L < 2) return;
  const int64_t s0 = lv.start[t] + 2 * p, b0 = nx.start[t] + p;
  if (2 * p + 1 < L) copy_thread<N>(nxt.A, b0, cur.A, s0 + 1, 3 * N + 2);
  if (p > 0 && !combine_thread<N>(nxt, b0 - 1, cur, s0, cur, s0)) atomicOr(flag, 2);
}
template <int N>
__global__ void __launch_bounds__(kThreads) up_smooth_thread(int T, ScanLevel lv, ScanLevel nx, SElems cur, SElems nxt)
{
  const int64_t item = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  if (item >= lv.nup) return;
  const int t = find_track(lv.up_items, T, item);
  const int64_t p = item - lv.up_items[t], s0 = lv.start[t] + 2 * p, o = nx.start[t] + p;
  if (2 * p + 1 >= lv.L[t]) copy_thread<N>(cur.E, s0, nxt.E, o, 2 * N + 1);
  else combine_smooth_thread<N>(cur, s0, cur, s0 + 1, nxt, o);
}
template <int N>
__global__ void __launch_bounds__(kThreads) down_smooth_thread(int T, ScanLevel lv, ScanLevel nx, SElems cur, SElems nxt)
{
  const int64_t item = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  if (item >= lv.ndown) return;
  const int t = find_track(lv.down_items, T, item);
  const int64_t p = item - lv.down_items[t], L = lv.L[t];
  if (L < 2) return;
  const int64_t s0 = lv.start[t] + 2 * p, b0 = nx.start[t] + p;
  if (2 * p + 1 < L) copy_thread<N>(nxt.E, b0, cur.E, s0 + 1, 2 * N + 1);
  if (p > 0) combine_smooth_thread<N>(nxt, b0 - 1, cur, s0, cur, s0);
}

/* the scan kernels of a state dimension; a level's launches by its items */
struct Scans {
  void (*up_f)(int, ScanLevel, ScanLevel, FElems, FElems, int*) = nullptr;
  void (*down_f)(int, ScanLevel, ScanLevel, FElems, FElems, int*) = nullptr;
  void (*up_s)(int, ScanLevel, ScanLevel, SElems, SElems) = nullptr;
  void (*down_s)(int, ScanLevel, ScanLevel, SElems, SElems) = nullptr;
  int smooth_per_block = 0, filter_per_block = kWarps, block = 32 * kWarps;
};
template <int N>
Scans scans_n(bool threads)
{
  Scans s;
  if constexpr (N <= 5)
    if (threads) {
      s.up_f = up_filter_thread<N>;
      s.down_f = down_filter_thread<N>;
      s.up_s = up_smooth_thread<N>;
      s.down_s = down_smooth_thread<N>;
      s.smooth_per_block = s.filter_per_block = s.block = kThreads;
      return s;
    }
  s.up_f = up_filter<N>;
  s.down_f = down_filter<N>;
  s.up_s = up_smooth<N>;
  s.down_s = down_smooth<N>;
  s.smooth_per_block = SmoothGroup<N>::per_block;
  return s;
}
/* Lanes up to eight rounds of a warp a scheduler: there a thread's chain takes as
 * long (10,000 steps, n = 1 to 5: by lanes alone 0.34, 0.48, 0.66, 0.89 and 1.20
 * ms, with threads for the 5,000 combines of the first level 0.33, 0.47, 0.65,
 * 0.88 and 1.21)                                                             */
constexpr int64_t kLaneItems = 4864;
inline Scans scans(int n, int64_t items)
{
  const bool threads = items > kLaneItems;
  switch (n) {
    case 1: return scans_n<1>(threads);
    case 2: return scans_n<2>(threads);
    case 3: return scans_n<3>(threads);
    case 4: return scans_n<4>(threads);
    case 5: return scans_n<5>(threads);
    case 6: return scans_n<6>(threads);
    case 7: return scans_n<7>(threads);
    case 8: return scans_n<8>(threads);
    default: return Scans();
  }
}

}  // namespace asmall
