/*
 * associative_small.cuh -- the scans of the associative smoother for up to 8
 * states, a warp (or half of one) per combine.  Included by associative.cu (it
 * uses that file's FElems, SElems, ScanLevel and find_track).
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

/* the scan kernels of a state dimension */
struct Scans {
  void (*up_f)(int, ScanLevel, ScanLevel, FElems, FElems, int*) = nullptr;
  void (*down_f)(int, ScanLevel, ScanLevel, FElems, FElems, int*) = nullptr;
  void (*up_s)(int, ScanLevel, ScanLevel, SElems, SElems) = nullptr;
  void (*down_s)(int, ScanLevel, ScanLevel, SElems, SElems) = nullptr;
  int smooth_per_block = 0;
};
template <int N>
Scans scans_n()
{
  Scans s;
  s.up_f = up_filter<N>;
  s.down_f = down_filter<N>;
  s.up_s = up_smooth<N>;
  s.down_s = down_smooth<N>;
  s.smooth_per_block = SmoothGroup<N>::per_block;
  return s;
}
inline Scans scans(int n)
{
  switch (n) {
    case 1: return scans_n<1>();
    case 2: return scans_n<2>();
    case 3: return scans_n<3>();
    case 4: return scans_n<4>();
    case 5: return scans_n<5>();
    case 6: return scans_n<6>();
    case 7: return scans_n<7>();
    case 8: return scans_n<8>();
    default: return Scans();
  }
}

}  // namespace asmall
