/*
 * associative_cols.cuh -- the associative smoother's scans and smoothing
 * elements for 9 to 64 states: one thread block per item, one thread per
 * matrix column (columns.cuh).  Included by associative.cu.
 *
 * The block-per-item kernels of associative_cta.cuh solve one system after the
 * other with their panels in global scratch.  Here the two systems of a
 * filtering combine are two blocks' work, columns in registers, and every
 * n x n product is columns times a matrix that all threads read at the same
 * place, half of the inner index per thread.  A combine is about 49,000 FP64
 * warp instructions at n = 48 (a third of them the reductions); at 19 cycles an
 * SM each that bounds the large levels, and the chain of n reflectors and four
 * half products the small ones.  5,000 steps, n = 48, m = 24: scans 74.5 ms
 * before, 51.5 now, smoothing elements 9.9 and 8.2.
 */
#pragma once
#include "columns.cuh"

namespace acols {

using acta::AArgs;
using acta::FEl;
using acta::RawS;
using acta::SEl;
using columns::back_subst;
using columns::load_rows;
using columns::matvec;
using columns::qr_square;
using columns::SquareShared;

/* threads: two per column of n (twice n columns, or n columns whose products
 * are split in two); four for the products of a filtering combine            */
template <int NP>
__host__ __device__ constexpr int threads2() { return (2 * NP + 31) / 32 * 32; }
template <int NP>
__host__ __device__ constexpr int threads4() { return (4 * NP + 31) / 32 * 32; }
/* blocks per SM that the registers are budgeted for */
template <int NP>
__host__ __device__ constexpr int blocks2() { return NP <= 16 ? 12 : NP <= 24 ? 8 : NP <= 32 ? 6 : NP <= 48 ? 4 : 2; }
template <int NP>
__host__ __device__ constexpr int blocks4() { return NP <= 16 ? 8 : NP <= 24 ? 5 : NP <= 32 ? 3 : NP <= 48 ? 2 : 1; }

/* rows of b, aligned to the end, to p */
template <int NP>
__device__ __forceinline__ void put_end(double* p, int n, const double (&b)[NP])
{
#pragma unroll
  for (int i = 0; i < NP; ++i)
    if (i - NP + n >= 0) p[i - NP + n] = b[i];
}
template <int NP>
__device__ __forceinline__ void put_rows(double* p, int n, const double (&b)[NP])
{
#pragma unroll
  for (int i = 0; i < NP; ++i)
    if (i < n) p[i] = b[i];
}

/* b += M s over half of the columns of M: the two threads of a column take one
 * each and add up through shared memory (join).                              */
template <int NP, class AT>
__device__ __forceinline__ void matvec_half(const double* M, int n, int half, double (&b)[NP], AT at)
{
  const int k0 = half ? (n + 1) / 2 : 0, k1 = half ? n : (n + 1) / 2;
  double s = at(k0 < n ? k0 : 0);
#pragma unroll 1
  for (int k = k0; k < k1; ++k) {
    const double next = k + 1 < k1 ? at(k + 1) : 0.0;
    const double* p = M + (int64_t)k * n;
#pragma unroll
    for (int i = 0; i < NP; i += 4)
      if (i < n) /* the same in every thread */
#pragma unroll
        for (int v = 0; v < 4; ++v)
          if (i + v < n) b[i + v] = fma(p[i + v], s, b[i + v]);
    s = next;
  }
}
/* the second thread's half to w (n entries), read by the first; a barrier on
 * each side for the whole block                                              */
template <int NP>
__device__ __forceinline__ void join(double* w, int n, bool on, int half, double (&b)[NP])
{
  if (on && half) put_rows<NP>(w, n, b);
  __syncthreads();
  if (on && !half)
#pragma unroll
    for (int i = 0; i < NP; ++i)
      if (i < n) b[i] += w[i];
}

/* filteringAssociativeOperation O = Xi (x) Xj (see acta::combine_filter), in two
 * kernels.  solve: X = Aj (I + Zi Jj)^{-1} (block 2 item) and Y = Ai^T (I + Jj
 * Zi)^{-1} (block 2 item + 1) into XY.  products: with X and Y every column of
 * the result is by itself -- Z = X (Zi Aj^T) + Zj and A = X Ai in block 2 item,
 * J = Y (Jj Ai) + Ji and the vectors in 2 item + 1, neither writing what the
 * other reads of Xj -- so a combine is spread over two SMs twice: 1.0 ms as one block, 0.3 ms this way at n = 48, which is what
 * the levels of few items take.                                              */
template <int NP>
__device__ bool solve_half(double* dyn, SquareShared<NP>& sm, int n, int which, const FEl& Xi, int64_t i, const FEl& Xj,
                           int64_t j, double* out)
{
  constexpr int NT = threads2<NP>();
  const int tid = threadIdx.x, nn = n * n;
  double* Zt = dyn; /* Zi^T, Jj^T */
  double* Jt = Zt + nn;
  double* R = Jt + nn;
  double* dv = R + nn;
  const double *Ai = &Xi.A.at(0, i), *Zi = &Xi.Z.at(0, i), *Aj = &Xj.A.at(0, j), *Jj = &Xj.J.at(0, j);
  for (int e = tid; e < nn; e += NT) {
    const int c = e / n, r = e - c * n;
    Zt[r * n + c] = Zi[e];
    Jt[r * n + c] = Jj[e];
  }
  __syncthreads();
  const int g = tid / n, q = tid - g * n; /* g: 0 pivots, 1 right-hand sides, 2 idle */
  const bool act = g < 2;
  double b[NP];
  /* column q of I + Jj^T Zi^T, or of I + Zi^T Jj^T, by both threads */
#pragma unroll
  for (int r = 0; r < NP; ++r) b[r] = g == 0 && r == q ? 1.0 : 0.0;
  if (act) {
    const double* s = (which ? Jt : Zt) + q * n;
    matvec_half<NP>(which ? Zt : Jt, n, g, b, [&](int k) { return s[k]; });
  }
  join<NP>(R + (act ? q : 0) * n, n, act, g, b);
  if (g == 1) { /* column q of Aj^T, or of Ai */
    const double* p = which ? Ai + (int64_t)q * n : Aj + q;
    const int st = which ? 1 : n;
#pragma unroll
    for (int r = 0; r < NP; ++r) b[r] = r < n ? p[r * st] : 0.0;
  }
  qr_square<NP>(sm, act, g ? n + q : q, n, b);
  bool bad = false;
  if (g == 0) {
    put_end<NP>(R + q * n, n, b);
    const double d = R[q * n + q]; /* this thread's own column */
    bad = d == 0.0;
    dv[q] = lanes::recip(d);
  }
  __syncthreads();
  if (g == 1) /* column q of X^T (Y^T) is row q of X (Y) */
    back_subst<double, NP>(R, dv, n, b, [&](int r, double v) { out[r * n + q] = v; });
  return bad;
}
inline size_t solve_smem(int n) { return (size_t)(3 * n * n + n) * sizeof(double); }

template <int NP>
__device__ void products(double* dyn, int n, int which, const FEl& Xi, int64_t i, const FEl& Xj, int64_t j,
                         const double* X, const FEl& O, int64_t o)
{
  const int tid = threadIdx.x, nn = n * n;
  const double* Y = X + nn;
  const double *Ai = &Xi.A.at(0, i), *Zi = &Xi.Z.at(0, i), *Ji = &Xi.J.at(0, i), *bi = &Xi.b.at(0, i);
  const double *Aj = &Xj.A.at(0, j), *Zj = &Xj.Z.at(0, j), *Jj = &Xj.J.at(0, j), *ej = &Xj.e.at(0, j);
  const int g = tid / n, q = tid - g * n, half = g & 1;
  const bool one = g < 2, two = !one && g < 4; /* threads 0..2n-1: Z or J, 2n..4n-1: A or the vectors */
  double* w = dyn + (one ? 0 : nn) + (one || two ? q : 0) * n;
  double b[NP];
#pragma unroll
  for (int r = 0; r < NP; ++r) b[r] = 0.0;
  /* Zi Aj^T, or Jj Ai; X Ai beside the first */
  if (one || (two && which == 0)) {
    const double* s = one && which == 0 ? Aj + q : Ai + (int64_t)q * n;
    const int st = one && which == 0 ? n : 1;
    matvec_half<NP>(two ? X : which ? Jj : Zi, n, half, b, [&](int k) { return s[(int64_t)k * st]; });
  }
  double* vv = dyn + nn; /* bi + Zi ej, ej - Jj bi */
  if (which && g == 2) {
    double s1 = bi[q], s2 = ej[q];
    for (int k = 0; k < n; ++k) {
      s1 = fma(Zi[(int64_t)k * n + q], ej[k], s1);
      s2 = fma(-Jj[(int64_t)k * n + q], bi[k], s2);
    }
    vv[q] = s1;
    vv[n + q] = s2;
  }
  join<NP>(w, n, one || (two && which == 0), half, b);
  double s1 = 0.0, s2 = 0.0;
  if (one && !half) put_rows<NP>(w, n, b);
  if (which && g == 2) {
    s1 = Xj.b.at(q, j), s2 = Xi.e.at(q, i);
    for (int k = 0; k < n; ++k) {
      s1 = fma(X[(int64_t)k * n + q], vv[k], s1);
      s2 = fma(Y[(int64_t)k * n + q], vv[n + k], s2);
    }
  }
  __syncthreads(); /* this block's entries of Xj but Zj have been read; the other block writes none of what it reads */
  if (two && !half && which == 0) put_rows<NP>(&O.A.at((int64_t)q * n, o), n, b);
  if (which && g == 2) {
    O.b.at(q, o) = s1;
    O.e.at(q, o) = s2;
  }
  if (one) {
    load_rows<double, NP>((which ? Ji : Zj) + (int64_t)q * n, n, !half, b);
    matvec_half<NP>(which ? Y : X, n, half, b, [&](int k) { return w[k]; });
  }
  __syncthreads(); /* w has been read */
  join<NP>(w, n, one, half, b);
  if (one && !half) put_rows<NP>(&(which ? O.J : O.Z).at((int64_t)q * n, o), n, b);
}
inline size_t products_smem(int n) { return (size_t)(2 * n * n + 2 * n) * sizeof(double); }

/* smoothingAssociativeOperation, a column by itself: L = Ej (Li Ej^T) + Lj on
 * the threads 0..n-1 and (second halves) 2n..3n-1, E = Ej Ei on the others,
 * g = Ej gi + gj a row per thread                                            */
template <int NP>
__device__ void combine_smooth(double* dyn, int n, const SEl& Xi, int64_t i, const SEl& Xj, int64_t j, const SEl& O,
                               int64_t o)
{
  constexpr int NT = threads4<NP>();
  const int tid = threadIdx.x, nn = n * n;
  double* E = dyn;
  double* W = E + nn; /* a column for each of the 2n results */
  const double* Ej = &Xj.E.at(0, j);
  for (int e = tid; e < nn; e += NT) E[e] = Ej[e];
  __syncthreads();
  const int g = tid / n, q = tid - g * n, half = g >> 1;
  const bool act = g < 4, isE = g & 1;
  double* w = W + (isE ? nn : 0) + (act ? q : 0) * n;
  double b[NP];
#pragma unroll
  for (int r = 0; r < NP; ++r) b[r] = 0.0;
  if (act && !isE) matvec_half<NP>(&Xi.L.at(0, i), n, half, b, [&](int k) { return E[k * n + q]; });
  join<NP>(w, n, act && !isE, half, b);
  if (act && !isE && !half) put_rows<NP>(w, n, b);
  __syncthreads();
  if (act && !isE && !half) load_rows<double, NP>(&Xj.L.at((int64_t)q * n, j), n, true, b);
  else
#pragma unroll
    for (int r = 0; r < NP; ++r) b[r] = 0.0;
  if (act) {
    const double* s = isE ? &Xi.E.at((int64_t)q * n, i) : w;
    matvec_half<NP>(E, n, half, b, [&](int k) { return s[k]; });
  }
  double gv = 0.0;
  if (g == 3) {
    gv = Xj.g.at(q, j);
    for (int k = 0; k < n; ++k) gv = fma(E[k * n + q], Xi.g.at(k, i), gv);
  }
  __syncthreads(); /* Xj and the columns in W have been read */
  join<NP>(w, n, act, half, b);
  if (act && !half) put_rows<NP>(&(isE ? O.E : O.L).at((int64_t)q * n, o), n, b);
  if (g == 3) O.g.at(q, o) = gv;
}
inline size_t smooth_smem(int n) { return (size_t)(3 * n * n) * sizeof(double); }

template <int NT>
__device__ __forceinline__ void copy(const cta::Aos<double>& X, int64_t s, const cta::Aos<double>& O, int64_t o)
{
  for (int e = threadIdx.x; e < (int)X.w; e += NT) O.at(e, o) = X.at(e, s);
}
template <int NT>
__device__ __forceinline__ void copy(const FEl& X, int64_t s, const FEl& O, int64_t o)
{
  copy<NT>(X.A, s, O.A, o), copy<NT>(X.Z, s, O.Z, o), copy<NT>(X.J, s, O.J, o);
  copy<NT>(X.b, s, O.b, o), copy<NT>(X.e, s, O.e, o);
}
template <int NT>
__device__ __forceinline__ void copy(const SEl& X, int64_t s, const SEl& O, int64_t o)
{
  copy<NT>(X.E, s, O.E, o), copy<NT>(X.L, s, O.L, o), copy<NT>(X.g, s, O.g, o);
}

/* an item of a sweep: what it combines (i and j; i < 0: nothing) and where the
 * result goes, and what it copies (up: an odd element; down: the prefix)     */
struct Item {
  int64_t i, j, o;
};
__device__ __forceinline__ Item up_item(int T, const ScanLevel& lv, const ScanLevel& nx, int64_t item)
{
  const int t = find_track(lv.up_items, T, item);
  const int64_t p = item - lv.up_items[t], s0 = lv.start[t] + 2 * p;
  return Item{2 * p + 1 < lv.L[t] ? s0 : -1, s0 + 1, nx.start[t] + p};
}
__device__ __forceinline__ Item down_item(int T, const ScanLevel& lv, const ScanLevel& nx, int64_t item, int64_t* copy_to)
{
  const int t = find_track(lv.down_items, T, item);
  const int64_t p = item - lv.down_items[t], L = lv.L[t];
  const int64_t s0 = lv.start[t] + 2 * p, b0 = nx.start[t] + p;
  *copy_to = L >= 2 && 2 * p + 1 < L ? s0 + 1 : -1;
  return Item{L >= 2 && p > 0 ? b0 - 1 : -1, s0, b0};
}

/* kUp: Xi, Xj = cur and O = nxt; else Xi = nxt, Xj = O = cur.  XY: 2 n^2
 * entries per item.                                                          */
template <int NP, bool kUp>
__global__ void __launch_bounds__(threads2<NP>(), blocks2<NP>()) filter_solve(int n, int T, ScanLevel lv, ScanLevel nx,
                                                                              FEl cur, FEl nxt, double* XY, int64_t item0,
                                                                              int* flag)
{
  extern __shared__ __align__(16) double acols_dyn[];
  __shared__ SquareShared<NP> sm;
  const int64_t rel = blockIdx.x >> 1, item = item0 + rel;
  const int which = blockIdx.x & 1;
  int64_t cp = -1;
  const Item I = kUp ? up_item(T, lv, nx, item) : down_item(T, lv, nx, item, &cp);
  if (I.i < 0) return;
  if (solve_half<NP>(acols_dyn, sm, n, which, kUp ? cur : nxt, I.i, cur, I.j, XY + (2 * rel + which) * n * n))
    atomicOr(flag, 2);
}
template <int NP, bool kUp>
__global__ void __launch_bounds__(threads4<NP>(), blocks4<NP>()) filter_products(int n, int T, ScanLevel lv, ScanLevel nx,
                                                                                 FEl cur, FEl nxt, const double* XY,
                                                                                 int64_t item0)
{
  extern __shared__ __align__(16) double acols_dyn[];
  const int64_t rel = blockIdx.x >> 1, item = item0 + rel;
  const int which = blockIdx.x & 1;
  int64_t cp = -1;
  const Item I = kUp ? up_item(T, lv, nx, item) : down_item(T, lv, nx, item, &cp);
  if (which && kUp && I.i < 0) copy<threads4<NP>()>(cur, I.j - 1, nxt, I.o);
  if (which && !kUp && cp >= 0) copy<threads4<NP>()>(nxt, I.o, cur, cp);
  if (I.i < 0) return;
  products<NP>(acols_dyn, n, which, kUp ? cur : nxt, I.i, cur, I.j, XY + 2 * rel * n * n, kUp ? nxt : cur, kUp ? I.o : I.j);
}
template <int NP, bool kUp>
__global__ void __launch_bounds__(threads4<NP>(), blocks4<NP>()) smooth_combine(int n, int T, ScanLevel lv, ScanLevel nx,
                                                                                SEl cur, SEl nxt)
{
  extern __shared__ __align__(16) double acols_dyn[];
  int64_t cp = -1;
  const Item I = kUp ? up_item(T, lv, nx, blockIdx.x) : down_item(T, lv, nx, blockIdx.x, &cp);
  if (kUp && I.i < 0) copy<threads4<NP>()>(cur, I.j - 1, nxt, I.o);
  if (cp >= 0) copy<threads4<NP>()>(nxt, I.o, cur, cp);
  if (I.i < 0) return;
  combine_smooth<NP>(acols_dyn, n, kUp ? cur : nxt, I.i, cur, I.j, kUp ? nxt : cur, kUp ? I.o : I.j);
}

/* the covariance of a factor (kalman_covariance_matrix_explicit,
 * c/kalman_base.c:178-214) for smooth_element, to R by rows: column q on thread
 * q < n.  Apart, so that its registers are not the caller's.                 */
template <int NP>
__device__ __noinline__ bool explicit_rows(char kt, const double* K, int n, double* S, double* R, double* dv,
                                           SquareShared<NP>& sm)
{
  constexpr int NT = threads2<NP>();
  const int tid = threadIdx.x, nn = n * n, g = tid / n, q = tid - g * n;
  double b[NP];
  bool bad = false;
  if (kt == 'W') { /* K = (W^T W)^{-1} = U U^T, U = (W's R factor)^{-1} */
    load_rows<double, NP>(K + (int64_t)q * n, n, g == 0, b);
    qr_square<NP>(sm, g == 0, q, n, b);
    if (g == 0) put_end<NP>(S + q * n, n, b);
    if (g == 0) {
      const double d = S[q * n + q];
      bad |= d == 0.0;
      dv[q] = lanes::recip(d);
    }
    __syncthreads();
#pragma unroll
    for (int p = 0; p < NP; ++p) b[p] = g == 0 && p - NP + n == q ? 1.0 : 0.0;
    if (g == 0) back_subst<double, NP>(S, dv, n, b, [&](int p, double u) { R[q * n + p] = u; });
    __syncthreads(); /* R: U, column-major */
#pragma unroll
    for (int p = 0; p < NP; ++p) b[p] = 0.0;
    if (g == 0) matvec<NP>(R, n, b, [&](int l) { return R[l * n + q]; });
    __syncthreads();
  } else {
    if (kt == 'U' || kt == 'F') {
      for (int e = tid; e < nn; e += NT) S[e] = e % n >= e / n ? K[e] : 0.0;
      __syncthreads();
    }
#pragma unroll
    for (int p = 0; p < NP; ++p) b[p] = 0.0;
    if (g == 0) {
      if (kt == 'w') {
        const double w = K[q];
#pragma unroll
        for (int p = 0; p < NP; ++p)
          if (p == q) b[p] = 1.0 / (w * w);
      } else if (kt == 'U' || kt == 'F') { /* L L^T, L in S */
        matvec<NP>(S, n, b, [&](int l) { return S[l * n + q]; });
      } else if (kt == 'C') {
        load_rows<double, NP>(K + (int64_t)q * n, n, true, b);
      } else {
        bad = true;
      }
    }
  }
  if (g == 0) { /* Q transposed: row q of Q is what column q of the system takes */
#pragma unroll
    for (int p = 0; p < NP; ++p)
      if (p < n) R[p * n + q] = b[p];
  }
  __syncthreads();
  return bad;
}

/* ---------------------------------------------------------------------------
 * smoothing elements (see acta::smooth_element_cta): E = P F^T (F P F^T + Q)^{-1},
 * g = x - E (F x + c), L = P - E F P, Q from the next step's K
 * ------------------------------------------------------------------------ */
template <int NP>
__global__ void __launch_bounds__(threads2<NP>(), NP <= 32 ? blocks2<NP>() : NP <= 48 ? 3 : 1) smooth_element(AArgs a, RawS raw, SEl out,
                                                                                const int64_t* seq_start)
{
  extern __shared__ __align__(16) double acols_dyn[];
  __shared__ SquareShared<NP> sm;
  constexpr int NT = threads2<NP>();
  const int n = a.n, tid = threadIdx.x, nn = n * n;
  const int64_t gs = blockIdx.x;
  const int t = find_track(a.track_start, a.ntracks, gs);
  const int64_t g0 = a.track_start[t], k = a.track_start[t + 1] - g0, i = gs - g0;
  const int64_t r = seq_start[t] + (k - 1 - i);
  const double* x = a.state + gs * n;
  const double* P = a.cov + gs * nn;
  if (i == k - 1) {
    for (int e = tid; e < nn; e += NT) {
      out.E.at(e, r) = 0.0;
      out.L.at(e, r) = P[e];
    }
    for (int p = tid; p < n; p += NT) out.g.at(p, r) = x[p];
    return;
  }
  double* S = acols_dyn; /* (P F^T)^T; at first W's factor */
  double* R = S + nn;    /* Q; then the factor */
  double* E = R + nn;    /* halves of products; then E */
  double* dv = E + nn;
  double* v = dv + n;
  const int64_t g1 = gs + 1;
  const double* F = raw.F + g1 * nn;
  const double* K = raw.K + g1 * nn;
  const double* c = raw.c + g1 * n;
  const char kt = raw.K_type[g1];
  const int g = tid / n, q = tid - g * n; /* g: 0 pivots, 1 right-hand sides */
  double b[NP];
  bool bad = explicit_rows<NP>(kt, K, n, S, R, dv, sm);
  for (int e = tid; e < nn; e += NT) S[e] = P[e];
  __syncthreads();
  /* P F^T, column q by two threads, stored by rows */
  const bool act = g < 2;
  double* w = E + (act ? q : 0) * n;
#pragma unroll
  for (int p = 0; p < NP; ++p) b[p] = 0.0;
  if (act) matvec_half<NP>(S, n, g, b, [&](int l) { return F[(int64_t)l * n + q]; });
  join<NP>(w, n, act, g, b);
  if (g == 0) {
#pragma unroll
    for (int p = 0; p < NP; ++p)
      if (p < n) S[p * n + q] = b[p];
  }
  __syncthreads();
  /* [(F P F^T + Q)^T | (P F^T)^T] */
  load_rows<double, NP>(R + (act ? q : 0) * n, n, g == 0, b);
  if (act) matvec_half<NP>(S, n, g, b, [&](int l) { return F[(int64_t)l * n + q]; });
  join<NP>(w, n, act, g, b);
  if (g == 1) load_rows<double, NP>(S + q * n, n, true, b);
  qr_square<NP>(sm, act, g == 1 ? n + q : q, n, b);
  if (g == 0) {
    put_end<NP>(R + q * n, n, b);
    const double d = R[q * n + q];
    bad |= d == 0.0;
    dv[q] = lanes::recip(d);
  }
  /* F x + c, a row per thread */
  if (g == 1) {
    double s = c[q];
    for (int l = 0; l < n; ++l) s = fma(F[(int64_t)l * n + q], x[l], s);
    v[q] = s;
  }
  __syncthreads();
  /* column q of E^T is row q of E */
  if (g == 1) back_subst<double, NP>(R, dv, n, b, [&](int p, double u) { E[p * n + q] = u; });
  __syncthreads();
  /* L = P - (E F) P.  Not P - E (P F^T)^T, a product less: P is symmetric only up
     to its rounding errors, which I - E F damps and I + E F would double (a
     covariance error of 0.8 instead of 3e-4 where the variances of 12 states
     go up and down by 16 decades)                                          */
#pragma unroll
  for (int p = 0; p < NP; ++p) b[p] = 0.0;
  if (act) matvec_half<NP>(E, n, g, b, [&](int l) { return F[(int64_t)q * n + l]; });
  join<NP>(R + (act ? q : 0) * n, n, act, g, b);
  if (g == 0) put_rows<NP>(S + q * n, n, b);
  __syncthreads();
  load_rows<double, NP>(P + (int64_t)(act ? q : 0) * n, n, g == 0, b);
  if (act) matvec_half<NP>(S, n, g, b, [&](int l) { return -P[(int64_t)q * n + l]; });
  join<NP>(R + (act ? q : 0) * n, n, act, g, b);
  if (g == 0) {
    put_rows<NP>(&out.L.at((int64_t)q * n, r), n, b);
    double s = x[q];
    for (int l = 0; l < n; ++l) s = fma(-E[l * n + q], v[l], s);
    out.g.at(q, r) = s;
  }
  for (int e = tid; e < nn; e += NT) out.E.at(e, r) = E[e];
  if (bad) atomicOr(a.flag, 2);
}
inline size_t element_smem(int n) { return (size_t)(3 * n * n + 2 * n) * sizeof(double); }

struct Kernels {
  void (*solve[2])(int, int, ScanLevel, ScanLevel, FEl, FEl, double*, int64_t, int*) = {nullptr, nullptr}; /* up, down */
  void (*products[2])(int, int, ScanLevel, ScanLevel, FEl, FEl, const double*, int64_t) = {nullptr, nullptr};
  void (*smooth[2])(int, int, ScanLevel, ScanLevel, SEl, SEl) = {nullptr, nullptr};
  void (*smooth_element)(AArgs, RawS, SEl, const int64_t*) = nullptr;
  int threads4 = 0, threads2 = 0;
};
template <int NP>
Kernels kernels_np()
{
  Kernels k;
  k.solve[0] = filter_solve<NP, true>, k.solve[1] = filter_solve<NP, false>;
  k.products[0] = filter_products<NP, true>, k.products[1] = filter_products<NP, false>;
  k.smooth[0] = smooth_combine<NP, true>, k.smooth[1] = smooth_combine<NP, false>;
  k.smooth_element = smooth_element<NP>;
  k.threads4 = threads4<NP>();
  k.threads2 = threads2<NP>();
  return k;
}
inline Kernels kernels(int n)
{
  if (n < 9) return Kernels(); /* more observation rows than 8 for fewer states */
  if (n <= 12) return kernels_np<12>();
  if (n <= 16) return kernels_np<16>();
  if (n <= 24) return kernels_np<24>();
  if (n <= 32) return kernels_np<32>();
  if (n <= 48) return kernels_np<48>();
  if (n <= 64) return kernels_np<64>();
  return Kernels();
}

}  // namespace acols
