/*
 * columns.cuh -- dense routines with one matrix column per thread, its rows in
 * registers (NP of them, n <= NP in use), shared by the odd-even and the
 * associative smoother for 9 states and more.
 */
#pragma once
#include <cstdint>

#include "lanes.cuh"

namespace columns {

/* b <- n (or `rows`) consecutive entries, zero past them */
template <typename T, int NP>
__device__ __forceinline__ void load_rows(const T* p, int rows, bool on, T (&b)[NP])
{
#pragma unroll
  for (int i = 0; i < NP; ++i) {
    b[i] = T(0);
    if (on && i < rows) b[i] = p[i];
  }
}

/* R x = b by columns: v_j = b_j / R_jj from the last row up, the rows moving
 * towards the end as they are done.  b is aligned to the end (row n - 1 at
 * NP - 1); R column-major in shared memory (ld n), dv the reciprocals of its
 * diagonal; put(j, v_j).
 * A loop for every four rows fewer, its length in the code.  One loop with a
 * test every four rows comes out with the tests as predicates, in some builds:
 * an FP64 instruction that is predicated off takes its time all the same (30 %
 * of those of a 48-state combine's solve, 3.4 ms or 5.3).                    */
template <typename T, int NP, class PUT>
__device__ __forceinline__ void back_subst(const T* R, const T* dv, int n, T (&b)[NP], PUT put)
{
  int j = n - 1;
#pragma unroll
  for (int p = NP; p > 0; p -= 4) /* rows 0 .. j, p - 4 <= j < p */
#pragma unroll 1
    for (; j >= p - 4; --j) {
      const T v = b[NP - 1] * dv[j];
      put(j, v);
      const T* Rj = R + j * n + j - NP; /* row of b[i - 1] is i - NP + j */
#pragma unroll
      for (int i = NP - 1; i > NP - p; --i) b[i] = i - NP + j >= 0 ? fma(-v, Rj[i], b[i - 1]) : b[i - 1];
    }
}
template <typename T, int NP>
__device__ __forceinline__ void load_end(const T* p, int n, bool on, T (&b)[NP])
{
#pragma unroll
  for (int i = 0; i < NP; ++i) {
    b[i] = T(0);
    if (on && i - NP + n >= 0) b[i] = p[i - NP + n];
  }
}

/* b += M s for the column-major M (n x n, ld n) and a vector s given entry by
 * entry, four at a time, the next four on their way; b from row 0 on          */
template <int NP, class AT>
__device__ __forceinline__ void matvec(const double* M, int n, double (&b)[NP], AT at)
{
  double s[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) s[u] = u < n ? at(u) : 0.0;
#pragma unroll 1
  for (int k = 0; k < n; k += 4) {
    double next[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) next[u] = k + 4 + u < n ? at(k + 4 + u) : 0.0;
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (k + u < n) {
        const double* p = M + (int64_t)(k + u) * n;
#pragma unroll
        for (int i = 0; i < NP; i += 4)
          if (i < n) /* the same in every thread */
#pragma unroll
            for (int v = 0; v < 4; ++v)
              if (i + v < n) b[i + v] = fma(p[i + v], s[u], b[i + v]);
      }
#pragma unroll
    for (int u = 0; u < 4; ++u) s[u] = next[u];
  }
}

/* Householder QR of a square panel (n x n pivots on the columns 0..n-1 and
 * further columns), FP64.  Row k is the first of b at step k; done, it goes to the
 * end, so after n steps a column's entries are in order, aligned to the end:
 * R (whose entries below the diagonal mean nothing) and Q^T of the others.   */
template <int NP>
struct SquareShared {
  double x[2][NP], amb[2], inv[2]; /* by the step's parity */
};
template <int NP>
__device__ __forceinline__ void qr_square(SquareShared<NP>& sm, bool act, int c, int n, double (&b)[NP])
{
  int k = 0;
#pragma unroll
  for (int p = NP; p >= 0; p -= 4) /* rows below row k: p - 4 < rows <= p (see back_subst) */
#pragma unroll 1
    for (; k < n && n - 1 - k > p - 4; ++k) {
      const int rows = n - 1 - k, buf = k & 1;
      double t = b[0];
#pragma unroll
      for (int i = 0; i + 1 < NP; ++i) b[i] = b[i + 1];
      double* x = sm.x[buf];
      const bool pivot = act && c == k;
      if (pivot)
#pragma unroll
        for (int i = 0; i < p; ++i) x[i] = i < rows ? b[i] : 0.0;
      __syncthreads();
      const bool on = act && c >= k; /* whole warps of finished pivots wait */
      double dot = 0.0;
      if (on) {
        double d0 = 0.0, d1 = 0.0;
#pragma unroll
        for (int i = 0; i < p; i += 4) {
          d0 = fma(x[i], b[i], d0);
          d1 = fma(x[i + 1], b[i + 1], d1);
          d0 = fma(x[i + 2], b[i + 2], d0);
          d1 = fma(x[i + 3], b[i + 3], d1);
        }
        dot = d0 + d1;
      }
      if (pivot) {
        lanes::Refl<double> r;
        r.beta = t;
        r.amb = r.inv = 0.0;
        if (dot != 0.0) r = lanes::reflector(t, dot);
        sm.amb[buf] = r.amb;
        sm.inv[buf] = r.inv;
        t = r.beta;
      }
      __syncthreads();
      const double amb = sm.amb[buf], inv = sm.inv[buf];
      if (on && !pivot && amb != 0.0) {
        const double d = fma(amb, t, dot) * inv;
        t = fma(-d, amb, t);
#pragma unroll
        for (int i = 0; i < p; ++i) b[i] = fma(-d, x[i], b[i]);
      }
      b[NP - 1] = t;
    }
}

}  // namespace columns
