/*
 * lanes.cuh -- Householder QR of a small panel whose columns lie on the lanes
 * of a warp (or of a quarter of one), in registers, for FP64, double-float and
 * FP32: shared by the odd-even smoother, the associative smoother and the filter
 * for up to 8 states.
 *
 * On GB300 an FP64 instruction of a warp occupies its scheduler's quarter of
 * the SM for 64 cycles, whether 1 or 32 lanes take part (measured), so what
 * counts is the number of instructions on the longest chain: a column per
 * lane makes that 2 n + 15 per reflector of a triangle on top of a square.
 */
#pragma once
#include <cstdint>

#include "df64.cuh"

namespace lanes {

/* 1/sqrt(s) and 1/d for s, d in FP32's range: one third-order step of the
 * series of (1 - e)^(-1/2) and (1 - e)^(-1) from an FP32 seed (e of about
 * 2^-21, the neglected term 2^-64): 5 and 3 FP64 instructions, where sqrt and
 * a division cost about 10 and 6 (610 and 370 cycles, measured).            */
__device__ __forceinline__ double rsqrt_series(double s)
{
  const double y = (double)rsqrtf((float)s);
  const double e = fma(-(s * y), y, 1.0);
  return fma(y, e * fma(e, 0.375, 0.5), y);
}
__device__ __forceinline__ double rcp_series(double d)
{
  const double y = (double)__fdividef(1.0f, (float)d);
  const double e = fma(-d, y, 1.0);
  return fma(y, fma(e, e, e), y);
}
/* 2^-100 <= |x| < 2^100: both series apply */
__device__ __forceinline__ bool series_range(double x)
{
  return ((((uint32_t)__double2hiint(x) >> 20) & 0x7ffu) - 923u) < 200u;
}

__device__ __forceinline__ double recip(double d) { return series_range(d) ? rcp_series(d) : 1.0 / d; }
__device__ __forceinline__ ukg_df::dd recip(ukg_df::dd d) { return ukg_df::dd(1) / d; }

__device__ __forceinline__ float recip(float d) { return 1.0f / d; }

/* 1 / sqrt(s), s > 0 */
template <typename T>
__device__ __forceinline__ T inv_root(T s) { return T(1) / sqrt(s); }
template <>
__device__ __forceinline__ double inv_root<double>(double s)
{
  return series_range(s) ? rsqrt_series(s) : rsqrt(s); /* either within one unit in the last place */
}

/* The reflector that maps (alpha, x) to (beta, 0), tail = x^T x != 0, as
 * H = I - inv u u^T with u = (amb, x): a column (a_k, a) takes
 * d = inv (x^T a + amb a_k), a_k -= d amb, a -= d x.  x stays unscaled.      */
template <typename T>
struct Refl {
  T beta, amb, inv;
};
__device__ __forceinline__ Refl<double> reflector(double alpha, double tail)
{
  Refl<double> r;
  const double s = fma(alpha, alpha, tail);
  if (series_range(s)) {
    const double nb = s * rsqrt_series(s);
    r.beta = -copysign(nb, alpha);
    r.amb = alpha - r.beta;
    r.inv = rcp_series(nb * fabs(r.amb));
  } else {
    const double nb = sqrt(s);
    r.beta = -copysign(nb, alpha);
    r.amb = alpha - r.beta;
    r.inv = 1.0 / (nb * fabs(r.amb));
  }
  return r;
}
__device__ __forceinline__ Refl<ukg_df::dd> reflector(ukg_df::dd alpha, ukg_df::dd tail)
{
  using ukg_df::dd;
  Refl<dd> r;
  const dd nb = sqrt(fma(alpha, alpha, tail));
  r.beta = -copysign(nb, alpha);
  r.amb = alpha - r.beta;
  r.inv = dd(1) / (nb * fabs(r.amb));
  return r;
}

__device__ __forceinline__ Refl<float> reflector(float alpha, float tail)
{
  Refl<float> r;
  const float nb = sqrtf(fmaf(alpha, alpha, tail));
  r.beta = -copysignf(nb, alpha);
  r.amb = alpha - r.beta;
  r.inv = 1.0f / (nb * fabsf(r.amb));
  return r;
}

/* a sum of products: FP64 adds them one by one; double-float keeps the sum
 * unnormalized until it is done (df64.cuh's acc, 12 instead of 15
 * instructions a term)                                                      */
template <typename T>
struct Dot {
  T s = T(0);
  __device__ __forceinline__ void add(T a, T b) { s = fma(a, b, s); }
  __device__ __forceinline__ T value() const { return s; }
};
template <>
struct Dot<ukg_df::dd> {
  ukg_df::acc s{0.0f, 0.0f};
  __device__ __forceinline__ void add(ukg_df::dd a, ukg_df::dd b) { ukg_df::add_prod(s, a, b); }
  __device__ __forceinline__ ukg_df::dd value() const { return ukg_df::finish(s); }
};

__device__ __forceinline__ float shfl(unsigned m, float v, int src, int w) { return __shfl_sync(m, v, src, w); }
__device__ __forceinline__ double shfl(unsigned m, double v, int src, int w) { return __shfl_sync(m, v, src, w); }
__device__ __forceinline__ ukg_df::dd shfl(unsigned m, ukg_df::dd v, int src, int w)
{
  return ukg_df::dd(__shfl_sync(m, v.hi, src, w), __shfl_sync(m, v.lo, src, w));
}

/* ---------------------------------------------------------------------------
 * QR of a panel held as columns over the LPI lanes of a group: lane `lane`
 * of the group holds in slot s the column s * LPI + lane, its rows 0..N-1 in
 * t[s] and N..2N-1 in b[s].  The pivots are the columns base .. base + N - 1,
 * all in slot 0 (base is 0 but for lanes that carry a second panel beside the
 * first).  Reflectors nref and up are left out (lanes of one panel agree).
 * Lanes of a finished pivot column go on with the others: reflector k leaves
 * the rows above k alone, so t keeps R, but their b means nothing afterwards.
 * ------------------------------------------------------------------------ */

/* The triangle on top of the square.  The loop is kept rolled (unrolled, a
 * cold pass spent half its time fetching instructions): row k of the top is
 * always at index 0, rotated to the end when it is done, so after N rounds
 * the rows are back in order.                                               */
template <typename T, int N, int LPI, int S>
__device__ __forceinline__ void lanes_qr_tri(T (&t)[S][N], T (&b)[S][N], unsigned gm, int lane, int base, int nref)
{
#pragma unroll 1
  for (int k = 0; k < N; ++k) {
    const int src = base + k;
    T x[N], dot[S], tk[S];
    const T alpha = shfl(gm, t[0][0], src, LPI);
#pragma unroll
    for (int i = 0; i < N; ++i) x[i] = shfl(gm, b[0][i], src, LPI);
#pragma unroll
    for (int s = 0; s < S; ++s) {
      Dot<T> d;
#pragma unroll
      for (int i = 0; i < N; ++i) d.add(x[i], b[s][i]);
      dot[s] = d.value();
      tk[s] = t[s][0];
    }
    const T tail = shfl(gm, dot[0], src, LPI);
    if (tail != T(0) && k < nref) {
      const Refl<T> r = reflector(alpha, tail);
#pragma unroll
      for (int s = 0; s < S; ++s) {
        const T d = fma(r.amb, tk[s], dot[s]) * r.inv;
        tk[s] = fma(-d, r.amb, tk[s]);
        if (s == 0 && lane == src) tk[s] = r.beta;
#pragma unroll
        for (int i = 0; i < N; ++i) b[s][i] = fma(-d, x[i], b[s][i]);
      }
    }
#pragma unroll
    for (int s = 0; s < S; ++s) {
#pragma unroll
      for (int i = 0; i + 1 < N; ++i) t[s][i] = t[s][i + 1];
      t[s][N - 1] = tk[s];
    }
  }
}

/* no structure: reflector k is rows k..N-1 of the top and the MB rows below */
template <typename T, int N, int LPI, int S, int MB>
__device__ __forceinline__ void lanes_qr_full(T (&t)[S][N], T (&b)[S][MB], unsigned gm, int lane, int base, int nref)
{
#pragma unroll
  for (int k = 0; k < N; ++k) {
    const int src = base + k;
    T x[N + MB], dot[S];
    const T alpha = shfl(gm, t[0][k], src, LPI);
#pragma unroll
    for (int i = k + 1; i < N; ++i) x[i] = shfl(gm, t[0][i], src, LPI);
#pragma unroll
    for (int i = 0; i < MB; ++i) x[N + i] = shfl(gm, b[0][i], src, LPI);
#pragma unroll
    for (int s = 0; s < S; ++s) {
      Dot<T> d;
#pragma unroll
      for (int i = k + 1; i < N; ++i) d.add(x[i], t[s][i]);
#pragma unroll
      for (int i = 0; i < MB; ++i) d.add(x[N + i], b[s][i]);
      dot[s] = d.value();
    }
    const T tail = shfl(gm, dot[0], src, LPI);
    if (tail != T(0) && k < nref) {
      const Refl<T> r = reflector(alpha, tail);
#pragma unroll
      for (int s = 0; s < S; ++s) {
        const T d = fma(r.amb, t[s][k], dot[s]) * r.inv;
        t[s][k] = fma(-d, r.amb, t[s][k]);
        if (s == 0 && lane == src) t[s][k] = r.beta;
#pragma unroll
        for (int i = k + 1; i < N; ++i) t[s][i] = fma(-d, x[i], t[s][i]);
#pragma unroll
        for (int i = 0; i < MB; ++i) b[s][i] = fma(-d, x[N + i], b[s][i]);
      }
    }
  }
}

}  // namespace lanes
