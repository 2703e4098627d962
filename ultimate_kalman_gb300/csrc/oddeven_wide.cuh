/*
 * oddeven_wide.cuh -- forward elimination of the FP32 odd-even smoother for 65
 * to 128 states (no more observation rows than states): one thread block of
 * eight warps per item, four columns by a quarter of their rows per thread.
 * Included by oddeven.cu.
 *
 * The structure is that of oddeven_cols.cuh: trapezoids of m rows on top of a
 * block of rows below, a top row read and written at its own step.  What
 * differs is where the rows below live.  A thread per column would read each
 * entry of a reflector's vector from shared memory for one multiply-add of its
 * own; a warp's read takes the cycle in which four warps could have multiplied,
 * so shared memory is what bounds such a kernel.  Here four lanes share four
 * columns, each with a quarter of the rows: an entry read serves four columns,
 * in the dot products and in the update, and the four dot products are summed
 * over the four lanes by three exchanges.
 *
 * Warps 0-3 (half 0) and 4-7 (half 1) take n columns each, warp 0 the right-hand
 * sides besides (a ninth warp would leave three on one scheduler and 168
 * registers a thread).  Three passes a pair, 256 columns being what the
 * registers hold:
 *   A    [G_j | 0; F | H]          half 0 pivots, half 1 what they leave of H
 *   B, C [R~; H_j] in half 0, [G_{j+1}; H~] in half 1, which holds H~ already
 *   B    the columns [Y~; 0] and [0; F_j], by the reflectors kept in shared memory
 * Rows used up stay where they are: the vectors of later reflectors have zeros
 * there.  The first form tried, a thread per column and two barriers a
 * reflector, took 27.9 ms where this takes 20.0: 5,000 steps of 128 states, 64
 * observations; the block-per-item kernels on panels in global scratch took 51.4
 * (tails 5.9, now 1.1; the triangularization is 1.5 ms more).  A reflector is
 * 1,100 cycles of its application, by two warps a scheduler, and 600 to 700 of
 * its forming.
 */
#pragma once

namespace wide {
using ctak::CArgs;
using lanes::Refl;
using lanes::reflector;

constexpr int NT = 256;

template <int RJ>
struct Shared {
  static constexpr int NP = 4 * RJ;
  float* V;        /* half 0's reflectors: vector k at V[k * NP] */
  float *am, *iv;  /* their entries in the top row (0 where it is used up) and inv (negative: no reflector) */
  float *X, *s1;   /* the last eight of half 1's own panel: X[(k & 7) * NP], am and iv at s1[2 * (k & 7)] */
  float *B, *Bt;   /* per half: four columns on their way to the whole warp, and their top entries */
  float* T;        /* stage A's R~ | rhs~, column c at T[c * (n | 1)] */
  __device__ explicit Shared(float* d)
      : V(d), am(V + NP * NP), iv(am + NP), X(iv + NP), s1(X + 8 * NP), B(s1 + 16), Bt(B + 8 * NP), T(Bt + 32)
  {
  }
  __device__ float* x(int panel, int k) const { return panel ? X + (k & 7) * NP : V + k * NP; }
  __device__ float* amb(int panel, int k) const { return panel ? s1 + 2 * (k & 7) : am + k; }
  __device__ float* inv(int panel, int k) const { return panel ? s1 + 2 * (k & 7) + 1 : iv + k; }
};
template <int RJ>
size_t smem(int n) { return (size_t)(16 * RJ * RJ + 72 * RJ + 48 + (n + 1) * (n | 1)) * sizeof(float); }

/* this thread's place: columns cb..cb + 3 of its half, of which it owns the top
 * entry of column c; rows 16 q + 4 l + u                                     */
struct Me {
  int half, lane, l, cb, c;
  bool rhs; /* warp 0 has the right-hand sides too */
  __device__ Me()
  {
    const int tid = threadIdx.x;
    half = tid >> 7;
    rhs = tid < 32;
    lane = tid & 31;
    l = tid & 3;
    cb = (tid & 127) & ~3;
    c = cb + l;
  }
};
__device__ __forceinline__ int row_of(const Me& me, int j) { return 16 * (j >> 2) + 4 * me.l + (j & 3); }

/* by value: a conditional of array elements is one of their addresses, and the
 * array would leave its registers                                            */
__device__ __forceinline__ float sel(bool c, float x, float y) { return c ? x : y; }

template <int RJ>
__device__ __forceinline__ void load_cols(const Me& me, const float* p, int ld, int n, int rows, float (&b)[4][RJ])
{
#pragma unroll
  for (int s = 0; s < 4; ++s)
#pragma unroll
    for (int j = 0; j < RJ; ++j) {
      b[s][j] = 0.f;
      if (me.cb + s < n && row_of(me, j) < rows) b[s][j] = p[(me.cb + s) * ld + row_of(me, j)];
    }
}
template <int RJ>
__device__ __forceinline__ void store_cols(const Me& me, float* p, int n, const float (&b)[4][RJ])
{
#pragma unroll
  for (int s = 0; s < 4; ++s)
#pragma unroll
    for (int j = 0; j < RJ; ++j)
      if (me.cb + s < n && row_of(me, j) < n) p[(me.cb + s) * n + row_of(me, j)] = b[s][j];
}
/* a right-hand side: rows 4 lane + u of warp 0 */
__device__ __forceinline__ void load_rhs(const Me& me, const float* p, int rows, float (&r)[4])
{
#pragma unroll
  for (int u = 0; u < 4; ++u) r[u] = 4 * me.lane + u < rows ? p[4 * me.lane + u] : 0.f;
}

/* x, a reflector's vector, and its products with the four columns, the product
 * with column cb + l returned in lane l.  Rows that are used up, or past n, are
 * zero in x: no test leaves them out, one for every 16 rows took three times as
 * long as the multiply-adds.                                                  */
template <int RJ>
__device__ __forceinline__ float dots(const Me& me, const float* xs, float (&x)[RJ], const float (&b)[4][RJ])
{
#pragma unroll
  for (int q = 0; q < RJ / 4; ++q) {
    const float4 v = *reinterpret_cast<const float4*>(xs + 16 * q + 4 * me.l);
    x[4 * q] = v.x, x[4 * q + 1] = v.y, x[4 * q + 2] = v.z, x[4 * q + 3] = v.w;
  }
  float d[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int j = 0; j < RJ; ++j)
#pragma unroll
    for (int s = 0; s < 4; ++s) d[s] = fmaf(x[j], b[s][j], d[s]);
  const bool hi = me.l & 2, odd = me.l & 1;
  const float e0 = sel(hi, d[2], d[0]) + __shfl_xor_sync(0xffffffffu, sel(hi, d[0], d[2]), 2);
  const float e1 = sel(hi, d[3], d[1]) + __shfl_xor_sync(0xffffffffu, sel(hi, d[1], d[3]), 2);
  return sel(odd, e1, e0) + __shfl_xor_sync(0xffffffffu, sel(odd, e0, e1), 1);
}
/* column cb + s -= d_s x, d_s from lane s */
template <int RJ>
__device__ __forceinline__ void update(const Me& me, float dc, const float (&x)[RJ], float (&b)[4][RJ])
{
  float d[4];
#pragma unroll
  for (int s = 0; s < 4; ++s) d[s] = __shfl_sync(0xffffffffu, dc, (me.lane & 28) + s);
#pragma unroll
  for (int j = 0; j < RJ; ++j)
#pragma unroll
    for (int s = 0; s < 4; ++s) b[s][j] = fmaf(-d[s], x[j], b[s][j]);
}
/* A panel's reduction: m top rows, the rows below from r0 on, `steps` reflectors */
struct Panel {
  int m, r0, steps;
};
__device__ __forceinline__ float sel4(int u, const float4& v) { return sel(u & 2, sel(u & 1, v.w, v.z), sel(u & 1, v.y, v.x)); }
__device__ __forceinline__ float dot4(const float4& x, const float4& y)
{
  return fmaf(x.x, y.x, fmaf(x.y, y.y, fmaf(x.z, y.z, x.w * y.w)));
}
__device__ __forceinline__ void sub4(float4& y, float d, const float4& x)
{
  y.x = fmaf(-d, x.x, y.x), y.y = fmaf(-d, x.y, y.y), y.z = fmaf(-d, x.z, y.z), y.w = fmaf(-d, x.w, y.w);
}
__device__ __forceinline__ float warp_sum(float d)
{
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
  return d;
}

/* Reflectors k0..k0 + 3 of a panel by the warp that holds these columns, each
 * applied to the columns after it at once: one barrier for four reflectors.
 * The columns' four lanes pass them on through shared memory, for here a lane
 * takes four rows of each (by the four lanes alone a reflector took 2,100
 * cycles, most of them fetching the long unrolled code).  The 4 x 4 block of
 * results is stored here.  t: the top entries k0..k0 + 3 of column cb + l.   */
template <int RJ, class ST>
__device__ __forceinline__ void factor4(const Shared<RJ>& sh, const Me& me, int n, int panel, int k0, const Panel P,
                                        const float (&b)[4][RJ], const float (&t)[4], ST store)
{
  constexpr int NP = 4 * RJ;
  float* B = sh.B + me.half * 4 * NP;
  float* Bt = sh.Bt + me.half * 16;
  if (me.cb == k0) {
#pragma unroll
    for (int s = 0; s < 4; ++s)
#pragma unroll
      for (int q = 0; q < RJ / 4; ++q)
        *reinterpret_cast<float4*>(B + s * NP + 16 * q + 4 * me.l) =
            make_float4(b[s][4 * q], b[s][4 * q + 1], b[s][4 * q + 2], b[s][4 * q + 3]);
    *reinterpret_cast<float4*>(Bt + 4 * me.l) = make_float4(t[0], t[1], t[2], t[3]);
  }
  __syncwarp();
  float4 y[4];
  float tt[4][4];
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    y[c] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (4 * me.lane < NP) y[c] = *reinterpret_cast<const float4*>(B + c * NP + 4 * me.lane);
    const float4 v = *reinterpret_cast<const float4*>(Bt + 4 * c);
    tt[c][0] = v.x, tt[c][1] = v.y, tt[c][2] = v.z, tt[c][3] = v.w;
  }
  float keep = 0.f;
#pragma unroll
  for (int s = 0; s < 4; ++s) {
    const int k = k0 + s;
    if (k < P.steps) { /* the same in every thread */
      const bool top = k < P.m;
      const int p = P.r0 + k - P.m, lo = top ? P.r0 : p, i = 4 * me.lane;
      float4 x = make_float4(sel(i >= lo, y[s].x, 0.f), sel(i + 1 >= lo, y[s].y, 0.f), sel(i + 2 >= lo, y[s].z, 0.f),
                             sel(i + 3 >= lo, y[s].w, 0.f));
      const int ps = top ? -1 : p; /* not part of the tail */
      const float alpha = top ? tt[s][s] : __shfl_sync(0xffffffffu, sel4(p, y[s]), (p >> 2) & 31);
      const float4 w = make_float4(sel(i == ps, 0.f, x.x), sel(i + 1 == ps, 0.f, x.y), sel(i + 2 == ps, 0.f, x.z),
                                   sel(i + 3 == ps, 0.f, x.w));
      const float tail = warp_sum(dot4(w, w));
      Refl<float> f;
      f.beta = alpha;
      f.amb = 0.f;
      f.inv = -1.f;
      if (tail != 0.f) f = reflector(alpha, tail);
      x = make_float4(sel(i == ps, f.amb, x.x), sel(i + 1 == ps, f.amb, x.y), sel(i + 2 == ps, f.amb, x.z),
                      sel(i + 3 == ps, f.amb, x.w));
      const float am = top ? f.amb : 0.f;
      if (i < NP) *reinterpret_cast<float4*>(sh.x(panel, k) + i) = x;
      if (me.lane == 0) {
        *sh.amb(panel, k) = am;
        *sh.inv(panel, k) = f.inv;
      }
      float v[4]; /* row k of the four columns */
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        if (c > s && tail != 0.f) {
          const float d = fmaf(am, tt[c][s], warp_sum(dot4(x, y[c]))) * f.inv;
          tt[c][s] = fmaf(-d, am, tt[c][s]);
          sub4(y[c], d, x);
        }
        v[c] = c < s ? 0.f : c == s ? f.beta : top ? tt[c][s] : __shfl_sync(0xffffffffu, sel4(p, y[c]), (p >> 2) & 31);
      }
      if ((me.lane >> 2) == s) keep = sel4(me.l, make_float4(v[0], v[1], v[2], v[3]));
    }
  }
  const int k = k0 + (me.lane >> 2), c = k0 + me.l;
  if (me.lane < 16 && k < P.steps && c < n) store(c, k, keep);
}

/* Up to two panels: half 0 holds P0's pivots; half 1 P1's or (steps of P1 < 0)
 * further columns of P0.  load(k): the top entries of column c; store(c, k, v)
 * takes the results; loadr(panel, k), storer(panel, k, v): those of the
 * right-hand sides r[panel].  Reflector k < m takes top row k and the rows
 * below; from k = m on its first row is row r0 + k - m of those below, where the
 * result stays until the end.  Every thread of the block calls it.           */
template <int RJ, class LD, class ST, class LDR, class STR>
__device__ __forceinline__ void reduce(const Shared<RJ>& sh, const Me& me, int n, const Panel P0, const Panel P1,
                                       float (&b)[4][RJ], float (&r)[2][4], LD load, ST store, LDR loadr, STR storer)
{
  constexpr int NP = 4 * RJ;
  const bool more = P1.steps < 0;
  const int panel = me.half == 1 && !more;
  const bool pivots = me.half == 0 || panel;
  const Panel P = panel ? P1 : P0;
  const bool own = me.c < n;
  const int wcol = me.cb & ~31; /* the warp's first column */
  const int all = P0.steps > P1.steps ? P0.steps : P1.steps;
  const int mt = P.m < P.steps ? P.m : P.steps; /* top rows in use */
  float next[4], rnext[2];
#pragma unroll
  for (int s = 0; s < 4; ++s) next[s] = own && s < mt ? load(s) : 0.f;
#pragma unroll
  for (int v = 0; v < 2; ++v) {
    const int qm = v ? P1.m : P0.m, qs = v ? P1.steps : P0.steps;
    rnext[v] = me.rhs && qm > 0 && qs > 0 ? loadr(v, 0) : 0.f;
  }
#pragma unroll 1
  for (int k0 = 0; k0 < all; k0 += 4) {
    const bool on = k0 < P.steps, mine = on && pivots && me.cb == k0; /* done by factor4 */
    float t[4];
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      t[s] = next[s];
      next[s] = own && k0 + 4 + s < mt ? load(k0 + 4 + s) : 0.f;
    }
    if (on && pivots && wcol == (k0 & ~31)) factor4<RJ>(sh, me, n, panel, k0, P, b, t, store);
    __syncthreads();
    if (on && !(pivots && wcol + 31 < k0)) /* warps of finished pivots wait */
#pragma unroll 1
      for (int s = 0; s < 4; ++s) { /* t turns with s: a short loop, and no array element by number */
        const int k = k0 + s;
        float tk = t[0];
        t[0] = t[1], t[1] = t[2], t[2] = t[3];
        const float iv = k < P.steps ? *sh.inv(panel, k) : -1.f;
        if (!(iv < 0.f)) { /* the same in every thread of a warp */
          float x[RJ];
          const float am = *sh.amb(panel, k);
          const float d = fmaf(am, tk, dots<RJ>(me, sh.x(panel, k), x, b)) * iv;
          tk = fmaf(-d, am, tk);
          update<RJ>(me, d, x, b);
        }
        t[3] = tk;
      }
    if (me.rhs) {
#pragma unroll
      for (int v = 0; v < 2; ++v) {
        const int qm = v ? P1.m : P0.m, qs = v ? P1.steps : P0.steps;
#pragma unroll 1
        for (int k = k0; k < k0 + 4 && k < qs; ++k) {
          const float iv = *sh.inv(v, k);
          float rk = rnext[v];
          rnext[v] = k + 1 < qm ? loadr(v, k + 1) : 0.f;
          if (!(iv < 0.f)) {
            float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
            if (4 * me.lane < NP) x = *reinterpret_cast<const float4*>(sh.x(v, k) + 4 * me.lane);
            float d = warp_sum(fmaf(x.x, r[v][0], fmaf(x.y, r[v][1], fmaf(x.z, r[v][2], x.w * r[v][3]))));
            const float am = *sh.amb(v, k);
            d = fmaf(am, rk, d) * iv;
            rk = fmaf(-d, am, rk);
            r[v][0] = fmaf(-d, x.x, r[v][0]);
            r[v][1] = fmaf(-d, x.y, r[v][1]);
            r[v][2] = fmaf(-d, x.z, r[v][2]);
            r[v][3] = fmaf(-d, x.w, r[v][3]);
          }
          if (me.lane == 0 && k < qm) storer(v, k, rk);
        }
      }
    }
    if (own && !mine)
#pragma unroll
      for (int s = 0; s < 4; ++s)
        if (k0 + s < mt) store(me.c, k0 + s, t[s]);
  }
  /* the results in the rows below */
#pragma unroll
  for (int s = 0; s < 4; ++s)
#pragma unroll
    for (int j = 0; j < RJ; ++j) {
      const int k = P.m + row_of(me, j) - P.r0;
      if (k >= P.m && k < P.steps && me.cb + s < n && !(pivots && (k & ~3) == me.cb)) store(me.cb + s, k, b[s][j]);
    }
  if (me.rhs)
#pragma unroll
    for (int v = 0; v < 2; ++v)
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int qm = v ? P1.m : P0.m, k = qm + 4 * me.lane + u - (v ? P1.r0 : P0.r0);
        if (k >= qm && k < (v ? P1.steps : P0.steps)) storer(v, k, r[v][u]);
      }
  __syncthreads();
}

/* the weighed observations of level 0, made upper trapezoidal: two steps a block */
template <int RJ>
__global__ void __launch_bounds__(NT, 1) triangularize(CArgs<float> a, int64_t nsteps)
{
  extern __shared__ __align__(16) float wide_dyn[];
  const Shared<RJ> sh(wide_dyn);
  const Me me;
  const int n = a.n;
  int64_t q[2];
  int m[2];
#pragma unroll
  for (int v = 0; v < 2; ++v) {
    const int64_t g = 2 * (int64_t)blockIdx.x + v;
    q[v] = 0;
    m[v] = 0;
    if (g < nsteps) {
      const int t = find_track(a.track_start, a.ntracks, g);
      q[v] = a.ct.slot[t] + (g - a.track_start[t]);
      m[v] = a.ce.m[q[v]];
    }
  }
  float b[4][RJ], r[2][4];
  const int64_t q0 = q[0], q1 = q[1];
  float* G = &a.ce.G.at(0, me.half ? q1 : q0);
  load_cols<RJ>(me, G, a.mx, n, me.half ? m[1] : m[0], b);
#pragma unroll
  for (int v = 0; v < 2; ++v) load_rhs(me, &a.ce.o.at(0, q[v]), me.rhs ? m[v] : 0, r[v]);
  reduce<RJ>(sh, me, n, Panel{0, 0, m[0]}, Panel{0, 0, m[1]}, b, r, [](int) { return 0.f; },
             [&](int c, int k, float v) { G[c * a.mx + k] = k > c ? 0.f : v; }, [](int, int) { return 0.f; },
             [&](int w, int k, float v) { a.ce.o.at(k, w ? q1 : q0) = v; });
}

template <int RJ>
__global__ void __launch_bounds__(NT, 1) pair_wide(CArgs<float> a)
{
  extern __shared__ __align__(16) float wide_dyn[];
  const Shared<RJ> sh(wide_dyn);
  const Me me;
  const int n = a.n, mx = a.mx, ldt = n | 1;
  const auto& C = a.ce;
  const auto& Nx = a.ne;
  const auto& Rr = a.cr;
  const int64_t item = blockIdx.x;
  const int t = find_track(a.ct.pair, a.ntracks, item);
  const int64_t p = item - a.ct.pair[t];
  const int64_t sj = a.ct.slot[t] + 2 * p, sj1 = sj + 1;
  const int64_t sn = a.nt.slot[t] + p, se = a.ct.solve[t] + p;
  const int mj = C.m[sj], mj1 = C.m[sj1], nC = mj + mj1 < n ? mj + mj1 : n;
  const bool h0 = me.half == 0, h1 = me.half == 1;
  float b[4][RJ], r[2][4];
  float* Tr = sh.T + n * ldt;
  float* Y = &Rr.Y.at(0, se); /* Y~ waits in the record */
  load_cols<RJ>(me, h0 ? &C.F.at(0, sj1) : &C.H.at(0, sj1), n, n, n, b);
  load_rhs(me, &C.c.at(0, sj1), me.rhs ? n : 0, r[0]);
  {
    const float* top = &C.G.at(me.c * mx, sj);
    const float* o = &C.o.at(0, sj);
    reduce<RJ>(sh, me, n, Panel{mj, 0, n}, Panel{0, 0, -1}, b, r, [&](int k) { return h0 && k <= me.c ? top[k] : 0.f; },
               [&](int c, int k, float v) {
                 if (h0) sh.T[c * ldt + k] = k > c ? 0.f : v;
                 else Y[c * n + k] = v;
               },
               [&](int, int k) { return o[k]; }, [&](int, int k, float v) { Tr[k] = v; });
  }
#pragma unroll
  for (int u = 0; u < 4; ++u) r[1][u] = r[0][u]; /* o~; H~ is in half 1's registers */
  if (h0) load_cols<RJ>(me, &C.H.at(0, sj), n, n, p > 0 ? n : 0, b);
  load_rhs(me, &C.c.at(0, sj), me.rhs && p > 0 ? n : 0, r[0]);
  {
    const float* top = &C.G.at(me.c * mx, sj1);
    const float* o = &C.o.at(0, sj1);
    const float* Tc = sh.T + me.c * ldt;
    float* out = h0 ? &Rr.R.at(0, se) : &Nx.G.at(0, sn);
    const int ld = h0 ? n : mx;
    reduce<RJ>(sh, me, n, Panel{n, 0, p > 0 ? n : 0}, Panel{mj1, n - mj, nC}, b, r,
               [&](int k) { return k > me.c ? 0.f : h0 ? Tc[k] : top[k]; },
               [&](int c, int k, float v) { out[c * ld + k] = k > c ? 0.f : v; },
               [&](int w, int k) { return w ? o[k] : Tr[k]; },
               [&](int w, int k, float v) { (w ? Nx.o.at(k, sn) : Rr.rhs.at(k, se)) = v; });
    if (threadIdx.x == 0) Nx.m[sn] = nC;
    if (p == 0) { /* no stage B: the record is stage A's */
      if (h0 && me.c < n)
        for (int k = 0; k < n; ++k) out[me.c * n + k] = Tc[k];
      if (me.rhs)
        for (int k = me.lane; k < n; k += 32) Rr.rhs.at(k, se) = Tr[k];
      for (int e = threadIdx.x; e < n * n; e += NT) Rr.Ft.at(e, se) = 0.f;
      return;
    }
  }
  if (me.rhs)
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (4 * me.lane + u < n) Nx.c.at(4 * me.lane + u, sn) = r[0][u];
  /* [Y~; 0] in half 1, whose threads wrote Y~, [0; F_j] in half 0; no barriers */
  load_cols<RJ>(me, &C.F.at(0, sj), n, n, h0 ? n : 0, b);
  const bool own = me.c < n;
  float* out = (h0 ? &Rr.Ft.at(0, se) : Y) + (own ? me.c : 0) * n;
  float next = own && h1 ? out[0] : 0.f;
#pragma unroll 1
  for (int k = 0; k < n; ++k) {
    float tk = next, x[RJ];
    next = own && h1 && k + 1 < n ? out[k + 1] : 0.f;
    const float am = sh.am[k], iv = sh.iv[k];
    if (!(iv < 0.f)) {
      const float d = fmaf(am, tk, dots<RJ>(me, sh.V + k * 4 * RJ, x, b)) * iv;
      tk = fmaf(-d, am, tk);
      update<RJ>(me, d, x, b);
    }
    if (own) out[k] = tk;
  }
  store_cols<RJ>(me, h0 ? &Nx.F.at(0, sn) : &Nx.H.at(0, sn), n, b);
}

template <int RJ>
__global__ void __launch_bounds__(NT, 1) tail_wide(CArgs<float> a)
{
  extern __shared__ __align__(16) float wide_dyn[];
  const Shared<RJ> sh(wide_dyn);
  const Me me;
  const int n = a.n, mx = a.mx, c = threadIdx.x;
  const auto& C = a.ce;
  const auto& Nx = a.ne;
  const auto& Rr = a.cr;
  const int t = (int)a.ct.tail[blockIdx.x];
  const int64_t L = a.ct.L[t], sb = a.ct.slot[t];
  if (L == 1) { /* base case: x = R^{-1} o */
    const bool piv = c < n;
    float* Rt = sh.T;
    double* x = a.state + orig_step(a.track_start, a.level, t, 0) * n;
    if (C.m[sb] < n) {
      if (piv) x[c] = NAN;
      if (c == 0) atomicOr(a.flag, 2);
      return;
    }
    for (int e = c; e < n * n; e += NT) {
      const int q = e / n, r = e - q * n;
      const float v = r <= q ? C.G.at(q * mx + r, sb) : 0.f;
      sh.V[e] = v;
      if (r == q && v == 0.f) atomicOr(a.flag, 2);
      if (a.baseR.p) a.baseR.at(e, t) = v;
    }
    if (piv) Rt[c] = C.o.at(c, sb);
    __syncthreads();
    for (int i = n - 1; i >= 0; --i) { /* thread r subtracts x_i R(r, i) */
      const float xi = Rt[i] / sh.V[i * n + i];
      __syncthreads();
      if (c == i) Rt[i] = xi;
      if (c < i) Rt[c] = fmaf(-xi, sh.V[i * n + c], Rt[c]);
      __syncthreads();
    }
    if (piv) x[c] = ukg_df::widen(Rt[c]);
    return;
  }
  const int64_t s = sb + L - 1, es = a.ct.solve[t] + (L - 1) / 2, sn = a.nt.slot[t] + L / 2 - 1;
  const int mt = C.m[s], gp = Nx.m[sn], nF = gp + mt < n ? gp + mt : n;
  const bool h0 = me.half == 0;
  float b[4][RJ], r[2][4];
  /* [R~ | o' | 0; H_s | c_s | F_s] */
  load_cols<RJ>(me, h0 ? &C.H.at(0, s) : &C.F.at(0, s), n, n, n, b);
  load_rhs(me, &C.c.at(0, s), me.rhs ? n : 0, r[0]);
  {
    const float* top = &C.G.at(me.c * mx, s);
    const float* o = &C.o.at(0, s);
    float* out = h0 ? &Rr.R.at(0, es) : &Rr.Ft.at(0, es);
    reduce<RJ>(sh, me, n, Panel{mt, 0, n}, Panel{0, 0, -1}, b, r, [&](int k) { return h0 && k <= me.c ? top[k] : 0.f; },
               [&](int c, int k, float v) { out[c * n + k] = h0 && k > c ? 0.f : v; },
               [&](int, int k) { return o[k]; }, [&](int, int k, float v) { Rr.rhs.at(k, es) = v; });
  }
  for (int e = c; e < n * n; e += NT) Rr.Y.at(e, es) = 0.f;
#pragma unroll
  for (int u = 0; u < 4; ++u) r[1][u] = r[0][u];
  /* fix-up: [G~ | o; Z | o''], Z in half 1's registers */
  {
    float* G = &Nx.G.at(0, sn);
    reduce<RJ>(sh, me, n, Panel{0, 0, 0}, Panel{gp, n - mt, nF}, b, r, [&](int k) { return k > me.c ? 0.f : G[me.c * mx + k]; },
               [&](int c, int k, float v) { G[c * mx + k] = k > c ? 0.f : v; }, [&](int, int k) { return Nx.o.at(k, sn); },
               [&](int, int k, float v) { Nx.o.at(k, sn) = v; });
  }
  if (c == 0) Nx.m[sn] = nF;
}

/* the kernels of a state dimension; mx == n */
struct Kernels {
  void (*triangularize)(CArgs<float>, int64_t) = nullptr;
  void (*pair)(CArgs<float>) = nullptr;
  void (*tail)(CArgs<float>) = nullptr;
  size_t smem = 0;
};
template <int RJ>
Kernels kernels_rj(int n)
{
  Kernels k;
  k.triangularize = triangularize<RJ>;
  k.pair = pair_wide<RJ>;
  k.tail = tail_wide<RJ>;
  k.smem = smem<RJ>(n);
  return k;
}
template <typename T> /* T: float, so that the other arithmetics' compilations have none of them */
Kernels kernels(int n, int mx)
{
  if (n != mx || n < 65 || n > 128) return Kernels();
  return n <= 96 ? kernels_rj<24>(n) : kernels_rj<32>(n);
}

}  // namespace wide
