/*
 * oddeven_small.cuh -- the odd-even smoother's kernels for 2 to 8 states (and no
 * more observation rows than states), in FP64, double-float and FP32 (whose
 * solves are oddeven.cu's), in two mappings with the same arithmetic, entry by
 * entry.  Included by oddeven.cu (it uses that file's Args, tables and views).
 *
 *   *_lanes   a group of LPI lanes (32 or 8) shares a work item, a column of
 *             the current panel per lane and slot, in registers; reflectors
 *             travel by shuffles.
 *   *_thread  one thread per item, its pivot block in registers.
 *
 * What bounds them: on GB300 a warp's FP64 instruction occupies its
 * scheduler's quarter of the SM for 64 cycles (76 with all four busy),
 * whether 1 or 32 of its lanes work, and independent chains do not overlap
 * (measured).  A thread that factors a pair alone is a chain of about 3,000
 * such instructions, 100 us; a warp with a column per lane needs 340, but a
 * full chip's worth of pairs costs three times as much that way.  So levels
 * with few items take lanes and levels with many take threads, and since both
 * run the same operations in the same order on every entry, which of them a
 * level takes (that is, how many tracks are smoothed together) changes no
 * result bit.
 *
 * Structure.  From level 1 on an observation block is the triangular factor
 * that stage C left, and stage B's R~ is triangular at every level.  With the
 * triangular block on top and the square one below, reflector k is one top
 * row and the n rows below: n rows instead of 2n - k - 1, and no fill-in (the
 * "triangle on top of a square" QR of blocked tile algorithms).  Items whose
 * observations have fewer than n rows (level 0, unobserved steps) stack the
 * rows without gaps instead: a zero row in between would pick up rounding
 * errors and count as an observation.
 */
#pragma once

namespace small {

using namespace ::lanes;

constexpr int kLaneWarps = 4; /* warps per block of the lane kernels: one per scheduler of an SM */

/* First entries (element indices) of the columns in a level's equations and
 * in its records: each is one array of elements with one stride (eq_at and
 * rec in run_plan), so a lane reaches any column of any kind with one base
 * address and one stride, without branches.                                 */
template <int N>
struct Col {
  static constexpr int F = 0, H = N * N, c = 2 * N * N, G = c + N, o = G + N * N; /* Eq, mx == N */
  static constexpr int R = 0, Ft = N * N, Y = 2 * N * N, rhs = 3 * N * N;         /* Rec         */
};
template <typename T, int N>
__device__ __forceinline__ void load_col(const Soa<T>& first, int e, int64_t s, bool on, T (&v)[N])
{
  const T* p = first.p + (int64_t)e * first.stride + s;
#pragma unroll
  for (int i = 0; i < N; ++i, p += first.stride) {
    v[i] = T(0);
    if (on) v[i] = *p;
  }
}
template <typename T, int N>
__device__ __forceinline__ void store_col(const Soa<T>& first, int e, int64_t s, int rows, const T (&v)[N])
{
  T* p = first.p + (int64_t)e * first.stride + s;
#pragma unroll
  for (int i = 0; i < N; ++i, p += first.stride)
    if (i < rows) *p = v[i];
}

/* ---------------------------------------------------------------------------
 * odd-length tracks, one warp each: the single last step s (observation QR,
 * then [H_s F_s c_s; R~ 0 o']) and the fix-up of the next level's last
 * observation, or the one-step base case.
 * ------------------------------------------------------------------------ */
template <typename T, int N>
__device__ __forceinline__ void tail_item(const Args<T, T>& a, int tr, T* hb, int lane)
{
  using K = Col<N>;
  const unsigned gm = 0xffffffffu;
  const Soa<T>&C = a.ce.F, &Nx = a.ne.F, &Rr = a.cr.R;
  const int64_t L = a.ct.L[tr], sb = a.ct.slot[tr];
  const int64_t s = sb + L - 1; /* the last step (the only one if L == 1) */
  const int ms = a.ce.m[s], mt = ms; /* m <= mx == N */
  T t[1][N], b[1][N];
  /* [G_s | o_s] on lanes 0..N; from level 1 on it is triangular already */
  load_col<T, N>(C, lane < N ? K::G + lane * N : K::o, s, lane <= N, t[0]);
  T q[N];
  load_col<T, N>(C, lane < N ? K::H + lane * N : lane == N ? K::c : K::F + (lane - N - 1) * N, s,
                 L > 1 && lane <= 2 * N, q);
#pragma unroll
  for (int i = 0; i < N; ++i) {
    b[0][i] = T(0);
    if (i >= ms) t[0][i] = T(0);
  }
  if (a.level == 0) lanes_qr_full<T, N, 32, 1, N>(t, b, gm, lane, 0, mt);

  if (L == 1) { /* base case: x = R^{-1} Q^T o, S = R^{-1} R^{-T} */
    const int64_t os = orig_step(a.track_start, a.level, tr, 0);
    double* x = a.state + os * N;
    double* Sg = a.cov ? a.cov + os * (int64_t)N * N : nullptr;
    if (ms < N) {
      if (lane < N) x[lane] = NAN;
      if (Sg)
        for (int e = lane; e < N * N; e += 32) Sg[e] = NAN;
      if (lane == 0) atomicOr(a.flag, 2);
      return;
    }
    if (lane < N) {
#pragma unroll
      for (int i = 0; i < N; ++i) hb[lane * N + i] = i <= lane ? t[0][i] : T(0);
    }
    if (lane < N && a.baseR.p)
#pragma unroll
      for (int i = 0; i < N; ++i) a.baseR.at(lane * N + i, tr) = i <= lane ? t[0][i] : T(0);
    __syncwarp();
    T dg = T(1);
    if (lane < N) dg = hb[lane * N + lane];
    if (lane < N && dg == T(0)) atomicOr(a.flag, 2);
    const T dv = recip(dg);
    /* R x = y on lane N, R r = e_q on lanes q < N */
    T v[N];
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = lane == N ? t[0][i] : i == lane ? T(1) : T(0);
#pragma unroll
    for (int j = N - 1; j >= 0; --j) {
      v[j] = v[j] * shfl(gm, dv, j, 32);
#pragma unroll
      for (int i = 0; i < j; ++i) v[i] = fma(-v[j], hb[j * N + i], v[i]);
    }
    if (lane == N)
#pragma unroll
      for (int i = 0; i < N; ++i) x[i] = ukg_df::widen(v[i]);
    if (Sg) {
      __syncwarp();
      if (lane < N)
#pragma unroll
        for (int i = 0; i < N; ++i) hb[lane * N + i] = v[i];
      __syncwarp();
      for (int e = lane; e < N * N; e += 32) {
        const int j = e / N, i = e - j * N;
        T sm = T(0);
        for (int k = i > j ? i : j; k < N; ++k) sm = fma(hb[k * N + i], hb[k * N + j], sm);
        Sg[e] = ukg_df::widen(sm);
      }
    }
    return;
  }

  const int64_t es = a.ct.solve[tr] + (L - 1) / 2;
  const int64_t sn = a.nt.slot[tr] + L / 2 - 1;
  const bool tri = mt == N; /* R~ is triangular after its QR at every level */
  /* [H_s | c_s | F_s; R~ | o' | 0]: pivots on lanes 0..N-1, the right-hand
     side on N, F_s on N+1..2N; R~ on top when it has all n rows */
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const T r = lane <= N && i <= lane && i < mt ? t[0][i] : T(0);
    t[0][i] = tri ? r : q[i];
    b[0][i] = tri ? q[i] : r;
  }
  if (tri) lanes_qr_tri<T, N, 32, 1>(t, b, gm, lane, 0, N);
  else lanes_qr_full<T, N, 32, 1, N>(t, b, gm, lane, 0, N);
  T zero[N];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    zero[i] = T(0);
    if (lane < N && i > lane) t[0][i] = T(0);
    if (lane >= N && lane <= 2 * N) hb[(lane == N ? N : lane - N - 1) * N + i] = b[0][i];
  }
  store_col<T, N>(Rr, lane < N ? K::R + lane * N : lane == N ? K::rhs : K::Ft + (lane - N - 1) * N, es,
                  lane <= 2 * N ? N : 0, t[0]);
  store_col<T, N>(Rr, K::Y + lane * N, es, lane < N ? N : 0, zero);
  __syncwarp();
  /* fix-up: [G~ | o; Z | o''], mt rows of Z; stacked without a gap unless both are full */
  const int gp = a.ne.m[sn], rF = gp + mt, nF = rF < N ? rF : N;
  const bool triF = tri && gp == N;
  const int eg = lane < N ? K::G + lane * N : K::o;
  const T* g = Nx.p + (int64_t)eg * Nx.stride + sn;
#pragma unroll
  for (int r = 0; r < 2 * N; ++r) {
    T v = T(0);
    if (lane <= N && r < gp) v = g[r * Nx.stride];
    else if (lane <= N && r < rF) v = hb[lane * N + r - gp];
    (r < N ? t[0][r] : b[0][r - N]) = v;
  }
  __syncwarp();
  if (triF) lanes_qr_tri<T, N, 32, 1>(t, b, gm, lane, 0, N);
  else lanes_qr_full<T, N, 32, 1, N>(t, b, gm, lane, 0, nF);
#pragma unroll
  for (int i = 0; i < N; ++i)
    if (lane < N && i > lane) t[0][i] = T(0);
  store_col<T, N>(Nx, eg, sn, lane <= N ? nF : 0, t[0]);
  if (lane == 0) a.ne.m[sn] = nF;
}

__host__ __device__ constexpr int tail_entries(int n) { return (2 * n + 1) * n; } /* tail_item's shared memory */

template <typename T, int N>
__global__ void __launch_bounds__(32 * kLaneWarps) tail_lanes(Args<T, T> a)
{
  __shared__ T buf[kLaneWarps][tail_entries(N)];
  const int w = threadIdx.x >> 5;
  const int64_t item = (int64_t)blockIdx.x * kLaneWarps + w;
  if (item < a.ct.ntail) tail_item<T, N>(a, (int)a.ct.tail[item], buf[w], threadIdx.x & 31); /* the whole warp */
}

/* ---------------------------------------------------------------------------
 * forward elimination of a pair (j, j+1) by a group of LPI lanes.
 * Stage A's columns: 0..N-1 pivots, N right-hand side, N+1..2N H_{j+1};
 * stage B's: the same with Y~ in place of H, then 2N+1..3N F_j; stage C's:
 * 0..N-1 pivots, N right-hand side -- with LPI = 32 and N <= 7 on the lanes
 * 3N+1..4N+1 at the same time as stage B.
 * With 32 lanes the level's tails are part of the launch: the warp of an odd
 * track's last pair goes on to the fix-up, and the warps past the pairs take
 * the tracks that have one step left.
 * ------------------------------------------------------------------------ */
template <typename T, int N, int LPI>
__global__ void __launch_bounds__(32 * kLaneWarps) pair_lanes(Args<T, T> a)
{
  using K = Col<N>;
  constexpr int S = (3 * N + 1 + LPI - 1) / LPI, SC = (N + 1 + LPI - 1) / LPI;
  constexpr bool kMerge = LPI == 32 && 4 * N + 2 <= 32;
  constexpr int GPB = 32 * kLaneWarps / LPI; /* groups per block */
  /* H~ and o~ of the group's item: column q's rows at q * N */
  __shared__ T hbuf[GPB][LPI == 32 ? tail_entries(N) : (N + 1) * N];
  const int grp = threadIdx.x / LPI, lane = threadIdx.x % LPI;
  const unsigned gm = LPI == 32 ? 0xffffffffu : ((1u << (LPI & 31)) - 1u) << ((threadIdx.x & 31) / LPI * LPI);
  const int64_t item = (int64_t)blockIdx.x * GPB + grp;
  T* hb = hbuf[grp];
  if (item >= a.ct.npairs) { /* the whole group */
    if (LPI == 32 && item - a.ct.npairs < a.ct.ntail) {
      const int tr = (int)a.ct.tail[item - a.ct.npairs];
      if (a.ct.L[tr] == 1) tail_item<T, N>(a, tr, hb, lane);
    }
    return;
  }
  const Soa<T>&C = a.ce.F, &Nx = a.ne.F, &Rr = a.cr.R;
  const int tr = find_track(a.ct.pair, a.ntracks, item);
  const int64_t p = item - a.ct.pair[tr];
  const int64_t sj = a.ct.slot[tr] + 2 * p, sj1 = sj + 1;
  const int64_t sn = a.nt.slot[tr] + p;
  const int64_t se = a.ct.solve[tr] + p;
  const int mj = a.ce.m[sj], mj1 = a.ce.m[sj1];

  /* everything the pair reads is on its way before the first reflector: the
     rows of G_j, those of F_{j+1} with H_{j+1}, stage B's lower rows
     [H_j | c_j | 0 | F_j] */
  constexpr bool kEarly = S < 4; /* n = 8 on eight lanes: the registers are needed */
  T t[S][N], b[S][N], lo[S][N];
  auto load_lo = [&](int s, T (&v)[N]) {
    const int c = s * LPI + lane;
    load_col<T, N>(C, c < N ? K::H + c * N : c == N ? K::c : K::F + (c - 2 * N - 1) * N, sj,
                   p > 0 && (c <= N || (c > 2 * N && c <= 3 * N)), v);
  };
#pragma unroll
  for (int s = 0; s < S; ++s) {
    const int c = s * LPI + lane;
    load_col<T, N>(C, c < N ? K::G + c * N : K::o, sj, c <= N, t[s]);
    load_col<T, N>(C, c < N ? K::F + c * N : c == N ? K::c : K::H + (c - N - 1) * N, sj1, c <= 2 * N, b[s]);
    if (kEarly) load_lo(s, lo[s]);
  }
  const int cm = lane - (3 * N + 1); /* kMerge: this lane's column of stage C */
  T tc[SC][N], bc[SC][N];
  auto load_tc = [&](int s) {
    const int c = kMerge ? cm : s * LPI + lane;
    load_col<T, N>(C, c < N ? K::G + c * N : K::o, sj1, c >= 0 && c <= N, tc[s]);
  };
  if (kEarly)
#pragma unroll
    for (int s = 0; s < SC; ++s) load_tc(s);
  const bool tri = a.level > 0 && mj == N && mj1 == N;
  /* stage A: [G_j | o_j | 0; F_{j+1} | c_{j+1} | H_{j+1}], the triangular G_j
     on top, or F_{j+1} on top and the rows of G_j below */
  if (tri) {
    lanes_qr_tri<T, N, LPI, S>(t, b, gm, lane, 0, N);
  } else {
#pragma unroll
    for (int s = 0; s < S; ++s)
#pragma unroll
      for (int i = 0; i < N; ++i) {
        const T g = i < mj ? t[s][i] : T(0);
        t[s][i] = b[s][i];
        b[s][i] = g;
      }
    lanes_qr_full<T, N, LPI, S, N>(t, b, gm, lane, 0, N);
  }
  /* H~ and o~ (m_j rows) to the group's buffer */
#pragma unroll
  for (int s = 0; s < S; ++s) {
    const int c = s * LPI + lane;
    if (c >= N && c <= 2 * N) {
      T* h = hb + (c == N ? N : c - N - 1) * N;
#pragma unroll
      for (int i = 0; i < N; ++i) h[i] = b[s][i];
    }
  }
  __syncwarp(gm);
  /* stage C's rows: the triangular [G_{j+1} | o_{j+1}] on top of [H~ | o~],
     or the m_j + m_{j+1} rows of both without a gap */
  const int rC = mj + mj1, nC = rC < N ? rC : N;
#pragma unroll
  for (int s = 0; s < SC; ++s) {
    if (!kEarly) load_tc(s);
    const int c = kMerge ? cm : s * LPI + lane;
    const bool on = c >= 0 && c <= N;
    const T* h = hb + (on ? c : 0) * N;
    if (tri) {
#pragma unroll
      for (int i = 0; i < N; ++i) bc[s][i] = on ? h[i] : T(0);
    } else { /* row r: H~'s for r < m_j, then G_{j+1}'s */
      const T* g = C.p + (int64_t)(c < N ? K::G + c * N : K::o) * C.stride + sj1;
#pragma unroll
      for (int r = 0; r < 2 * N; ++r) {
        T v = T(0);
        if (on && r < mj) v = h[r];
        else if (on && r < rC) v = g[(r - mj) * C.stride];
        (r < N ? tc[s][r] : bc[s][r - N]) = v;
      }
    }
  }
  /* stage B's panel: R~, rhs~, Y~ stay where stage A left them; [0 ; F_j] joins */
#pragma unroll
  for (int s = 0; s < S; ++s) {
    const int c = s * LPI + lane;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      if ((c < N && i > c) || c > 2 * N) t[s][i] = T(0);
      if (kEarly) b[s][i] = lo[s][i];
    }
    if (!kEarly) load_lo(s, b[s]);
  }
  if constexpr (kMerge) {
    const bool lc = cm >= 0;
    if (lc)
#pragma unroll
      for (int i = 0; i < N; ++i) t[0][i] = tc[0][i], b[0][i] = bc[0][i];
    const int nref = lc ? nC : p > 0 ? N : 0, base = lc ? 3 * N + 1 : 0;
    if (tri) lanes_qr_tri<T, N, LPI, S>(t, b, gm, lane, base, nref);
    else lanes_qr_full<T, N, LPI, S, N>(t, b, gm, lane, base, nref);
#pragma unroll
    for (int i = 0; i < N; ++i) tc[0][i] = t[0][i];
  } else {
    if (tri) lanes_qr_tri<T, N, LPI, SC>(tc, bc, gm, lane, 0, nC);
    else lanes_qr_full<T, N, LPI, SC, N>(tc, bc, gm, lane, 0, nC);
    if (p > 0) lanes_qr_tri<T, N, LPI, S>(t, b, gm, lane, 0, N);
  }
  if (lane == 0) a.ne.m[sn] = nC;
  /* the next level's observation */
#pragma unroll
  for (int s = 0; s < SC; ++s) {
    const int c = kMerge ? cm : s * LPI + lane;
#pragma unroll
    for (int i = 0; i < N; ++i)
      if (c < N && i > c) tc[s][i] = T(0);
    store_col<T, N>(Nx, c < N ? K::G + c * N : K::o, sn, c >= 0 && c <= N ? nC : 0, tc[s]);
  }
  /* records (Ft is zero for a track's first pair) and the next level's evolution */
#pragma unroll
  for (int s = 0; s < S; ++s) {
    const int c = s * LPI + lane;
#pragma unroll
    for (int i = 0; i < N; ++i)
      if (c < N && i > c) t[s][i] = T(0);
    const int er = c < N ? K::R + c * N : c == N ? K::rhs : c <= 2 * N ? K::Y + (c - N - 1) * N
                                                                       : K::Ft + (c - 2 * N - 1) * N;
    const int en = c == N ? K::c : c <= 2 * N ? K::H + (c - N - 1) * N : K::F + (c - 2 * N - 1) * N;
    store_col<T, N>(Rr, er, se, c <= 3 * N ? N : 0, t[s]);
    store_col<T, N>(Nx, en, sn, p > 0 && c >= N && c <= 3 * N ? N : 0, b[s]);
  }
  if constexpr (LPI == 32) {
    const int64_t L = a.ct.L[tr];
    if ((L & 1) && 2 * p + 3 == L) {
      __syncwarp(); /* the next level's slot is this warp's own */
      tail_item<T, N>(a, tr, hb, lane);
    }
  }
}

/* ---------------------------------------------------------------------------
 * forward elimination of a pair by one thread: the operations of pair_lanes,
 * column by column.  The pivot block, its reflectors and the column they are
 * streamed over are registers; Y~ and H~ wait in the record and next-level
 * arrays they go to.  Stage B runs before stage C, so R~ stays in registers.
 * ------------------------------------------------------------------------ */
/* triangle t on top of the square x: reflectors stay in x, am, iv */
template <typename T, int N>
__device__ __forceinline__ void thread_qr_tri(T (&t)[N][N], T (&x)[N][N], T (&am)[N], T (&iv)[N])
{
#pragma unroll
  for (int k = 0; k < N; ++k) {
    Dot<T> sq;
#pragma unroll
    for (int i = 0; i < N; ++i) sq.add(x[k][i], x[k][i]);
    const T tail = sq.value();
    am[k] = iv[k] = T(0);
    if (tail == T(0)) continue;
    const Refl<T> r = reflector(t[k][k], tail);
    t[k][k] = r.beta;
    am[k] = r.amb;
    iv[k] = r.inv;
#pragma unroll
    for (int c = k + 1; c < N; ++c) {
      Dot<T> xa;
#pragma unroll
      for (int i = 0; i < N; ++i) xa.add(x[k][i], x[c][i]);
      const T d = fma(r.amb, t[c][k], xa.value()) * r.inv;
      t[c][k] = fma(-d, r.amb, t[c][k]);
#pragma unroll
      for (int i = 0; i < N; ++i) x[c][i] = fma(-d, x[k][i], x[c][i]);
    }
  }
}
template <typename T, int N>
__device__ __forceinline__ void thread_apply_tri(const T (&x)[N][N], const T (&am)[N], const T (&iv)[N], T (&ct)[N],
                                                 T (&cb)[N])
{
#pragma unroll
  for (int k = 0; k < N; ++k) {
    Dot<T> xa;
#pragma unroll
    for (int i = 0; i < N; ++i) xa.add(x[k][i], cb[i]);
    const T d = fma(am[k], ct[k], xa.value()) * iv[k];
    ct[k] = fma(-d, am[k], ct[k]);
#pragma unroll
    for (int i = 0; i < N; ++i) cb[i] = fma(-d, x[k][i], cb[i]);
  }
}
/* R x N panel p (columns), reflectors below the diagonal in p */
template <typename T, int N, int R>
__device__ __forceinline__ void thread_qr_full(T (&p)[N][R], T (&am)[N], T (&iv)[N], int nref)
{
#pragma unroll
  for (int k = 0; k < N; ++k) {
    am[k] = iv[k] = T(0);
    if (k >= R) continue;
    Dot<T> sq;
#pragma unroll
    for (int i = k + 1; i < R; ++i) sq.add(p[k][i], p[k][i]);
    const T tail = sq.value();
    if (tail == T(0) || k >= nref) continue;
    const Refl<T> r = reflector(p[k][k], tail);
    p[k][k] = r.beta;
    am[k] = r.amb;
    iv[k] = r.inv;
#pragma unroll
    for (int c = k + 1; c < N; ++c) {
      Dot<T> xa;
#pragma unroll
      for (int i = k + 1; i < R; ++i) xa.add(p[k][i], p[c][i]);
      const T d = fma(r.amb, p[c][k], xa.value()) * r.inv;
      p[c][k] = fma(-d, r.amb, p[c][k]);
#pragma unroll
      for (int i = k + 1; i < R; ++i) p[c][i] = fma(-d, p[k][i], p[c][i]);
    }
  }
}
template <typename T, int N, int R>
__device__ __forceinline__ void thread_apply_full(const T (&p)[N][R], const T (&am)[N], const T (&iv)[N], T (&c)[R])
{
#pragma unroll
  for (int k = 0; k < N; ++k) {
    if (k >= R) continue;
    Dot<T> xa;
#pragma unroll
    for (int i = k + 1; i < R; ++i) xa.add(p[k][i], c[i]);
    const T d = fma(am[k], c[k], xa.value()) * iv[k];
    c[k] = fma(-d, am[k], c[k]);
#pragma unroll
    for (int i = k + 1; i < R; ++i) c[i] = fma(-d, p[k][i], c[i]);
  }
}

struct PairIdx {
  int64_t sj, sj1, sn, se;
  int mj, mj1;
};

/* stage A with F_{j+1} on top and up to MB rows of G_j below */
template <typename T, int N, int MB>
__device__ __forceinline__ void thread_a_full(const Args<T, T>& a, const PairIdx& I, T (&t)[N][N], T (&vt)[N])
{
  constexpr int R = N + MB;
  const Eq<T>& C = a.ce;
  T p[N][R], v[R], am[N], iv[N];
#pragma unroll
  for (int c = 0; c < N; ++c) {
#pragma unroll
    for (int i = 0; i < N; ++i) p[c][i] = C.F.at(c * N + i, I.sj1);
#pragma unroll
    for (int i = 0; i < MB; ++i) p[c][N + i] = i < I.mj ? C.G.at(c * N + i, I.sj) : T(0);
  }
#pragma unroll
  for (int i = 0; i < N; ++i) v[i] = C.c.at(i, I.sj1);
#pragma unroll
  for (int i = 0; i < MB; ++i) v[N + i] = i < I.mj ? C.o.at(i, I.sj) : T(0);
  thread_qr_full<T, N, R>(p, am, iv, N);
  thread_apply_full<T, N, R>(p, am, iv, v);
#pragma unroll
  for (int i = 0; i < MB; ++i)
    if (i < I.mj) a.ne.o.at(i, I.sn) = v[N + i];
  T hn[N]; /* the next column, on its way */
#pragma unroll
  for (int i = 0; i < N; ++i) hn[i] = C.H.at(i, I.sj1);
#pragma unroll 1
  for (int q = 0; q < N; ++q) {
    T h[R];
#pragma unroll
    for (int i = 0; i < R; ++i) h[i] = i < N ? hn[i] : T(0);
    if (q + 1 < N)
#pragma unroll
      for (int i = 0; i < N; ++i) hn[i] = C.H.at((q + 1) * N + i, I.sj1);
    thread_apply_full<T, N, R>(p, am, iv, h);
#pragma unroll
    for (int i = 0; i < N; ++i) a.cr.Y.at(q * N + i, I.se) = h[i];
#pragma unroll
    for (int i = 0; i < MB; ++i)
      if (i < I.mj) a.ne.G.at(q * N + i, I.sn) = h[N + i];
  }
#pragma unroll
  for (int c = 0; c < N; ++c)
#pragma unroll
    for (int i = 0; i < N; ++i) t[c][i] = i <= c ? p[c][i] : T(0);
#pragma unroll
  for (int i = 0; i < N; ++i) vt[i] = v[i];
}

/* stage C on up to RC stacked rows */
template <typename T, int N, int RC>
__device__ __forceinline__ void thread_c_full(const Args<T, T>& a, const PairIdx& I)
{
  const Eq<T>& C = a.ce;
  const Eq<T>& Nx = a.ne;
  const int rC = I.mj + I.mj1, nC = rC < N ? rC : N;
  T p[N][RC], v[RC], am[N], iv[N];
#pragma unroll
  for (int c = 0; c < N; ++c)
#pragma unroll
    for (int i = 0; i < RC; ++i)
      p[c][i] = i < I.mj ? Nx.G.at(c * N + i, I.sn) : i < rC ? C.G.at(c * N + i - I.mj, I.sj1) : T(0);
#pragma unroll
  for (int i = 0; i < RC; ++i) v[i] = i < I.mj ? Nx.o.at(i, I.sn) : i < rC ? C.o.at(i - I.mj, I.sj1) : T(0);
  thread_qr_full<T, N, RC>(p, am, iv, nC);
  thread_apply_full<T, N, RC>(p, am, iv, v);
#pragma unroll
  for (int c = 0; c < N; ++c)
#pragma unroll
    for (int i = 0; i < N; ++i)
      if (i < nC && i < RC) Nx.G.at(c * N + i, I.sn) = i <= c ? p[c][i] : T(0);
#pragma unroll
  for (int i = 0; i < N; ++i)
    if (i < nC && i < RC) Nx.o.at(i, I.sn) = v[i];
}

template <typename T, int N, int BS, int MINB>
__global__ void __launch_bounds__(BS, MINB) pair_thread(Args<T, T> a)
{
  const int64_t item = (int64_t)blockIdx.x * BS + threadIdx.x;
  if (item >= a.ct.npairs) return;
  const Eq<T>& C = a.ce;
  const Eq<T>& Nx = a.ne;
  const Rec<T>& Rr = a.cr;
  const int tr = find_track(a.ct.pair, a.ntracks, item);
  const int64_t p = item - a.ct.pair[tr];
  PairIdx I;
  I.sj = a.ct.slot[tr] + 2 * p;
  I.sj1 = I.sj + 1;
  I.sn = a.nt.slot[tr] + p;
  I.se = a.ct.solve[tr] + p;
  I.mj = C.m[I.sj];
  I.mj1 = C.m[I.sj1];
  const bool tri = a.level > 0 && I.mj == N && I.mj1 == N;
  constexpr int MH = (N + 1) / 2;
  T t[N][N], vt[N];
  /* stage A */
  if (tri) {
    T x[N][N], am[N], iv[N], vb[N];
#pragma unroll
    for (int c = 0; c < N; ++c)
#pragma unroll
      for (int i = 0; i < N; ++i) {
        t[c][i] = i <= c ? C.G.at(c * N + i, I.sj) : T(0);
        x[c][i] = C.F.at(c * N + i, I.sj1);
      }
#pragma unroll
    for (int i = 0; i < N; ++i) vt[i] = C.o.at(i, I.sj), vb[i] = C.c.at(i, I.sj1);
    thread_qr_tri<T, N>(t, x, am, iv);
    thread_apply_tri<T, N>(x, am, iv, vt, vb);
#pragma unroll
    for (int i = 0; i < N; ++i) Nx.o.at(i, I.sn) = vb[i];
    T hn[N]; /* the next column, on its way */
#pragma unroll
    for (int i = 0; i < N; ++i) hn[i] = C.H.at(i, I.sj1);
#pragma unroll 1
    for (int q = 0; q < N; ++q) {
      T ht[N], hb[N];
#pragma unroll
      for (int i = 0; i < N; ++i) ht[i] = T(0), hb[i] = hn[i];
      if (q + 1 < N)
#pragma unroll
        for (int i = 0; i < N; ++i) hn[i] = C.H.at((q + 1) * N + i, I.sj1);
      thread_apply_tri<T, N>(x, am, iv, ht, hb);
#pragma unroll
      for (int i = 0; i < N; ++i) {
        Rr.Y.at(q * N + i, I.se) = ht[i];
        Nx.G.at(q * N + i, I.sn) = hb[i];
      }
    }
  } else if (I.mj <= MH) {
    thread_a_full<T, N, MH>(a, I, t, vt);
  } else {
    thread_a_full<T, N, N>(a, I, t, vt);
  }
  /* stage B: [R~ | rhs~ | Y~ | 0; H_j | c_j | 0 | F_j] */
  if (p > 0) {
    T x[N][N], am[N], iv[N], vb[N];
#pragma unroll
    for (int c = 0; c < N; ++c)
#pragma unroll
      for (int i = 0; i < N; ++i) x[c][i] = C.H.at(c * N + i, I.sj);
#pragma unroll
    for (int i = 0; i < N; ++i) vb[i] = C.c.at(i, I.sj);
    thread_qr_tri<T, N>(t, x, am, iv);
    thread_apply_tri<T, N>(x, am, iv, vt, vb);
#pragma unroll
    for (int i = 0; i < N; ++i) Nx.c.at(i, I.sn) = vb[i];
    T nx[N]; /* the next column, on its way: F_j's, then Y~'s */
#pragma unroll
    for (int i = 0; i < N; ++i) nx[i] = C.F.at(i, I.sj);
#pragma unroll 1
    for (int q = 0; q < 2 * N; ++q) {
      const bool isF = q < N;
      const int c = isF ? q : q - N;
      T ct[N], cb[N];
#pragma unroll
      for (int i = 0; i < N; ++i) {
        ct[i] = isF ? T(0) : nx[i];
        cb[i] = isF ? nx[i] : T(0);
      }
      if (q + 1 < 2 * N) {
        const T* src = q + 1 < N ? &C.F.at((q + 1) * N, I.sj) : &Rr.Y.at((q + 1 - N) * N, I.se);
        const int64_t st = q + 1 < N ? C.F.stride : Rr.Y.stride;
#pragma unroll
        for (int i = 0; i < N; ++i) nx[i] = src[i * st];
      }
      thread_apply_tri<T, N>(x, am, iv, ct, cb);
      const Soa<T> top{&(isF ? Rr.Ft : Rr.Y).at(c * N, I.se), Rr.R.stride};
      const Soa<T> bot{&(isF ? Nx.F : Nx.H).at(c * N, I.sn), Nx.F.stride};
#pragma unroll
      for (int i = 0; i < N; ++i) {
        top.at(i, 0) = ct[i];
        bot.at(i, 0) = cb[i];
      }
    }
  } else {
    for (int e = 0; e < N * N; ++e) Rr.Ft.at(e, I.se) = T(0);
  }
#pragma unroll
  for (int c = 0; c < N; ++c)
#pragma unroll
    for (int i = 0; i < N; ++i) Rr.R.at(c * N + i, I.se) = i <= c ? t[c][i] : T(0);
#pragma unroll
  for (int i = 0; i < N; ++i) Rr.rhs.at(i, I.se) = vt[i];
  /* stage C */
  if (tri) {
    T x[N][N], am[N], iv[N], vb[N];
#pragma unroll
    for (int c = 0; c < N; ++c)
#pragma unroll
      for (int i = 0; i < N; ++i) {
        t[c][i] = i <= c ? C.G.at(c * N + i, I.sj1) : T(0);
        x[c][i] = Nx.G.at(c * N + i, I.sn);
      }
#pragma unroll
    for (int i = 0; i < N; ++i) vt[i] = C.o.at(i, I.sj1), vb[i] = Nx.o.at(i, I.sn);
    thread_qr_tri<T, N>(t, x, am, iv);
    thread_apply_tri<T, N>(x, am, iv, vt, vb);
#pragma unroll
    for (int c = 0; c < N; ++c)
#pragma unroll
      for (int i = 0; i < N; ++i) Nx.G.at(c * N + i, I.sn) = i <= c ? t[c][i] : T(0);
#pragma unroll
    for (int i = 0; i < N; ++i) Nx.o.at(i, I.sn) = vt[i];
    Nx.m[I.sn] = N;
  } else {
    const int rC = I.mj + I.mj1;
    if (rC <= N) thread_c_full<T, N, N>(a, I);
    else thread_c_full<T, N, 2 * N>(a, I);
    Nx.m[I.sn] = rC < N ? rC : N;
  }
}

/* ---------------------------------------------------------------------------
 * odd-length tracks by one thread each, the operations of tail_item: for levels
 * that end many tracks.  A warp a tail is 32 lanes for 2 N + 1 columns, and
 * thousands of tracks of a few steps are little but tails: 20,000 tracks of 3
 * steps, FP64, n = 4, the tails of both levels (with the pairs' launch) 461 us
 * before, 126 now, n = 6 880 and 297.
 * ------------------------------------------------------------------------ */
constexpr int kTailThreadBS = 64;

template <typename T, int N>
__device__ __forceinline__ void load_cols(const Soa<T>& first, int e, int64_t s, int rows, T (&p)[N][N])
{
#pragma unroll
  for (int c = 0; c < N; ++c)
#pragma unroll
    for (int i = 0; i < N; ++i) p[c][i] = i < rows ? first.at(e + c * N + i, s) : T(0);
}

/* x = R^{-1} y, S = R^{-1} R^{-T} of a track's only step */
template <typename T, int N>
__device__ __forceinline__ void base_thread(const Args<T, T>& a, int tr, const T (&R)[N][N], T (&y)[N], PVc<T, kTailThreadBS> Ri)
{
  const int64_t os = orig_step(a.track_start, a.level, tr, 0);
  double* x = a.state + os * N;
  T dv[N];
  bool bad = false;
#pragma unroll
  for (int c = 0; c < N; ++c) {
    bad |= R[c][c] == T(0);
    dv[c] = recip(R[c][c]);
    if (a.baseR.p)
#pragma unroll
      for (int i = 0; i < N; ++i) a.baseR.at(c * N + i, tr) = i <= c ? R[c][i] : T(0);
  }
  if (bad) atomicOr(a.flag, 2);
  auto solve = [&](T (&v)[N], int top) {
#pragma unroll
    for (int j = N - 1; j >= 0; --j) {
      if (j > top) continue;
      v[j] = v[j] * dv[j];
#pragma unroll
      for (int i = 0; i < j; ++i) v[i] = fma(-v[j], R[j][i], v[i]);
    }
  };
  solve(y, N - 1);
#pragma unroll
  for (int i = 0; i < N; ++i) x[i] = ukg_df::widen(y[i]);
  if (!a.cov) return;
  double* S = a.cov + os * (int64_t)N * N;
#pragma unroll
  for (int q = 0; q < N; ++q) {
    T v[N];
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = i == q ? T(1) : T(0);
    solve(v, q);
#pragma unroll
    for (int i = 0; i < N; ++i) Ri[q * N + i] = v[i];
  }
#pragma unroll 1
  for (int j = 0; j < N; ++j)
#pragma unroll 1
    for (int i = 0; i < N; ++i) {
      T sm = T(0);
      for (int k = i > j ? i : j; k < N; ++k) sm = fma(Ri[k * N + i], Ri[k * N + j], sm);
      S[j * N + i] = ukg_df::widen(sm);
    }
}

template <typename T, int N>
__global__ void __launch_bounds__(kTailThreadBS) tail_thread(Args<T, T> a)
{
  __shared__ T buf[kTailThreadBS * (N + 1) * N];
  const PVc<T, kTailThreadBS> Z{buf + threadIdx.x}; /* the rows left over, column by column; or R^{-1} */
  const int64_t item = (int64_t)blockIdx.x * kTailThreadBS + threadIdx.x;
  if (item >= a.ct.ntail) return;
  using K = Col<N>;
  const int tr = (int)a.ct.tail[item];
  const Soa<T>&C = a.ce.F, &Nx = a.ne.F, &Rr = a.cr.R;
  const int64_t L = a.ct.L[tr], s = a.ct.slot[tr] + L - 1;
  const int mt = a.ce.m[s];
  T p[N][N], v[N], am[N], iv[N];
  load_cols<T, N>(C, K::G, s, mt, p);
#pragma unroll
  for (int i = 0; i < N; ++i) v[i] = i < mt ? C.at(K::o + i, s) : T(0);
  if (a.level == 0) {
    thread_qr_full<T, N, N>(p, am, iv, mt);
    thread_apply_full<T, N, N>(p, am, iv, v);
  }
  if (L == 1) {
    if (mt < N) {
      const int64_t os = orig_step(a.track_start, a.level, tr, 0);
      for (int i = 0; i < N; ++i) a.state[os * N + i] = NAN;
      if (a.cov)
        for (int i = 0; i < N * N; ++i) a.cov[os * N * N + i] = NAN;
      atomicOr(a.flag, 2);
    } else {
      base_thread<T, N>(a, tr, p, v, Z);
    }
    return;
  }
  const int64_t es = a.ct.solve[tr] + (L - 1) / 2, sn = a.nt.slot[tr] + L / 2 - 1;
  const bool tri = mt == N;
  T q[N][N], w[N];
  load_cols<T, N>(C, K::H, s, N, q);
#pragma unroll
  for (int i = 0; i < N; ++i) w[i] = C.at(K::c + i, s);
#pragma unroll
  for (int c = 0; c < N; ++c)
#pragma unroll
    for (int i = 0; i < N; ++i)
      if (i > c || i >= mt) p[c][i] = T(0);
  /* [R~ | o' | 0; H_s | c_s | F_s], or H_s on top of the mt rows of R~ */
  if (tri) {
    thread_qr_tri<T, N>(p, q, am, iv);
    thread_apply_tri<T, N>(q, am, iv, v, w);
#pragma unroll
    for (int i = 0; i < N; ++i) Rr.at(K::rhs + i, es) = v[i], Z[N * N + i] = w[i];
#pragma unroll 1
    for (int c = 0; c < N; ++c) {
      T ft[N], fb[N];
#pragma unroll
      for (int i = 0; i < N; ++i) ft[i] = T(0), fb[i] = C.at(K::F + c * N + i, s);
      thread_apply_tri<T, N>(q, am, iv, ft, fb);
#pragma unroll
      for (int i = 0; i < N; ++i) Rr.at(K::Ft + c * N + i, es) = ft[i], Z[c * N + i] = fb[i];
    }
  } else {
    T g[N][2 * N], u[2 * N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
      u[i] = w[i], u[N + i] = v[i];
#pragma unroll
      for (int c = 0; c < N; ++c) g[c][i] = q[c][i], g[c][N + i] = p[c][i];
    }
    thread_qr_full<T, N, 2 * N>(g, am, iv, N);
    thread_apply_full<T, N, 2 * N>(g, am, iv, u);
#pragma unroll
    for (int i = 0; i < N; ++i) {
      Rr.at(K::rhs + i, es) = u[i], Z[N * N + i] = u[N + i];
#pragma unroll
      for (int c = 0; c < N; ++c) p[c][i] = g[c][i];
    }
#pragma unroll 1
    for (int c = 0; c < N; ++c) {
#pragma unroll
      for (int i = 0; i < N; ++i) u[i] = C.at(K::F + c * N + i, s), u[N + i] = T(0);
      thread_apply_full<T, N, 2 * N>(g, am, iv, u);
#pragma unroll
      for (int i = 0; i < N; ++i) Rr.at(K::Ft + c * N + i, es) = u[i], Z[c * N + i] = u[N + i];
    }
  }
#pragma unroll
  for (int c = 0; c < N; ++c)
#pragma unroll
    for (int i = 0; i < N; ++i) {
      Rr.at(K::R + c * N + i, es) = i <= c ? p[c][i] : T(0);
      Rr.at(K::Y + c * N + i, es) = T(0);
    }
  /* fix-up: [G~ | o; Z | o''], mt rows of Z; stacked without a gap unless both are full */
  const int gp = a.ne.m[sn], rF = gp + mt, nF = rF < N ? rF : N;
  if (tri && gp == N) {
    load_cols<T, N>(Nx, K::G, sn, N, p);
#pragma unroll
    for (int i = 0; i < N; ++i) {
      v[i] = Nx.at(K::o + i, sn), w[i] = Z[N * N + i];
#pragma unroll
      for (int c = 0; c < N; ++c) q[c][i] = Z[c * N + i];
    }
    thread_qr_tri<T, N>(p, q, am, iv);
    thread_apply_tri<T, N>(q, am, iv, v, w);
  } else {
    T g[N][2 * N], u[2 * N];
#pragma unroll
    for (int c = 0; c <= N; ++c)
#pragma unroll
      for (int r = 0; r < 2 * N; ++r) {
        T x = T(0);
        if (r < gp) x = Nx.at((c < N ? K::G + c * N : K::o) + r, sn);
        else if (r < rF) x = Z[c * N + r - gp];
        (c < N ? g[c < N ? c : 0][r] : u[r]) = x;
      }
    thread_qr_full<T, N, 2 * N>(g, am, iv, nF);
    thread_apply_full<T, N, 2 * N>(g, am, iv, u);
#pragma unroll
    for (int i = 0; i < N; ++i) {
      v[i] = u[i];
#pragma unroll
      for (int c = 0; c < N; ++c) p[c][i] = g[c][i];
    }
  }
#pragma unroll
  for (int i = 0; i < N; ++i)
    if (i < nF) {
      Nx.at(K::o + i, sn) = v[i];
#pragma unroll
      for (int c = 0; c < N; ++c) Nx.at(K::G + c * N + i, sn) = i <= c ? p[c][i] : T(0);
    }
  a.ne.m[sn] = nF;
}

/* ---------------------------------------------------------------------------
 * back-substitution of an even step, with its covariance and the blocks
 * cov(x_{j-1}, x_j), cov(x_j, x_{j+1}):
 *   W = B Sigma, M = I + W B^T (its lower triangle), X = R^{-1} M,
 *   S = R^{-1} X^T (its lower triangle), blocks -R^{-1} W.
 * One warp per step: lanes 0..2N-1 a column of Sigma each, lane 2N the
 * neighbours' states (so x_j is one more column), lanes 2N+1..3N the columns
 * of M; every entry in the order of solve_thread.
 * ------------------------------------------------------------------------ */
struct SolveIdx {
  int tr;
  int64_t j, oj, om, op, smp;
  bool hp, hn;
};
template <typename T>
__device__ __forceinline__ SolveIdx solve_index(const Args<T, T>& a, int64_t item)
{
  SolveIdx I;
  I.tr = find_track(a.ct.solve, a.ntracks, item);
  I.j = 2 * (item - a.ct.solve[I.tr]);
  const int64_t L = a.ct.L[I.tr];
  I.hp = I.j > 0;
  I.hn = I.j + 1 < L;
  I.oj = orig_step(a.track_start, a.level, I.tr, I.j);
  I.om = I.hp ? orig_step(a.track_start, a.level, I.tr, I.j - 1) : 0;
  I.op = I.hn ? orig_step(a.track_start, a.level, I.tr, I.j + 1) : 0;
  I.smp = I.hp && I.hn ? a.nt.slot[I.tr] + (I.j + 1) / 2 : 0; /* U of the next level */
  return I;
}

template <typename T, int N>
__global__ void __launch_bounds__(32 * kLaneWarps) solve_lanes(Args<T, T> a)
{
  constexpr int NN = N * N;
  struct Buf {
    T B[2 * NN], W[2 * NN], R[NN], M[NN];
  };
  __shared__ Buf bufs[kLaneWarps];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t item = (int64_t)blockIdx.x * kLaneWarps + w;
  if (item >= a.ct.nsolve) return; /* the whole warp */
  const unsigned gm = 0xffffffffu;
  Buf& B = bufs[w];
  const Rec<T>& Rr = a.cr;
  const SolveIdx I = solve_index(a, item);
  const bool isx = lane == 2 * N;
  T sg[2 * N], pv[N];
  { /* column `lane` of Sigma: FP64 outputs from one side, U from the other; the negated states on lane 2N */
    const double* d = isx ? a.state + I.om * N : lane < N ? a.cov + I.om * NN + lane * N
                                                          : a.cov + I.op * NN + (lane - N) * N;
    const double* d2 = a.state + I.op * N;
    const int64_t us = a.nr.U.stride;
    const T* u = a.nr.U.p + (lane < N ? (int64_t)lane : (int64_t)(lane - N) * N) * us + I.smp;
    const int64_t ui = lane < N ? N * us : us;
    const bool ond = lane < N ? I.hp : lane < 2 * N ? I.hn : isx && I.hp;
    const bool onu = lane < 2 * N && I.hp && I.hn, on2 = isx && I.hn;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      double v = 0.0, v2 = 0.0;
      T w2 = T(0);
      if (ond) v = d[i];
      if (on2) v2 = d2[i];
      if (onu) w2 = u[i * ui];
      if (isx) v = -v, v2 = -v2;
      const T x = ukg_df::narrow<T>(v), x2 = on2 ? ukg_df::narrow<T>(v2) : w2;
      sg[i] = lane < N || isx ? x : w2;
      sg[N + i] = lane < N ? w2 : isx ? x2 : x;
      pv[i] = isx ? Rr.rhs.at(i, item) : T(0);
    }
  }
  for (int e = lane; e < NN; e += 32) {
    B.B[e] = I.hp ? Rr.Ft.at(e, item) : T(0);
    B.B[NN + e] = I.hn ? Rr.Y.at(e, item) : T(0);
    B.R[e] = Rr.R.at(e, item);
  }
  __syncwarp();
  T dg = T(1);
  if (lane < N) dg = B.R[lane * N + lane];
  if (lane < N && dg == T(0)) atomicOr(a.flag, 2);
  const T dv = recip(dg);
  if (I.hp)
#pragma unroll
    for (int k = 0; k < N; ++k)
#pragma unroll
      for (int i = 0; i < N; ++i) pv[i] = fma(B.B[k * N + i], sg[k], pv[i]);
  if (I.hn)
#pragma unroll
    for (int k = 0; k < N; ++k)
#pragma unroll
      for (int i = 0; i < N; ++i) pv[i] = fma(B.B[NN + k * N + i], sg[N + k], pv[i]);
  if (lane < 2 * N)
#pragma unroll
    for (int i = 0; i < N; ++i) B.W[lane * N + i] = pv[i];
  __syncwarp();
  const int q0 = I.hp ? 0 : N, q1 = I.hn ? 2 * N : N;
  for (int e = lane; e < N * (N + 1) / 2; e += 32) { /* entry (i, c) of M, i >= c */
    int c = 0, r = e;
    while (r >= N - c) r -= N - c, ++c;
    const int i = c + r;
    T m = T(0);
    for (int q = q0; q < q1; ++q) m = fma(B.W[q * N + i], B.B[q * N + c], m);
    if (i == c) m += T(1);
    B.M[c * N + i] = B.M[i * N + c] = m;
  }
  __syncwarp();
  const int mc = lane - (2 * N + 1); /* this lane's column of M */
  const bool ism = mc >= 0 && mc < N;
  if (ism)
#pragma unroll
    for (int i = 0; i < N; ++i) pv[i] = B.M[mc * N + i];
#pragma unroll
  for (int j = N - 1; j >= 0; --j) {
    pv[j] = pv[j] * shfl(gm, dv, j, 32);
#pragma unroll
    for (int i = 0; i < j; ++i) pv[i] = fma(-pv[j], B.R[j * N + i], pv[i]);
  }
  if (isx)
#pragma unroll
    for (int i = 0; i < N; ++i) a.state[I.oj * N + i] = ukg_df::widen(pv[i]);
  if (a.level > 0 && lane < 2 * N) { /* level 0's off-diagonal blocks are not needed */
    const int64_t sU = a.ct.slot[I.tr] + I.j;
    /* cov(x_{j-1}, x_j): row `lane`; cov(x_j, x_{j+1}): column lane - N */
    const int64_t us = Rr.U.stride;
    T* u = Rr.U.p + (lane < N ? lane * us + sU : (lane - N) * N * us + sU + 1);
    const int64_t ui = lane < N ? N * us : us;
    if (lane < N ? I.hp : I.hn)
#pragma unroll
      for (int i = 0; i < N; ++i) u[i * ui] = -pv[i];
  }
  __syncwarp();
  if (ism)
#pragma unroll
    for (int i = 0; i < N; ++i) B.M[mc * N + i] = pv[i]; /* X, column mc */
  __syncwarp();
  if (ism)
#pragma unroll
    for (int i = 0; i < N; ++i) pv[i] = B.M[i * N + mc]; /* X^T, column mc */
#pragma unroll
  for (int j = N - 1; j >= 0; --j) {
    pv[j] = pv[j] * shfl(gm, dv, j, 32);
#pragma unroll
    for (int i = 0; i < j; ++i) pv[i] = fma(-pv[j], B.R[j * N + i], pv[i]);
  }
  if (ism) {
    double* So = a.cov + I.oj * NN;
#pragma unroll
    for (int i = 0; i < N; ++i)
      if (i >= mc) {
        const double v = ukg_df::widen(pv[i]);
        So[mc * N + i] = v;
        So[i * N + mc] = v;
      }
  }
}

/* One thread per even step: R, the reciprocals of its diagonal and the lower
 * triangle of M in registers, F~ and Y in the thread's shared-memory slice.
 * The symmetric halves of M and S are computed once (a sixth of the FP64
 * instructions of the full products).                                       */
template <typename T, int N, int BS>
__global__ void __launch_bounds__(BS) solve_thread(Args<T, T> a)
{
  extern __shared__ unsigned char smem_raw[];
  T* smem = reinterpret_cast<T*>(smem_raw);
  const int64_t item = (int64_t)blockIdx.x * BS + threadIdx.x;
  if (item >= a.ct.nsolve) return;
  constexpr int NN = N * N;
  const Rec<T>& Rr = a.cr;
  const SolveIdx I = solve_index(a, item);
  const bool hp = I.hp, hn = I.hn;
  PVc<T, BS> Fs{smem + threadIdx.x}, Ys = Fs + NN;
  T R[N][N], dv[N];
  bool bad = false;
#pragma unroll
  for (int c = 0; c < N; ++c)
#pragma unroll
    for (int i = 0; i <= c; ++i) R[i][c] = Rr.R.at(c * N + i, item);
#pragma unroll 6
  for (int k = 0; k < NN; ++k) {
    Fs[k] = hp ? Rr.Ft.at(k, item) : T(0);
    Ys[k] = hn ? Rr.Y.at(k, item) : T(0);
  }
#pragma unroll
  for (int i = 0; i < N; ++i) {
    bad |= (R[i][i] == T(0));
    dv[i] = recip(R[i][i]);
  }
  auto solve = [&](T (&x)[N], int r0) { /* x <- R^{-1} x, entries r0 and up */
#pragma unroll
    for (int j = N - 1; j >= 0; --j) {
      if (j < r0) continue;
      x[j] = x[j] * dv[j];
#pragma unroll
      for (int i = 0; i < j; ++i)
        if (i >= r0) x[i] = fma(-x[j], R[i][j], x[i]);
    }
  };
  T pv[N];
#pragma unroll
  for (int i = 0; i < N; ++i) pv[i] = Rr.rhs.at(i, item);
  if (hp)
    for (int k = 0; k < N; ++k) {
      const T xk = ukg_df::narrow<T>(a.state[I.om * N + k]);
#pragma unroll
      for (int i = 0; i < N; ++i) pv[i] = fma(-Fs[k * N + i], xk, pv[i]);
    }
  if (hn)
    for (int k = 0; k < N; ++k) {
      const T xk = ukg_df::narrow<T>(a.state[I.op * N + k]);
#pragma unroll
      for (int i = 0; i < N; ++i) pv[i] = fma(-Ys[k * N + i], xk, pv[i]);
    }
  solve(pv, 0);
#pragma unroll
  for (int i = 0; i < N; ++i) a.state[I.oj * N + i] = ukg_df::widen(pv[i]);

  const double* Smm = hp ? a.cov + I.om * NN : nullptr;
  const double* Spp = hn ? a.cov + I.op * NN : nullptr;
  T M[N][N]; /* M[c][i]: column c, row i >= c */
#pragma unroll
  for (int c = 0; c < N; ++c)
#pragma unroll
    for (int i = c; i < N; ++i) M[c][i] = T(0);
  const int q0 = hp ? 0 : N, q1 = hn ? 2 * N : N;
#pragma unroll 1
  for (int q = q0; q < q1; ++q) {
    T sg[2 * N];
    if (q < N) {
#pragma unroll
      for (int i = 0; i < N; ++i) {
        sg[i] = ukg_df::narrow<T>(Smm[q * N + i]);
        sg[N + i] = hn ? a.nr.U.at(i * N + q, I.smp) : T(0);
      }
    } else {
#pragma unroll
      for (int i = 0; i < N; ++i) {
        sg[i] = hp ? a.nr.U.at((q - N) * N + i, I.smp) : T(0);
        sg[N + i] = ukg_df::narrow<T>(Spp[(q - N) * N + i]);
      }
    }
#pragma unroll
    for (int i = 0; i < N; ++i) pv[i] = T(0);
    if (hp)
#pragma unroll
      for (int k = 0; k < N; ++k)
#pragma unroll
        for (int i = 0; i < N; ++i) pv[i] = fma(Fs[k * N + i], sg[k], pv[i]);
    if (hn)
#pragma unroll
      for (int k = 0; k < N; ++k)
#pragma unroll
        for (int i = 0; i < N; ++i) pv[i] = fma(Ys[k * N + i], sg[N + k], pv[i]);
    PVc<T, BS> bq = q < N ? Fs + q * N : Ys + (q - N) * N; /* column q of B = [F~ | Y] */
#pragma unroll
    for (int c = 0; c < N; ++c) {
      const T bc = bq[c];
#pragma unroll
      for (int i = c; i < N; ++i) M[c][i] = fma(pv[i], bc, M[c][i]);
    }
    if (a.level == 0) continue;
    solve(pv, 0);
    const int64_t sU = a.ct.slot[I.tr] + I.j;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      if (q < N) Rr.U.at(i * N + q, sU) = -pv[i];
      else Rr.U.at((q - N) * N + i, sU + 1) = -pv[i];
    }
  }
  /* X = R^{-1} M column by column into the slice (F~ and Y are spent), then
     the columns of X^T */
#pragma unroll
  for (int c = 0; c < N; ++c) {
    T x[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
      x[i] = i >= c ? M[c][i] : M[i][c];
      if (i == c) x[i] += T(1);
    }
    solve(x, 0);
#pragma unroll
    for (int i = 0; i < N; ++i) Fs[c * N + i] = x[i];
  }
  double* So = a.cov + I.oj * NN;
#pragma unroll
  for (int c = 0; c < N; ++c) {
    T x[N];
#pragma unroll
    for (int i = 0; i < N; ++i) x[i] = Fs[i * N + c];
    solve(x, c);
#pragma unroll
    for (int i = c; i < N; ++i) {
      const double v = ukg_df::widen(x[i]);
      So[c * N + i] = v;
      So[i * N + c] = v;
    }
  }
  if (bad) atomicOr(a.flag, 2);
}

/* the state alone: the same operations as the other two solves' state       */
template <typename T, int N>
__global__ void __launch_bounds__(64) solve_state(Args<T, T> a)
{
  const int64_t item = (int64_t)blockIdx.x * 64 + threadIdx.x;
  if (item >= a.ct.nsolve) return;
  const Rec<T>& Rr = a.cr;
  const SolveIdx I = solve_index(a, item);
  T pv[N], x[N];
#pragma unroll
  for (int i = 0; i < N; ++i) pv[i] = Rr.rhs.at(i, item);
  if (I.hp) {
#pragma unroll
    for (int k = 0; k < N; ++k) x[k] = -ukg_df::narrow<T>(a.state[I.om * N + k]);
#pragma unroll
    for (int k = 0; k < N; ++k)
#pragma unroll
      for (int i = 0; i < N; ++i) pv[i] = fma(Rr.Ft.at(k * N + i, item), x[k], pv[i]);
  }
  if (I.hn) {
#pragma unroll
    for (int k = 0; k < N; ++k) x[k] = -ukg_df::narrow<T>(a.state[I.op * N + k]);
#pragma unroll
    for (int k = 0; k < N; ++k)
#pragma unroll
      for (int i = 0; i < N; ++i) pv[i] = fma(Rr.Y.at(k * N + i, item), x[k], pv[i]);
  }
  bool bad = false;
#pragma unroll
  for (int j = N - 1; j >= 0; --j) {
    const T d = Rr.R.at(j * N + j, item);
    bad |= d == T(0);
    pv[j] = pv[j] * recip(d);
#pragma unroll
    for (int i = 0; i < j; ++i) pv[i] = fma(-pv[j], Rr.R.at(j * N + i, item), pv[i]);
  }
#pragma unroll
  for (int i = 0; i < N; ++i) a.state[I.oj * N + i] = ukg_df::widen(pv[i]);
  if (bad) atomicOr(a.flag, 2);
}

}  // namespace small
