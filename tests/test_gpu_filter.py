"""Filtered estimates on the device (kalman_gpu_filter_packed, the sequential
UltimateKalman filter of c/kalman_ultimate.c run per track): the estimate and
covariance of step s equal the oracle's smoothed estimate and covariance of
the last step of the track cut after s (the filtered estimate is the smoothed
one of the prefix problem).  Tolerance 1e-10 relative (states and
covariances): different elimination orders of the same FP64 least-squares
problems."""
import numpy as np
import pytest

import oracle
from ultimate_kalman_gb300 import native
from ultimate_kalman_gb300 import problem as pb

pytestmark = pytest.mark.gpu
TOL = 1e-10


def _cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    return torch


def prefixes(P):
    """Every prefix of every track as its own track; returns the packed
    problem and, per original step, the index of its prefix's last step."""
    idx, lens, last = [], [], []
    for t in range(P.ntracks):
        a, b = int(P.track_start[t]), int(P.track_start[t + 1])
        for L in range(1, b - a + 1):
            idx.extend(range(a, a + L))
            lens.append(L)
            last.append(len(idx) - 1)
    idx = np.array(idx)
    ts = np.zeros(len(lens) + 1, dtype=np.int64)
    ts[1:] = np.cumsum(lens)
    Q = pb.PackedProblem(n=P.n, mmax=P.mmax, track_start=ts, **{f: getattr(P, f)[idx] for f in (
        "H", "F", "c", "K", "K_type", "G", "o", "C", "C_type", "obs_rows")})
    return Q, np.array(last)


@pytest.mark.parametrize("n,m,kt,ct", [(6, 3, "C", "C"), (4, 2, "W", "w"), (12, 6, "C", "W"), (9, 4, "F", "C")])
def test_filtered_estimates_equal_prefix_smoothing(n, m, kt, ct):
    _cuda()
    P = pb.random_dynamics([23, 1, 9, 14], n, m, seed=40 + n, per_step=True, missing=0.15, K_type=kt, C_type=ct)
    D = native.DeviceProblem(P, covariance=True)
    D.filter()
    X, S = D.results()
    Q, last = prefixes(P)
    st, Xo, So = oracle.smooth(Q, "oddeven", covariance=True)
    assert st == 0
    assert oracle.rel_err_states(X, Xo[last]) < TOL
    assert oracle.rel_err_covs(S, So[last]) < TOL


def test_last_filtered_estimate_is_the_smoothed_one():
    """At a track's last step filtering and smoothing use the same equations."""
    _cuda()
    P = pb.random_dynamics([300, 77], 8, 4, seed=5, missing=0.1)
    D = native.DeviceProblem(P, covariance=True)
    D.filter()
    Xf, Sf = D.results()
    D.smooth("oddeven")
    Xs, Ss = D.results()
    ends = P.track_start[1:] - 1
    assert oracle.rel_err_states(Xf[ends], Xs[ends]) < TOL
    assert oracle.rel_err_covs(Sf[ends], Ss[ends]) < TOL


def test_states_only_and_undetermined_steps():
    """Without covariances only states are written; steps whose state is not
    yet determined (step 0 unobserved, then 2 observation rows a step for 4
    states) are NaN and the call reports it."""
    torch = _cuda()
    P = pb.random_dynamics([12], 4, 2, seed=8)
    P.obs_rows[0] = 0
    P.obs_rows[1:] = 2
    D = native.DeviceProblem(P, covariance=False)
    status = D.filter(covariance=False, check=False)
    assert status == native.KALMAN_GPU_ESINGULAR
    X = D.state.cpu().numpy()
    assert np.isnan(X[:2]).all()
    assert np.isfinite(X[2:]).all()


@pytest.mark.parametrize("n,m,mmax,kt,ct", [(1, 1, 1, "C", "C"), (3, 2, 8, "w", "F"), (5, 2, 5, "F", "W"),
                                            (7, 8, 8, "C", "w"), (8, 4, 8, "W", "C")])
def test_small_states_in_rounds(n, m, mmax, kt, ct):
    """Up to 8 states the tracks are filtered a round of steps at a time (128 MiB
    of weighed equations): one track alone (one round) equals the oracle's
    prefix smoothing, and enough copies of it for several rounds give the
    same bits."""
    _cuda()
    P = pb.random_dynamics([41], n, m, seed=n + 50, per_step=True, missing=0.2, K_type=kt, C_type=ct)
    if P.mmax < mmax:
        g = np.zeros((41, n, mmax))
        g[:, :, :P.mmax] = P.G
        o = np.zeros((41, mmax))
        o[:, :P.mmax] = P.o
        c = np.zeros((41, mmax, mmax))
        for s in range(41):
            if P.C_type[s] == ord("w"):
                c[s].reshape(-1)[:P.mmax] = P.C[s].reshape(-1)[:P.mmax]
            else:
                c[s, :P.mmax, :P.mmax] = P.C[s]
        P = pb.PackedProblem(n, mmax, P.track_start, P.H, P.F, P.c, P.K, P.K_type, g, o, c, P.C_type, P.obs_rows)
    D = native.DeviceProblem(P, covariance=True)
    D.filter()
    X, S = D.results()
    Q, last = prefixes(P)
    st, Xo, So = oracle.smooth(Q, "oddeven", covariance=True)
    assert st == 0
    assert oracle.rel_err_states(X, Xo[last]) < TOL
    assert oracle.rel_err_covs(S, So[last]) < TOL
    T = int((128 << 20) // (8 * ((2 * n + 1) * n + (n + 1) * mmax) * 41)) * 5 // 2 if n >= 7 else 50
    B = P.select_tracks([0] * T)
    D = native.DeviceProblem(B, covariance=True)
    D.filter()
    Xb, Sb = D.results()
    assert (Xb.reshape(T, 41, n) == X).all() and (Sb.reshape(T, 41, n, n) == S).all()


def _no_prior(n, rows, F, K=None, seed=0):
    """One track without a prior: step s observes the rows `rows[s]` (a list of
    vectors of n entries, maybe none); covariances drawn per step."""
    rng = np.random.default_rng(seed)
    k, m = len(rows), max(len(r) for r in rows)
    P = pb.empty_problem(n, max(n, m), [k])
    x = rng.standard_normal(n)
    for s in range(k):
        P.H[s] = np.eye(n)
        P.F[s] = F.T
        P.c[s] = 0.1 * rng.standard_normal(n)
        P.K[s] = pb.random_spd(rng, n) if K is None else K
        x = F @ x + rng.standard_normal(n)
        r = len(rows[s])
        P.obs_rows[s] = r
        if r:
            G = np.array(rows[s])
            P.G[s, :, :r] = G.T
            P.o[s, :r] = G @ x + rng.standard_normal(r)
            P.C[s, :r, :r] = pb.random_spd(rng, r)
    return P


def _pv(n, order):
    """Positions that move by 0.1 times their velocities: [p.. v..], [v.. p..] or [p v p v ..]."""
    h = n // 2
    p = {"pv": np.arange(h), "vp": h + np.arange(h), "mixed": 2 * np.arange(h)}[order]
    v = {"pv": h + np.arange(h), "vp": np.arange(h), "mixed": 2 * np.arange(h) + 1}[order]
    F = np.eye(n)
    F[p, v] = 0.1
    return F, p


def _undetermined_starts():
    out = {}
    for n, order in ((2, "vp"), (4, "mixed"), (4, "vp"), (6, "pv"), (6, "vp"), (8, "mixed"), (8, "vp"), (10, "vp")):
        F, p = _pv(n, order)
        out[f"{order}{n}"] = (n, [np.eye(n)[p]] * 6, F)
    F, p = _pv(4, "mixed")
    e = np.eye(4)
    out["alternating"] = (4, [[e[2 * (s % 2)]] for s in range(8)], F)
    out["late"] = (4, [[], []] + [e[p]] * 5, F)
    out["between"] = (4, [e[p], [], e[p], [], [], e[p]], F)
    F, _ = _pv(2, "pv")
    e = np.eye(2)
    out["repeated_row"] = (2, [e[[0, 0]], [], e[[0]], e[[0]]], F)
    F3 = np.array([[1, 0.1, 0.005], [0, 1, 0.1], [0, 0, 1.0]])
    e = np.eye(3)
    out["position_acceleration"] = (3, [e[[0, 2]]] * 6, F3)
    out["one_position"] = (3, [e[[0]]] * 6, F3)
    out["last_first"] = (3, [e[[2]], e[[0]], e[[0, 2]], e[[0]], e[[0]]], F3)
    for n in (3, 6, 8, 9):  # the leading columns depend on each other
        rng = np.random.default_rng(n)
        G = rng.standard_normal((2, n))
        G[:, 1] = 2.0 * G[:, 0]
        out[f"dependent{n}"] = (n, [G] * (n // 2 + 4), pb.random_orthogonal(rng, n))
    return out


@pytest.mark.parametrize("cov", [True, False], ids=["cov", "states"])
@pytest.mark.parametrize("name", list(_undetermined_starts()))
def test_tracks_without_a_prior(name, cov):
    """A track's first observations may leave columns of the factor empty: none
    of them may be lost.  Every step that its prefix determines equals the
    dense least-squares solution of that prefix, every other is NaN."""
    _cuda()
    n, rows, F = _undetermined_starts()[name]
    P = _no_prior(n, rows, F, seed=n)
    D = native.DeviceProblem(P, covariance=cov)
    assert D.filter(covariance=cov, check=False) == native.KALMAN_GPU_ESINGULAR
    X, S = D.results()
    seen = 0
    for s in range(P.nsteps):
        Q = P.step_range(0, s + 1)
        enough = P.obs_rows[:s + 1].sum() >= n
        if not enough or np.linalg.matrix_rank(oracle.dense_system(Q, 0)[0]) < (s + 1) * n:
            assert np.isnan(X[s]).all() and (not cov or np.isnan(S[s]).all()), f"step {s}"
            continue
        seen += 1
        Xd, Sd = oracle.dense_smooth(Q)
        assert oracle.rel_err_states(X[s:s + 1], Xd[-1:]) < TOL, f"step {s}"
        if cov:
            assert oracle.rel_err_covs(S[s:s + 1], Sd[-1:]) < TOL, f"step {s}"
    assert seen > 0


def _kalman(F, K, G, C, x, Pm, c, o):
    """The covariance form of the filter in extended precision, K and C
    diagonal: estimates and covariances after every step but the first."""
    t = np.longdouble
    F, G, x, Pm, c, o = (np.asarray(a).astype(t) for a in (F, G, x, Pm, c, o))
    X, S = [], []
    for s in range(len(o)):
        x = F @ x + c[s]
        Pm = F @ Pm @ F.T + np.diag(np.asarray(K).astype(t))
        for r in range(len(G)):  # one observation at a time
            h = Pm @ G[r]
            g = h / (G[r] @ h + t(C[r]))
            x = x + g * (o[s, r] - G[r] @ x)
            Pm = Pm - np.outer(g, h)
        X.append(x.astype(float))
        S.append(Pm.astype(float))
    return np.array(X), np.array(S)


@pytest.mark.parametrize("n", [2, 4, 6, 8])
@pytest.mark.parametrize("k,c", [(1e-14, 0.1), (1e-10, 1e4), (1.0, 0.1)])
def test_small_process_noise(n, k, c):
    """The weighed evolution's rows are up to 1e9 times as large as the factor's:
    the information on the next state must not come from their differences."""
    _cuda()
    F, p = _pv(n, "pv")
    rng = np.random.default_rng(n)
    G = np.eye(n)[p]
    N, m = 60, len(p)
    P = pb.empty_problem(n, n, [N])
    P.H[:], P.F[:], P.K[:] = np.eye(n), F.T, k * np.eye(n)
    P.c[:] = 0.1 * rng.standard_normal((N, n))
    P.G[:, :, :m], P.C[:, :m, :m] = G.T, c * np.eye(m)
    P.o[:, :m] = rng.standard_normal((N, m))
    P.obs_rows[:] = m
    P.G[0], P.C[0], P.o[0], P.obs_rows[0] = np.eye(n), np.eye(n), rng.standard_normal(n), n
    X, S = _kalman(F, [k] * n, G, [c] * m, P.o[0], np.eye(n), P.c[1:], P.o[1:, :m])
    D = native.DeviceProblem(P, covariance=True)
    D.filter()
    Xg, Sg = D.results()
    assert oracle.rel_err_states(Xg[1:], X) < TOL
    assert oracle.rel_err_covs(Sg[1:], S) < TOL


def test_many_uneven_tracks_in_bounded_memory():
    """Up to 8 states the workspace is a round's (128 MiB) and the tracks' tables,
    whatever their number; every track is a prefix of one and gives its bits."""
    _cuda()
    P = pb.random_dynamics([900], 8, 4, seed=3, missing=0.2)
    D = native.DeviceProblem(P, covariance=True)
    D.filter()
    X, S = D.results()
    rng = np.random.default_rng(0)
    for lens in (np.r_[rng.integers(0, 4, 100000), 900, 1, 700], np.r_[rng.integers(1, 40, 4000), np.full(5, 900)],
                 np.full(260, 900)):
        ts = np.zeros(len(lens) + 1, dtype=np.int64)
        ts[1:] = np.cumsum(lens)
        idx = np.arange(ts[-1]) - np.repeat(ts[:-1], lens)
        B = pb.PackedProblem(8, 8, ts, *[np.ascontiguousarray(getattr(P, f)[idx]) for f in (
            "H", "F", "c", "K", "K_type", "G", "o", "C", "C_type", "obs_rows")])
        for cov in (True, False):
            native.release()
            D = native.DeviceProblem(B, covariance=cov)
            D.filter(covariance=cov)
            assert native.workspace_held() <= (130 << 20) + 24 * len(lens)
            Xb, Sb = D.results()
            np.testing.assert_array_equal(Xb, X[idx])
            if cov:
                np.testing.assert_array_equal(Sb, S[idx])
