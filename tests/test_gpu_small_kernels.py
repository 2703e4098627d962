"""The FP64 and double-float kernels for up to 8 states take 32 lanes, eight
lanes or one thread per work item, by the number of items of a level: the
same track smoothed alone and in batches that cross those limits must give
the same bits, and the oracle's estimates (1e-11 in FP64, 1e-9 in
double-float: the bars of those forms)."""
import numpy as np
import pytest

import oracle
from ultimate_kalman_gb300 import native, problem as pb

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    native.load()


# 37 steps: 18 pairs at level 0 and an odd length at levels 0, 2 and the base;
# 40 tracks: 720 pairs (32 lanes), 100: 1,800 and 160: 2,880 (eight lanes in
# FP64 and in double-float), 420: 7,560 (threads)
@pytest.mark.parametrize("n,m,cov,missing", [(2, 2, "C", 0.0), (3, 1, "W", 0.3), (4, 2, "C", 0.1), (6, 3, "F", 0.0),
                                             (6, 6, "C", 0.3), (7, 4, "w", 0.1), (8, 8, "C", 0.0), (8, 3, "C", 0.2)])
@pytest.mark.parametrize("df", [False, True], ids=["f64", "double-float"])
def test_same_bits_alone_and_batched(n, m, cov, missing, df):
    P = pb.random_dynamics([37], n, m, seed=10 * n + m, K_type=cov, C_type=cov, missing=missing, per_step=True)
    X, S = native.smooth(P, "oddeven", fp32_refine=df)
    st, Xo, So = oracle.smooth(P, "oddeven")
    assert st == 0
    tol = 1e-9 if df else 1e-11
    assert oracle.rel_err_states(X, Xo) < tol
    assert oracle.rel_err_covs(S, So) < tol
    if not df:
        Xs, _ = native.smooth(P, "oddeven", covariance=False)
        np.testing.assert_array_equal(Xs, X)
    for T in (40, 100, 160, 420):
        B = P.select_tracks([0] * T)
        Xb, Sb = native.smooth(B, "oddeven", fp32_refine=df)
        for t in (0, T - 1):
            np.testing.assert_array_equal(Xb[37 * t:37 * t + 37], X, err_msg=f"{T} tracks")
            np.testing.assert_array_equal(Sb[37 * t:37 * t + 37], S, err_msg=f"{T} tracks")


@pytest.mark.parametrize("k", [1, 2, 3, 5, 8, 31])
def test_unobservable_is_reported(k):
    """One observation row in total: every form reports the zero pivot."""
    P = pb.random_dynamics([k], 6, 1, seed=k, missing=0.0, fold=False)
    P.obs_rows[1:] = 0
    for df in (False, True):
        with pytest.raises(native.KalmanError) as e:
            native.smooth(P, "oddeven", fp32_refine=df)
        assert e.value.status == native.KALMAN_GPU_ESINGULAR


@pytest.mark.parametrize("n,k", [(2, 1023), (3, 1), (4, 1025), (6, 2047), (6, 2), (7, 1024), (8, 2500)])
@pytest.mark.parametrize("sweeps", [1, 2])
def test_upper_levels_in_one_launch(n, k, sweeps):
    """The precision form takes the levels of at most 1,024 steps a track in
    one launch for up to 304 tracks, and level by level above: the same bits."""
    P = pb.random_dynamics([k], n, n, seed=n + k, K_type="C", C_type="C")
    st, Xo, _ = oracle.smooth(P, "oddeven")
    assert st == 0
    X, _ = native.smooth(P, "oddeven", covariance=False, fp32_refine=True, sweeps=sweeps)
    if sweeps == 2:
        assert oracle.rel_err_states(X, Xo) < 1e-9
    for T in (304, 305):
        Xb, _ = native.smooth(P.select_tracks([0] * T), "oddeven", covariance=False, fp32_refine=True, sweeps=sweeps)
        for t in (0, T - 1):
            np.testing.assert_array_equal(Xb[k * t:k * t + k], X, err_msg=f"{T} tracks")


@pytest.mark.parametrize("n,m,cov,missing", [(2, 2, "C", 0.0), (3, 1, "W", 0.3), (4, 2, "C", 0.1), (5, 5, "w", 0.2),
                                             (6, 3, "F", 0.0), (6, 6, "C", 0.4), (8, 4, "C", 0.2)])
def test_many_tails_same_bits(n, m, cov, missing):
    """Tracks of odd length at a level: a warp each, up to 6 states a thread each
    past 4,864 of them (level 0: 7,500 here, level 1: 5,000), with the same bits
    in FP64, double-float and FP32."""
    P = pb.random_dynamics([1, 2, 3, 5], n, m, seed=20 * n + m, K_type=cov, C_type=cov, missing=missing, per_step=True)
    B = P.select_tracks([0, 1, 2, 3] * 2500)
    k = P.nsteps
    st, Xo, So = oracle.smooth(P, "oddeven")
    assert st == 0
    for kw, tol in ((dict(), 1e-11), (dict(fp32_refine=True), 1e-9), (dict(fp32_refine=True, covariance=False), 1e-9)):
        X, S = native.smooth(P, "oddeven", **kw)
        assert oracle.rel_err_states(X, Xo) < tol
        assert S is None or oracle.rel_err_covs(S, So) < tol
        Xb, Sb = native.smooth(B, "oddeven", **kw)
        for t in (0, 1249, 2499):
            np.testing.assert_array_equal(Xb[k * t:k * t + k], X)
            if S is not None:
                np.testing.assert_array_equal(Sb[k * t:k * t + k], S)


def test_many_unobservable_tails_are_reported():
    P = pb.random_dynamics([1, 3], 4, 1, seed=2, fold=False)
    P.obs_rows[1:] = 0
    B = P.select_tracks([0, 1] * 3000)
    for kw in (dict(), dict(fp32_refine=True)):
        with pytest.raises(native.KalmanError) as e:
            native.smooth(B, "oddeven", **kw)
        assert e.value.status == native.KALMAN_GPU_ESINGULAR
