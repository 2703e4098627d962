"""The thread-per-column kernels (9 to 64 states) at the edges of their register
sizes (12, 16, 24, 32, 48, 64 rows) and the precision form's kernels of four
columns by a quarter of the rows per thread (65 to 128 states; to 96 and to 128
rows) against the oracle: every covariance type, unobserved steps (the
trapezoids then run out of rows), odd and even lengths.  Bars as elsewhere: 1e-11 in FP64, 1e-9
in the precision form and in double-float."""
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


@pytest.mark.parametrize("n,m,cov", [(9, 4, "C"), (12, 12, "W"), (13, 1, "w"), (16, 7, "F"), (17, 17, "C"),
                                     (24, 11, "W"), (25, 12, "F"), (31, 30, "C"), (32, 9, "w"), (33, 16, "C"),
                                     (48, 47, "F"), (49, 20, "W"), (63, 5, "C"), (64, 32, "C"), (65, 31, "C"),
                                     (96, 40, "C"), (97, 33, "F")])
def test_register_sizes(n, m, cov):
    P = pb.random_dynamics([1, 2, 11, 14], n, m, seed=n + m, K_type=cov, C_type=cov, missing=0.3, per_step=True)
    st, Xo, So = oracle.smooth(P, "oddeven")
    assert st == 0
    X, S = native.smooth(P, "oddeven")
    assert oracle.rel_err_states(X, Xo) < 1e-11 and oracle.rel_err_covs(S, So) < 1e-11
    X, _ = native.smooth(P, "oddeven", covariance=False)
    assert oracle.rel_err_states(X, Xo) < 1e-11
    X, S = native.smooth(P, "oddeven", fp32_refine=True)
    assert oracle.rel_err_states(X, Xo) < 1e-9 and oracle.rel_err_covs(S, So) < 1e-9
    X, _ = native.smooth(P, "oddeven", covariance=False, fp32_refine=True, sweeps=3)
    assert oracle.rel_err_states(X, Xo) < 1e-9


@pytest.mark.parametrize("n", [12, 40])
def test_unobservable_is_reported(n):
    P = pb.random_dynamics([9], n, 2, seed=n, fold=False)
    P.obs_rows[1:] = 0
    for refine in (False, True):
        with pytest.raises(native.KalmanError) as e:
            native.smooth(P, "oddeven", fp32_refine=refine)
        assert e.value.status == native.KALMAN_GPU_ESINGULAR


@pytest.mark.parametrize("n,m,cov", [(9, 3, "W"), (12, 6, "C"), (15, 15, "w"), (16, 8, "F"), (24, 10, "C"),
                                     (31, 8, "U"), (33, 40, "C"), (48, 24, "W"), (50, 20, "C"), (64, 30, "F"),
                                     (65, 10, "C")])
def test_associative_register_sizes(n, m, cov):
    P = pb.random_dynamics([1, 2, 9, 14], n, m, seed=2 * n + m, K_type=cov, C_type=cov, missing=0.3, per_step=True)
    st, Xo, So = oracle.smooth(P, "oddeven")
    assert st == 0
    X, S = native.smooth(P, "associative")
    assert oracle.rel_err_states(X, Xo) < 1e-11 and oracle.rel_err_covs(S, So) < 1e-11


@pytest.mark.parametrize("n,m,cov", [(97, 97, "C"), (99, 1, "w"), (100, 40, "W"), (113, 112, "C"), (127, 20, "F"),
                                     (128, 128, "C"), (128, 64, "W"), (120, 128, "C")])
def test_two_pass_sizes(n, m, cov):
    """97 to 128 states in the precision form: 32 rows a lane, three passes a pair."""
    P = pb.random_dynamics([1, 2, 7, 12, 13], n, m, seed=n + m, K_type=cov, C_type=cov, missing=0.3, per_step=True)
    st, Xo, So = oracle.smooth(P, "oddeven")
    assert st == 0
    X, S = native.smooth(P, "oddeven", fp32_refine=True)
    assert oracle.rel_err_states(X, Xo) < 1e-9 and oracle.rel_err_covs(S, So) < 1e-9
    X, _ = native.smooth(P, "oddeven", covariance=False, fp32_refine=True, sweeps=3)
    assert oracle.rel_err_states(X, Xo) < 1e-9
    X, _ = native.smooth(P, "oddeven", covariance=False)
    assert oracle.rel_err_states(X, Xo) < 1e-11


@pytest.mark.parametrize("n,m", [(9, 3), (12, 5), (24, 8), (48, 24)])
def test_associative_variances_up_and_down(n, m):
    """Process noise whose variance goes from 1e-6 over 1 to 1e6 and back, in
    the associative smoother: a filtered variance is up to 1e6 times the
    smoothed one, so a covariance is right to about 1e6 n k eps (1e-7 at most
    here), unless an unsymmetric rounding error of the filtered one survives."""
    k = 10 if n < 24 else 7
    P = pb.random_dynamics([k], n, m, seed=n, per_step=True)
    P.K[1:] *= np.array([1.0, 1e6, 1e-6])[np.arange(1, k) % 3][:, None, None]
    st, Xo, So = oracle.smooth(P, "oddeven")
    assert st == 0
    X, S = native.smooth(P, "associative")
    assert oracle.rel_err_states(X, Xo) < 1e-7 and oracle.rel_err_covs(S, So) < 1e-7


@pytest.mark.parametrize("n,m,cov", [(34, 34, "C"), (37, 1, "W"), (40, 20, "C"), (41, 13, "F"), (45, 44, "w"), (50, 50, "C"),
                                     (51, 25, "W"), (56, 8, "F"), (57, 19, "C"), (61, 61, "w")])
def test_sizes_above_32(n, m, cov):
    """Above 32 states the block kernel weighs and the observations are
    triangularized after; FP64 and double-float have register sizes of 40 (pairs,
    even steps) and 56 (even steps to 50 states) besides 48 and 64."""
    P = pb.random_dynamics([1, 2, 11, 14], n, m, seed=3 * n + m, K_type=cov, C_type=cov, missing=0.3, per_step=True)
    st, Xo, So = oracle.smooth(P, "oddeven")
    assert st == 0
    X, S = native.smooth(P, "oddeven")
    assert oracle.rel_err_states(X, Xo) < 1e-11 and oracle.rel_err_covs(S, So) < 1e-11
    Xb, Sb = native.smooth(P.select_tracks([0, 1, 2, 3] * 60), "oddeven")
    np.testing.assert_array_equal(Xb[-P.nsteps:], X)
    np.testing.assert_array_equal(Sb[-P.nsteps:], S)
    X, S = native.smooth(P, "oddeven", fp32_refine=True)
    assert oracle.rel_err_states(X, Xo) < 1e-9 and oracle.rel_err_covs(S, So) < 1e-9
    X, _ = native.smooth(P, "oddeven", covariance=False, fp32_refine=True, sweeps=3)
    assert oracle.rel_err_states(X, Xo) < 1e-9


@pytest.mark.parametrize("n,m", [(66, 66), (67, 1), (68, 30), (80, 80), (93, 46), (95, 12)])
def test_wide_sizes_up_to_96(n, m):
    """The precision form of 65 to 96 states (24 rows a lane) between its ends."""
    P = pb.random_dynamics([1, 2, 7, 13], n, m, seed=n + m, missing=0.3, per_step=True)
    st, Xo, _ = oracle.smooth(P, "oddeven")
    assert st == 0
    X, _ = native.smooth(P, "oddeven", covariance=False, fp32_refine=True, sweeps=3)
    assert oracle.rel_err_states(X, Xo) < 1e-9
