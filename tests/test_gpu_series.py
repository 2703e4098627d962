"""The FP64 reciprocal, reciprocal root and reflector of csrc/lanes.cuh -- a
series step on an FP32 seed between 2^-100 and 2^100, CUDA's division and root
outside -- against the same in extended precision, and whole problems whose
scale lies on either side of the hand-over.

Bounds: a seed is right to 2^-21, a series' next term is 2^-63.  The reciprocal
is one rounding (0.5 ulp); the residual of the root's step has the rounding of
s y (2^-53), half of which is left, so 2^-54 + 2^-53 relative, 1 ulp; s times it
2.5 2^-53, 2.5 ulp."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import oracle
from ultimate_kalman_gb300 import build, native, problem as pb

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "lanes.cuh"
__global__ void run(const double* s, double* out, long long n)
{
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  out[i] = lanes::recip(s[i]);
  out[n + i] = lanes::inv_root(fabs(s[i]));
  const double a = s[i], t = s[(i + 1) % n] * s[(i + 1) % n];
  const lanes::Refl<double> r = lanes::reflector(a, t);
  out[2 * n + i] = r.beta;
  out[3 * n + i] = r.inv * fma(r.amb, a, t); /* u^T (a, x) / (u^T u / 2) = 1 */
}
extern "C" int run_series(const double* s, double* out, long long n)
{
  run<<<(unsigned)((n + 255) / 256), 256>>>(s, out, n);
  return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def series(tmp_path_factory):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    d = tmp_path_factory.mktemp("series")
    src, lib = str(d / "series.cu"), str(d / "series.so")
    with open(src, "w") as f:
        f.write(SOURCE)
    subprocess.run([build.nvcc(), *build.ARCH, "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "-I", build.CSRC,
                    src, "-o", lib], check=True)
    f = ctypes.CDLL(lib).run_series
    f.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_longlong]

    def run(s):
        x = torch.as_tensor(s, device="cuda")
        out = torch.empty(4 * len(s), dtype=torch.float64, device="cuda")
        assert f(x.data_ptr(), out.data_ptr(), len(s)) == 0
        return out.cpu().numpy().reshape(4, -1)
    return run


def _ulps(x, ref):
    """|x - ref| in units of ref's last place; ref in extended precision"""
    return np.abs(x.astype(np.longdouble) - ref) / np.spacing(np.abs(ref).astype(np.float64))


@pytest.mark.parametrize("lo,hi", [(-110, -90), (-100.001, -99.999), (-1, 1), (99.999, 100.001), (90, 110), (-110, 110)])
def test_series(series, lo, hi):
    rng = np.random.default_rng(0)
    s = np.exp2(rng.uniform(lo, hi, 200000)) * rng.choice([-1.0, 1.0], 200000)
    s[:64] = np.exp2(np.round(rng.uniform(lo, hi, 64)))  # powers of two, the hand-over itself
    rcp, root, beta, one = series(s)
    x = s.astype(np.longdouble)
    assert _ulps(rcp, 1 / x).max() < 0.51
    assert _ulps(root, 1 / np.sqrt(np.abs(x))).max() < 1.01
    t = np.roll(s, -1) ** 2
    nb = np.sqrt(x * x + t.astype(np.longdouble))
    assert (np.signbit(beta) != np.signbit(s)).all()
    assert _ulps(np.abs(beta), nb).max() < 3.1  # 0.5 of the sum's rounding, halved by the root, more
    assert np.abs(one - 1).max() < 16 * 2.0**-52


@pytest.mark.parametrize("n,m", [(4, 2), (6, 6), (12, 6), (40, 12)])
@pytest.mark.parametrize("e", [-240, -204, -200, -196, 196, 200, 204, 240])
def test_problems_on_both_sides_of_the_series_range(n, m, e):
    """Covariances times 2^e: the weights' squares cross 2^-100 and 2^100, the
    states stay and the covariances scale."""
    P = pb.random_dynamics([9, 2, 1], n, m, seed=n, per_step=True, missing=0.2)
    st, Xo, So = oracle.smooth(P, "oddeven")
    assert st == 0
    first = np.zeros(P.nsteps, dtype=bool)
    first[P.track_start[:-1]] = True
    P.K[:] *= 2.0**e
    P.C[~first] *= 2.0**e
    P.C[first] *= 2.0**(-e // 2)  # 'W'
    for alg in ("oddeven", "associative"):
        X, S = native.smooth(P, alg)
        assert oracle.rel_err_states(X, Xo) < 1e-11
        assert oracle.rel_err_covs(S * 2.0**-e, So) < 1e-11
    D = native.DeviceProblem(P, covariance=True)
    D.filter()
    X, S = D.results()
    ends = P.track_start[1:] - 1
    assert oracle.rel_err_states(X[ends], Xo[ends]) < 1e-11
    assert oracle.rel_err_covs(S[ends] * 2.0**-e, So[ends]) < 1e-11
