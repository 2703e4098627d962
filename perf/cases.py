"""The smoothing work this framework is measured on: one case per way a program uses it,
from a sliding window of a few dozen steps to thousands of long tracks, in every arithmetic
form and through every kind of entry point (direct calls on device arrays, replayed plans,
host arrays, the filter).

Inputs are made on the GPU from a seed: constant-velocity tracks (the batched workload of
bench.py) for even n with m = n/2 observed positions, and damped rotations F = rho Q with
random covariances (the larger-state workloads of ultimate_kalman_gb300/shapes.py) for the
other shapes.  Every step carries its own copy of its matrices, as callers store them.
"""
import math

import numpy as np
import torch

from ultimate_kalman_gb300 import native

DEFAULTS = {"algorithm": "oddeven", "entry": "call", "form": "f64", "cov": True, "sweeps": 0, "model": "cv",
            "tracks": 1, "lengths": 0, "missing": 0.0, "type": "C"}


def _case(name=None, **kw):
    c = dict(DEFAULTS, **kw)
    if name is not None:
        c["name"] = name
    return c


def listed():
    return [
        # a tracker that re-smooths a short sliding window of 2-D positions at every frame: latency
        _case("window_n4", n=4, m=2, lo=64, hi=64),
        # the same for 3-D positions over a longer window, replayed from a prepared plan
        _case("window_n6_plan", n=6, m=3, lo=1000, hi=1000, entry="plan_status", form="f32", cov=False),
        # one long recorded track, states and covariances, plain FP64 (bench.py's single track)
        _case("track_n6", n=6, m=3, lo=100000, hi=100000),
        # one recorded track through the associative-scan smoother
        _case("track_n6_associative", n=6, m=3, lo=20000, hi=20000, algorithm="associative"),
        # bench.py's headline: thousands of uneven tracks, precision form, one sweep, a replayed plan
        _case("batch_n6_precision", n=6, m=3, tracks=4096, lo=100, hi=20000, entry="plan", form="f32", cov=False,
              sweeps=1),
        # the same kind of batch with covariances, plain FP64
        _case("batch_n6_f64", n=6, m=3, tracks=1024, lo=100, hi=20000),
        # and in double-float arithmetic (the precision form with covariances)
        _case("batch_n6_df", n=6, m=3, tracks=1024, lo=100, hi=20000, form="f32"),
        # a served batch of one shape class: a few tracks of 12 states, some steps unobserved
        _case("batch_n12_f64", n=12, m=6, tracks=16, lo=64, hi=4000, model="rotation", missing=0.05),
        # 48 states through the associative smoother, 5 % of the steps unobserved
        _case("track_n48_associative", n=48, m=24, lo=5000, hi=5000, algorithm="associative", model="rotation",
              missing=0.05),
        # 128 states, 64 observations, ill-conditioned covariances, precision form
        _case("track_n128_precision", n=128, m=64, lo=5000, hi=5000, model="rotation_log", form="f32", cov=False,
              sweeps=1),
        # tracks that live in page-locked host memory: copies in and out are part of the call
        _case("host_n6_precision", n=6, m=3, tracks=256, lo=100, hi=2000, entry="host", form="f32", cov=False,
              sweeps=1),
        # filtered estimates of many tracks at once
        _case("filter_n6", n=6, m=3, tracks=512, lo=50, hi=500, algorithm="filter"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    seed = rng.randrange(1 << 30)
    missing = rng.choice([0.0, 0.0, 0.05, 0.2])
    kind = rng.choice(["window", "window", "track", "batch", "batch", "mid", "mid", "large", "associative", "host",
                       "filter"])
    form, cov = rng.choice([("f64", True), ("f64", False), ("f32", False), ("f32", True)])
    if kind == "window":  # one short track
        n = rng.choice([2, 3, 4, 5, 6, 6, 7, 8])
        return _case(n=n, m=rng.randint(1, n), lo=(k := _log_int(rng, 16, 3000)), hi=k, form=form, cov=cov,
                     entry=rng.choice(["call", "call", "plan_status"]), model="rotation", missing=missing,
                     type=rng.choice("CCWF"))
    if kind == "track":  # one long track
        n = rng.choice([4, 6, 6])
        return _case(n=n, m=n // 2, lo=(k := _log_int(rng, 3000, 200000)), hi=k, form=form, cov=cov, missing=missing)
    if kind == "batch":  # many uneven tracks
        n = rng.choice([4, 6, 6, 8])
        return _case(n=n, m=n // 2, tracks=_log_int(rng, 32, 1500), lo=rng.randint(50, 200),
                     hi=_log_int(rng, 300, 8000), lengths=seed, form=form, cov=cov, sweeps=rng.choice([0, 1]),
                     entry=rng.choice(["call", "plan"]), missing=missing, type=rng.choice("CCw"))
    if kind == "mid":  # 9 to 31 states
        n = rng.choice([9, 12, 12, 15, 18, 24, 24, 31])
        tracks = _log_int(rng, 1, 16)
        return _case(n=n, m=rng.choice([n // 2, n // 3, n]), tracks=tracks, lo=64,
                     hi=max(65, _log_int(rng, 500, 40000 // tracks)), lengths=seed, form=form, cov=cov,
                     model="rotation", missing=missing, type=rng.choice("CCWF"))
    if kind == "large":  # 32 to 128 states
        n = rng.choice([32, 48, 48, 65, 96, 128])
        k = _log_int(rng, 200, max(400, int(5000 * (64 / n) ** 2)))
        return _case(n=n, m=rng.choice([n // 2, n // 2, n // 4]), lo=k, hi=k, form=form, cov=cov,
                     algorithm="associative" if form == "f64" and cov and n <= 65 else "oddeven", model="rotation",
                     missing=missing)
    if kind == "associative":
        n = rng.choice([3, 4, 6, 6, 8, 12, 20])
        k = _log_int(rng, 100, 30000 if n <= 8 else 6000)
        return _case(n=n, m=max(1, n // 2), lo=k, hi=k, algorithm="associative", model="rotation", missing=missing)
    if kind == "host":
        return _case(n=6, m=3, tracks=_log_int(rng, 8, 500), lo=100, hi=2000, lengths=seed, entry="host", form=form,
                     cov=cov, missing=missing)
    n = rng.choice([3, 4, 6, 6, 8, 12])
    return _case(n=n, m=max(1, n // 2), tracks=_log_int(rng, 1, 1000), lo=20, hi=_log_int(rng, 40, 400), lengths=seed,
                 algorithm="filter", model="rotation", missing=missing)


def _lengths(case):
    if case["lo"] == case["hi"]:
        return np.full(case["tracks"], case["lo"], dtype=np.int64)
    rng = np.random.default_rng(case["lengths"])
    return np.floor(np.exp(rng.uniform(np.log(case["lo"]), np.log(case["hi"]), case["tracks"]))).astype(np.int64)


def _orthogonal(rng, T, n):
    Q, R = np.linalg.qr(rng.standard_normal((T, n, n)))
    return Q * np.sign(np.diagonal(R, axis1=1, axis2=2))[:, None, :]


def _model(case, seed):
    """Per-track matrices, [T, rows, cols]: F, G, K, C (explicit covariances)."""
    n, m, T = case["n"], case["m"], case["tracks"]
    rng = np.random.default_rng(seed)
    if case["model"] == "cv":
        h = n // 2
        F = np.tile(np.eye(n), (T, 1, 1))
        F[:, :h, h:] += 0.1 * np.eye(h)
        G = np.tile(np.eye(m, n), (T, 1, 1))
        K = 1e-2 * rng.uniform(0.5, 2.0, (T, 1, 1)) * np.eye(n)
        C = 1e-1 * rng.uniform(0.5, 2.0, (T, 1, 1)) * np.eye(m)
        return F, G, K, C
    if case["model"] == "rotation_log":
        eig = lambda d: np.exp(rng.uniform(np.log(1e-3), 0.0, (T, d)))  # noqa: E731
    else:
        eig = lambda d: rng.uniform(0.1, 1.0, (T, d))  # noqa: E731
    U, V = _orthogonal(rng, T, n), _orthogonal(rng, T, m)
    K = np.einsum("tij,tj,tkj->tik", U, eig(n), U)
    C = np.einsum("tij,tj,tkj->tik", V, eig(m), V)
    F = (0.995 if n >= 128 else 0.99) * _orthogonal(rng, T, n)
    G = rng.standard_normal((T, m, n)) / math.sqrt(m)
    if case["type"] == "w":  # standard deviations: diagonal covariances
        K, C = K * np.eye(n), C * np.eye(m)
    return F, G, 0.5 * (K + K.transpose(0, 2, 1)), 0.5 * (C + C.transpose(0, 2, 1))


def _factor(cov, kind):
    """The stored form of a covariance: 'C' itself, 'F' its Cholesky factor, 'W' the factor's
    inverse, 'w' reciprocal standard deviations in its first column."""
    if kind == "C":
        return cov
    if kind == "w":
        out = np.zeros_like(cov)
        out[:, :, 0] = 1.0 / np.sqrt(np.diagonal(cov, axis1=1, axis2=2))
        return out
    L = np.linalg.cholesky(cov)
    return L if kind == "F" else np.linalg.inv(L)


def _vectors(case, seed):
    """Observations o [N, m], inputs c [N, n], prior means x0 [T, n], observed [N], track of each step, starts."""
    L = _lengths(case)
    start = np.zeros(len(L) + 1, dtype=np.int64)
    start[1:] = np.cumsum(L)
    N, T, n, m = int(start[-1]), len(L), case["n"], case["m"]
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    f64 = dict(dtype=torch.float64, device="cuda", generator=g)
    first = torch.as_tensor(start[:-1], device="cuda")
    tid = torch.repeat_interleave(torch.arange(T, device="cuda"), torch.as_tensor(L, device="cuda"))
    x0 = torch.randn((T, n), **f64)
    c = 0.01 * torch.randn((N, n), **f64)
    o = torch.randn((N, m), **f64)
    if case["model"] == "cv" and m == n // 2:  # positions of a random walk in velocity, with measurement noise
        h = n // 2
        v = torch.cumsum(0.1 * torch.randn((N, h), **f64), 0)
        v = v - v[first][tid] + x0[:, h:][tid]
        p = torch.cumsum(0.1 * v, 0)
        o = 0.3 * o + (p - p[first][tid] + x0[:, :h][tid])
    seen = torch.rand((N,), **f64) >= case["missing"]
    return o, c, x0, seen, tid, start


def _packed(case, seed):
    """The packed arrays of kalman_gpu_problem_t on the GPU (every block transposed: column-major)."""
    n, m, kind = case["n"], case["m"], case["type"]
    mx = max(n, m)
    F, G, K, C = _model(case, seed)
    dev = lambda a: torch.as_tensor(np.ascontiguousarray(a), device="cuda")  # noqa: E731
    o, c, x0, seen, tid, start = _vectors(case, seed)
    N, first = len(tid), torch.as_tensor(start[:-1], device="cuda")

    def pad(a, rows, cols):  # [T, r, c] -> transposed blocks of cols x rows entries
        out = np.zeros((a.shape[0], cols, rows))
        out[:, :a.shape[2], :a.shape[1]] = a.transpose(0, 2, 1)
        return dev(out)

    A = {"H": torch.eye(n, dtype=torch.float64, device="cuda").expand(N, n, n).contiguous(),
         "F": pad(F, n, n)[tid], "c": c, "K": pad(_factor(K, kind), n, n)[tid],
         "K_type": torch.full((N,), ord(kind), dtype=torch.uint8, device="cuda"),
         "G": pad(G, mx, n)[tid], "o": torch.zeros((N, mx), dtype=torch.float64, device="cuda"),
         "C": pad(_factor(C, kind), mx, mx)[tid],
         "C_type": torch.full((N,), ord(kind), dtype=torch.uint8, device="cuda"),
         "obs_rows": torch.where(seen, m, 0).to(torch.int32)}
    A["o"][:, :m] = o
    # the first step observes the whole state: the prior N(x0, I)
    eye = torch.zeros((n, mx), dtype=torch.float64, device="cuda")
    eye[:, :n] = torch.eye(n, dtype=torch.float64, device="cuda")
    A["G"][first] = eye
    square = torch.zeros((mx, mx), dtype=torch.float64, device="cuda")
    square[:n, :n] = torch.eye(n, dtype=torch.float64, device="cuda")
    A["C"][first] = square
    A["C_type"][first] = ord("C")
    A["obs_rows"][first] = n
    A["o"][first] = 0.0
    A["o"][first, :n] = x0
    return A, start


class _Shape:
    """What native.host_struct_from_tensors reads of a problem."""

    def __init__(self, n, mmax, start):
        self.n, self.mmax, self.track_start = n, mmax, start
        self.ntracks, self.nsteps = len(start) - 1, int(start[-1])


def prepare(case, seed):
    A, start = _packed(case, seed)
    n, mx = case["n"], max(case["n"], case["m"])
    kw = dict(covariance=case["cov"], fp32_refine=case["form"] == "f32", sweeps=case["sweeps"])
    s = {"case": case, "kw": kw}
    if case["entry"] == "host":
        s["arrays"] = {k: torch.empty(v.shape, dtype=v.dtype, pin_memory=True).copy_(v) for k, v in A.items()}
        N = int(start[-1])
        s["state"] = torch.empty((N, n), dtype=torch.float64, pin_memory=True)
        s["cov"] = torch.empty((N, n, n), dtype=torch.float64, pin_memory=True) if case["cov"] else None
        s["struct"] = native.host_struct_from_tensors(_Shape(n, mx, start), s["arrays"], s["state"], s["cov"])
        return s
    s["problem"] = D = native.DeviceProblem.from_arrays(n, mx, start, A, case["cov"])
    if case["entry"].startswith("plan"):
        s["plan"] = D.plan(**kw)
    return s


def run(s):
    case = s["case"]
    if case["entry"] == "host":
        native.smooth_struct(case["algorithm"], s["struct"], **s["kw"])
        return {"state": s["state"], "cov": s["cov"]}
    D = s["problem"]
    if case["entry"] == "plan":
        s["plan"].execute()
    elif case["entry"] == "plan_status":  # a frame loop looks at the status before it uses the estimates
        s["plan"].execute()
        s["plan"].status()
    elif case["algorithm"] == "filter":
        D.filter(case["cov"])
    else:
        D.smooth(case["algorithm"], **s["kw"])
    return {"state": D.state, "cov": D.cov}


def work(case):
    """Bytes: every step's equations at their real sizes once in, the results once out.  Flops: the Householder
    smoother's QR reductions, back-substitution and covariance recurrence (multiply-add = 2)."""
    n, m, N = case["n"], case["m"], float(_lengths(case).sum())
    out = n + (n * n if case["cov"] else 0)
    data = N * 8 * (3 * n * n + n + m * n + m + m * m + out)
    if case["algorithm"] == "associative":  # elements, two combines per element of either scan
        per = 70 * n ** 3
    elif case["algorithm"] == "filter":
        per = 16 * n ** 3
    else:
        per = (48 if case["cov"] else 33) * n ** 3
    return {"bytes": data, "flops": N * per}


# ---------------------------------------------------------------------------
# the same estimates in plain 64-bit torch
# ---------------------------------------------------------------------------

def _solve(A, B):
    """A^{-1} B for batches of small matrices, in pieces the batched LU takes."""
    if len(A) <= 65536:
        return torch.linalg.solve(A, B)
    return torch.cat([torch.linalg.solve(a, b) for a, b in zip(A.split(65536), B.split(65536))])


def _chain(D, Lw, r, want_cov):
    """x (and the diagonal blocks of the inverse, and its blocks (i, i-1)) of the symmetric block-tridiagonal system
    with diagonal D [N,n,n], lower blocks Lw (Lw[i] couples i to i-1; Lw[0] = 0) and right-hand side r, by cyclic
    reduction: the even unknowns are eliminated, the odd ones form the same kind of system of half the size."""
    N, n = r.shape
    if N == 1:
        X = _solve(D, torch.cat([r[:, :, None], torch.eye(n, dtype=r.dtype, device=r.device)[None]], 2))
        return X[:, :, 0], X[:, :, 1:], torch.zeros_like(D)
    De, Dodd = D[0::2], D[1::2]
    no = len(Dodd)
    up = Lw[1::2].transpose(1, 2)  # couples an even unknown to the odd one after it
    up = up if len(De) == no else torch.cat([up, torch.zeros_like(D[:1])])
    # D_e^{-1} [L_e | U_e | r_e]
    S = _solve(De, torch.cat([Lw[0::2], up, r[0::2, :, None]], 2))
    SL, SU, sr = S[:, :, :n], S[:, :, n:2 * n], S[:, :, 2 * n]
    has = len(De) > no  # an even unknown after the last odd one
    Dn = Dodd - Lw[1::2] @ SU[:no]
    rn = r[1::2] - (Lw[1::2] @ sr[:no, :, None])[:, :, 0]
    nxt = no if has else no - 1  # odd unknowns with an even one behind them
    Ut = Lw[0::2][1:1 + nxt].transpose(1, 2)
    Dn[:nxt] -= Ut @ SL[1:1 + nxt]
    rn[:nxt] -= (Ut @ sr[1:1 + nxt, :, None])[:, :, 0]
    Ln = -(Lw[1::2] @ SL[:no])
    Ln[0] = 0.0
    xo, So, Co = _chain(Dn, Ln, rn, want_cov)
    zero = torch.zeros_like(xo[:1])
    xm = torch.cat([zero, xo])[:len(De)]
    xp = xo if not has else torch.cat([xo, zero])
    x = torch.empty_like(r)
    x[1::2] = xo
    x[0::2] = sr - (SL @ xm[:, :, None] + SU @ xp[:, :, None])[:, :, 0]
    if not want_cov:
        return x, So, Co
    Z = torch.zeros_like(So[:1])
    Smm = torch.cat([Z, So])[:len(De)]
    Spp = So if not has else torch.cat([So, Z])
    Spm = Co if not has else torch.cat([Co, Z])  # cov(x_{j+1}, x_{j-1}); zero where one of them is missing
    Em = -(SL @ Smm + SU @ Spm)                  # cov(x_j, x_{j-1})
    Ep = -(SL @ Spm.transpose(1, 2) + SU @ Spp)  # cov(x_j, x_{j+1})
    Sig, Cr = torch.empty_like(D), torch.empty_like(D)
    Sig[1::2] = So
    Inv = _solve(De, torch.eye(n, dtype=D.dtype, device=D.device).expand(len(De), n, n))
    Sig[0::2] = Inv - Em @ SL.transpose(1, 2) - Ep @ SU.transpose(1, 2)
    Cr[0::2] = Em
    Cr[1::2] = Ep[:no].transpose(1, 2)
    return x, Sig, Cr


def _exact_smooth(case, seed):
    F, G, K, C = (torch.as_tensor(a, device="cuda") for a in _model(case, seed))
    o, c, x0, seen, tid, start = _vectors(case, seed)
    N, n = len(tid), case["n"]
    first = torch.as_tensor(start[:-1], device="cuda")
    inner = torch.ones(N, dtype=torch.bool, device="cuda")
    inner[first] = False
    seen = seen & inner
    Ki, Ci = torch.linalg.inv(K), torch.linalg.inv(C)
    GtC = G.transpose(1, 2) @ Ci
    # per step: the evolution into it, the observation of it, the evolution out of it
    D = torch.zeros((N, n, n), dtype=torch.float64, device="cuda")
    D += torch.where(inner[:, None, None], Ki[tid], torch.eye(n, dtype=torch.float64, device="cuda"))
    D += seen[:, None, None] * (GtC @ G)[tid]
    out = torch.zeros(N, dtype=torch.bool, device="cuda")
    out[:-1] = inner[1:]
    D += out[:, None, None] * (F.transpose(1, 2) @ Ki @ F)[tid]
    Lw = -(inner[:, None, None] * (Ki @ F)[tid])
    r = seen[:, None] * (GtC[tid] @ o[:, :, None])[:, :, 0]
    r[first] += x0
    Kc = inner[:, None] * (Ki[tid] @ c[:, :, None])[:, :, 0]
    r += Kc
    r[:-1] -= (F.transpose(1, 2)[tid[1:]] @ Kc[1:, :, None])[:, :, 0]
    x, S, _ = _chain(D, Lw, r, case["cov"])
    return {"state": x, "cov": S if case["cov"] else None}


def _exact_filter(case, seed):
    F, G, K, C = (torch.as_tensor(a, device="cuda") for a in _model(case, seed))
    o, c, x0, seen, _, start = _vectors(case, seed)
    n = case["n"]
    lengths = np.diff(start)
    eye = torch.eye(n, dtype=torch.float64, device="cuda")
    X = torch.empty((int(start[-1]), n), dtype=torch.float64, device="cuda")
    S = torch.empty((int(start[-1]), n, n), dtype=torch.float64, device="cuda")
    x, P = x0.clone(), eye.repeat(case["tracks"], 1, 1)
    for i in range(int(lengths.max())):
        on = torch.as_tensor(np.nonzero(lengths > i)[0], device="cuda")
        at = torch.as_tensor(start[:-1], device="cuda")[on] + i
        xi, Pi = x[on], P[on]
        if i > 0:
            xi = (F[on] @ xi[:, :, None])[:, :, 0] + c[at]
            Pi = F[on] @ Pi @ F[on].transpose(1, 2) + K[on]
            W = torch.linalg.solve(G[on] @ Pi @ G[on].transpose(1, 2) + C[on], G[on] @ Pi).transpose(1, 2)
            W = W * seen[at][:, None, None]
            xi = xi + (W @ (o[at] - (G[on] @ xi[:, :, None])[:, :, 0])[:, :, None])[:, :, 0]
            J = eye - W @ G[on]
            Pi = J @ Pi @ J.transpose(1, 2) + W @ C[on] @ W.transpose(1, 2)
        x[on], P[on] = xi, Pi
        X[at], S[at] = xi, Pi
    return {"state": X, "cov": S if case["cov"] else None}


def exact(case, seed):
    return _exact_filter(case, seed) if case["algorithm"] == "filter" else _exact_smooth(case, seed)
