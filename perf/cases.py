"""What a user of this framework has it do, as cases that can be timed and compared.

Kinds:
  loglik   one likelihood + score + Fisher evaluation of ordered data from host arrays
           (``vecchia_profile_loglik``), or of a kept ``DeviceProblem`` (``handle``: the objective
           call of a fit's iterations)
  batched  one round of many uneven problems through a captured ``BatchedLikelihood``
  order    ``maximin_order`` and ``find_ordered_nn`` of scaled inputs (a reorder)
  predict  ``ScaledVecchiaGP.predict`` of a fitted model (restored from its saved attributes)
  joint    ``ScaledVecchiaGP.sample_joint`` of such a model
  fit      a whole ``ScaledVecchiaGP.fit``
"""
import math

import numpy as np
import torch

from pyscaledvecchia_gb300 import (ScaledVecchiaGP, find_ordered_nn, maximin_order,
                                   vecchia_profile_loglik)
from pyscaledvecchia_gb300.batched import BatchedLikelihood, BatchProblem
from pyscaledvecchia_gb300.likelihood import DeviceProblem
from pyscaledvecchia_gb300.ordering import _nn_groups

TRENDS = ("zero", "constant", "linear")
NU_H = 1e-3  # step of the central difference an estimated nu's score is defined by


def listed():
    return [
        # a fit's objective on a small data set with few neighbours: latency and launches
        dict(name="loglik_n500_m10", kind="loglik", n=500, d=4, m=10, nu=2.5, est=False,
             trend="constant", precision="float64", handle=True),
        # the default estimation subset (n_est = 5000) at the default m
        dict(name="loglik_n5000_m30", kind="loglik", n=5000, d=8, m=30, nu=2.5, est=False,
             trend="constant", precision="float64", handle=True),
        # the method at scale, in both arithmetics, from the caller's host arrays
        dict(name="loglik_n200k", kind="loglik", n=200000, d=10, m=30, nu=2.5, est=False,
             trend="constant", precision="float64", handle=False),
        dict(name="loglik_n200k_split", kind="loglik", n=200000, d=10, m=30, nu=2.5, est=False,
             trend="constant", precision="split", handle=False),
        # an estimated smoothness with a linear trend, ragged sizes
        dict(name="loglik_nu_est_n10007", kind="loglik", n=10007, d=5, m=27, nu=1.3, est=True,
             trend="linear", precision="float64", handle=True),
        # one round of batched fits of uneven problems
        dict(name="batched_64", kind="batched", count=64, nmin=500, nmax=8000, precision="float64"),
        # a fit's reorder, and the ordering of a large data set
        dict(name="order_n5000", kind="order", n=5000, d=8, m=30),
        dict(name="order_n200k", kind="order", n=200000, d=10, m=30),
        # marginal prediction with the default m_pred, in both arithmetics
        dict(name="predict_n100k", kind="predict", n=100000, ns=20000, d=6, m=140,
             precision="float64"),
        dict(name="predict_split", kind="predict", n=30011, ns=9001, d=7, m=140,
             precision="split"),
        # joint sample paths
        dict(name="joint_100_paths", kind="joint", n=10000, ns=5000, d=6, m=140, sims=100,
             precision="float64"),
        # fit of a small emulator, start to end
        dict(name="fit_n2000", kind="fit", n=2000, d=8, m=30, precision="float64"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("loglik", "loglik", "loglik", "batched", "order", "predict", "joint"))
    d = rng.randint(3, 12)
    if kind == "loglik":
        nu, est = rng.choice(((2.5, False), (2.5, False), (1.5, False), (0.5, False),
                              (0.8, False), (1.3, True)))
        top = 200000 if nu in (0.5, 1.5, 2.5) else 20000
        return dict(kind=kind, n=_log_int(rng, 300, top), d=d, m=rng.randint(8, 31), nu=nu, est=est,
                    trend=rng.choice(TRENDS), precision=rng.choice(("float64", "split")),
                    handle=rng.random() < 0.5)
    if kind == "batched":
        return dict(kind=kind, count=_log_int(rng, 4, 64), nmin=500, nmax=_log_int(rng, 1000, 8000),
                    precision=rng.choice(("float64", "split")))
    if kind == "order":
        return dict(kind=kind, n=_log_int(rng, 500, 200000), d=rng.randint(3, 10), m=rng.randint(10, 31))
    d = rng.randint(3, 8)
    precision = rng.choice(("float64", "split"))
    if kind == "predict":
        return dict(kind=kind, n=_log_int(rng, 1000, 100000), ns=_log_int(rng, 100, 20000), d=d,
                    m=rng.randint(20, 140), precision=precision)
    return dict(kind=kind, n=_log_int(rng, 1000, 10000), ns=_log_int(rng, 200, 5000), d=d,
                m=rng.randint(20, 140), sims=rng.randint(20, 100), precision=precision)


# ------------------------------------------------------------------ inputs

def _field(X, lam, nu, rng, features=256):
    """An approximate draw of a unit-variance Matern field at the rows of X (random Fourier
    features: frequencies are a multivariate t with 2 nu degrees of freedom)."""
    g = rng.standard_normal((features, X.shape[1]))
    chi = rng.chisquare(2.0 * nu, features)
    W = torch.from_numpy(g * np.sqrt(2.0 * nu / chi)[:, None] / lam).cuda()
    b = torch.from_numpy(rng.uniform(0.0, 2.0 * math.pi, features)).cuda()
    f = torch.cos(torch.addmm(b, torch.from_numpy(X).cuda(), W.T)).sum(1)
    return (f * math.sqrt(2.0 / features)).cpu().numpy()


def _design(X, trend):
    if trend == "zero":
        return None
    one = np.ones((X.shape[0], 1))
    return one if trend == "constant" else np.hstack([one, X])


def _problem(rng, n, d, m, nu, est, trend, lam_hi):
    """Ordered data of one likelihood: ranges log-uniform in [0.05, lam_hi] and a nugget
    log-uniform in [1e-4, 1e-1], as in the batched-fits workload's estimated half."""
    X = rng.random((n, d))
    lam = np.exp(rng.uniform(math.log(0.05), math.log(lam_hi), d))
    s2, tau = math.exp(rng.uniform(-0.5, 0.7)), math.exp(rng.uniform(math.log(1e-4), math.log(1e-1)))
    y = math.sqrt(s2) * (_field(X, lam, nu, rng) + math.sqrt(tau) * rng.standard_normal(n)) + 0.5
    Xs = X / lam
    order = maximin_order(Xs)
    nn = find_ordered_nn(Xs[order], m)
    theta = np.concatenate([[math.log(s2)], np.log(lam), [math.log(nu)] if est else [], [math.log(tau)]])
    Xo = np.ascontiguousarray(X[order])
    return dict(theta=theta, X=Xo, y=np.ascontiguousarray(y[order]), Z=_design(Xo, trend), nn=nn, m=m)


def _batch(case, rng):
    """Problems of the case's own sizes (the same for every seed), their data from rng."""
    size = np.random.default_rng((case["count"], case["nmin"], case["nmax"]))
    out = []
    for i in range(case["count"]):
        n = int(round(math.exp(size.uniform(math.log(case["nmin"]), math.log(case["nmax"])))))
        d, m = int(size.integers(3, 13)), int(size.choice((10, 20, 30)))
        out.append(_problem(rng, n, d, m, 2.5, False, "constant", 50.0))
    return out


def _model_parts(case, rng):
    n, ns, d = case["n"], case["ns"], case["d"]
    lam = np.exp(rng.uniform(math.log(0.1), math.log(20.0), d))
    tau = math.exp(rng.uniform(math.log(1e-4), math.log(1e-2)))
    X, Xn = rng.random((n, d)), rng.uniform(-0.1, 1.1, (ns, d))
    y = _field(X, lam, 2.5, rng) + math.sqrt(tau) * rng.standard_normal(n)
    theta = np.concatenate([[0.1], np.log(lam), [math.log(tau)]])
    return dict(X=X, y=y, Xn=Xn, theta=theta, beta=np.array([0.05]))


def _model(case, p):
    gp = ScaledVecchiaGP(m_pred=case["m"], precision=case["precision"], random_state=0)
    d = case["d"]
    gp.X_, gp.y_, gp.theta_, gp.beta_, gp.b_, gp.d_ = p["X"], p["y"], p["theta"], p["beta"], 1.1, d
    gp._nu_fit, gp._estimate_nu = 2.5, False
    gp._lo, gp._span, gp._ymu, gp._ysd = np.zeros(d), np.ones(d), 0.3, 1.7
    return gp


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "loglik":
        p = _problem(rng, case["n"], case["d"], case["m"], case["nu"], case["est"], case["trend"], 50.0)
        groups = _nn_groups(p["nn"], p["m"])
        handle = DeviceProblem(p["X"], p["y"], p["Z"], groups) if case["handle"] else None
        return dict(case=case, p=p, groups=groups, handle=handle)
    if kind == "batched":
        ps = _batch(case, rng)
        batch = BatchedLikelihood([BatchProblem(p["X"], p["y"], p["Z"], _nn_groups(p["nn"], p["m"]))
                                   for p in ps], precisions=(case["precision"],))
        batch.capture()
        return dict(case=case, batch=batch, thetas=[p["theta"] for p in ps])
    if kind == "order":
        lam = np.exp(rng.uniform(math.log(0.05), math.log(50.0), case["d"]))
        return dict(case=case, Xs=rng.random((case["n"], case["d"])) / lam)
    if kind in ("predict", "joint"):
        p = _model_parts(case, rng)
        return dict(case=case, gp=_model(case, p), Xn=p["Xn"])
    lam = np.array([0.2, 0.3, 0.5, 1.0, 2.0, 5.0, 3.0, 0.8])[:case["d"]]
    X = rng.random((case["n"], case["d"]))
    y = _field(X, lam, 2.5, rng) + 0.1 * rng.standard_normal(case["n"]) + 0.5
    return dict(case=case, X=X, y=y)


def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind == "loglik":
        p = state["p"]
        nu = None if c["est"] else c["nu"]
        if state["handle"] is not None:
            return state["handle"].evaluate(p["theta"], nu, estimate_nu=c["est"], precision=c["precision"])
        return vecchia_profile_loglik(p["theta"], p["X"], p["y"], p["Z"], state["groups"], nu,
                                      estimate_nu=c["est"], precision=c["precision"])
    if kind == "batched":
        res = state["batch"].evaluate(state["thetas"])
        return dict(ll=np.array([r[1] for r in res]), grad=np.concatenate([r[2] for r in res]),
                    fisher=np.concatenate([r[3].ravel() for r in res]),
                    beta=np.concatenate([r[4] for r in res]))
    if kind == "order":
        order = maximin_order(state["Xs"])
        return order, find_ordered_nn(state["Xs"][order], c["m"])
    if kind == "predict":
        return state["gp"].predict(state["Xn"], return_std=True)
    if kind == "joint":
        return state["gp"].sample_joint(state["Xn"], n_sim=c["sims"])
    gp = ScaledVecchiaGP(m_est=c["m"], precision=c["precision"]).fit(state["X"], state["y"])
    return dict(theta=gp.theta_, beta=gp.beta_, loglik=gp.loglik_, b=gp.b_)


# ------------------------------------------------------------------ work

def _loglik_work(n, d, m, q, est):
    """Per block: inputs and conditioning set once, K^3/3 + (P + 2 + q) K^2 for the factor and the
    solves, the distances and the products dSigma a, the Gram products."""
    K, P = min(m + 1, n), d + 2 + int(est)
    flops = n * (K**3 / 3 + (P + 1 + q) * K**2 + 3 * d * K**2 + K * P * (P + 1 + 2 * q + 2))
    return 8.0 * n * (d + 1 + q) + 4.0 * n * m, flops


def work(case):
    kind, n = case["kind"], case.get("n")
    q = {"zero": 0, "constant": 1, "linear": 1 + case.get("d", 0)}[case.get("trend", "constant")]
    if kind == "loglik":
        b, f = _loglik_work(n, case["d"], case["m"], q, case["est"])
    elif kind == "batched":
        # the mean over the drawn sizes (log-uniform), dimensions and neighbour counts
        lo, hi = case["nmin"], case["nmax"]
        mean = (hi - lo) / math.log(hi / lo)
        b, f = _loglik_work(case["count"] * mean, 7.5, 20, 1, False)
    elif kind == "order":
        # screens of all earlier rows, by both searches
        b, f = 8.0 * n * (case["d"] + 1 + case["m"] + 1), 3.0 * case["d"] * float(n) * n
    elif kind == "predict":
        K = min(case["m"], n) + 1
        b = 8.0 * (n + case["ns"]) * (case["d"] + 2)
        f = case["ns"] * (K**3 / 3 + K**2 + 1.5 * case["d"] * K**2 + 3.0 * case["d"] * n)
    elif kind == "joint":
        K, ns = min(case["m"], n) + 1, case["ns"]
        b = 8.0 * (n + ns) * (case["d"] + 2) + 16.0 * ns * case["sims"]
        f = ns * (K**3 / 3 + K**2 + 1.5 * case["d"] * K**2 + 2.0 * K * case["sims"]
                  + 3.0 * case["d"] * (n + ns)) + 1.5 * case["d"] * float(n) * n
    else:
        # about 25 objective calls and 5 reorders
        b, f = _loglik_work(n, case["d"], case["m"], 1, False)
        b, f = 30 * b, 25 * f + 15.0 * case["d"] * float(n) * n
    return {"bytes": float(b), "flops": float(f)}


# ------------------------------------------------------------------ 64-bit values

def _kv(nu, x):
    """K_nu(x) by the trapezoidal rule on its integral of exp(-x cosh t) cosh(nu t)."""
    t = torch.arange(0, 481, dtype=torch.float64, device=x.device) * 0.04
    s = 0.5 * torch.exp(-x)
    for v in t[1:].tolist():
        s = s + torch.exp(-x * math.cosh(v)) * math.cosh(nu * v)
    return 0.04 * s


def _general(r, nu, want_g):
    c = math.sqrt(2.0 * nu) * r
    near = c < 1e-6
    x = torch.where(near, torch.ones_like(c), c)
    k = math.exp((1.0 - nu) * math.log(2.0) - math.lgamma(nu))
    M = torch.where(near, torch.ones_like(c), k * x**nu * _kv(nu, x))
    if not want_g:
        return M
    g = torch.where(near, torch.zeros_like(c), -(2.0 * nu / x) * k * x**nu * _kv(nu - 1.0, x))
    return M, g


def _matern(r, nu):
    if nu == 0.5:
        e = torch.exp(-r)
        return e, torch.where(r > 0, -e / torch.where(r > 0, r, torch.ones_like(r)), torch.zeros_like(r))
    if nu == 1.5:
        c = math.sqrt(3.0) * r
        e = torch.exp(-c)
        return (1.0 + c) * e, -3.0 * e
    if nu == 2.5:
        c = math.sqrt(5.0) * r
        e = torch.exp(-c)
        return (1.0 + c + c * c / 3.0) * e, -(5.0 / 3.0) * (1.0 + c) * e
    return _general(r, nu, True)


def _exact_loglik(p, nu, est):
    th = p["theta"]
    n, d = p["X"].shape
    s2, lam, tau = math.exp(th[0]), np.exp(th[1:1 + d]), math.exp(th[-1])
    nu = math.exp(th[1 + d]) if est else nu
    P = len(th)
    U = torch.from_numpy(p["X"] / lam).cuda()
    q = 0 if p["Z"] is None else p["Z"].shape[1]
    D = torch.from_numpy(np.hstack([p["y"][:, None], p["Z"]] if q else [p["y"][:, None]])).cuda()
    nn = torch.from_numpy(p["nn"]).cuda()
    logl, zk, wk, wz, aD = [], [], [], [], []
    F = torch.zeros(P, P, dtype=torch.float64, device="cuda")
    spans = [(i, i + 1, i) for i in range(min(p["m"], n))]
    spans += [(a, min(a + 4096, n), p["m"]) for a in range(p["m"], n, 4096)]
    for a0, a1, k in spans:
        idx = torch.cat([nn[a0:a1, 1:k + 1], nn[a0:a1, :1]], 1)
        u = U[idx]
        K, B = k + 1, a1 - a0
        sq = (u[:, :, None, :] - u[:, None, :, :]).square()
        r = sq.sum(3).sqrt()
        M, g = _matern(r, nu)
        S = s2 * M
        S.diagonal(dim1=1, dim2=2).add_(s2 * tau)
        L = torch.linalg.cholesky(S)
        e = torch.zeros(B, K, 1, dtype=torch.float64, device="cuda")
        e[:, -1] = 1.0
        a = torch.linalg.solve_triangular(L.transpose(1, 2), e, upper=True)
        cols = [S @ a]
        G = -s2 * g * a.transpose(1, 2)
        cols += [(G * sq[..., l]).sum(2, keepdim=True) for l in range(d)]
        if est:
            dM = (_general(r, nu + NU_H, False) - _general(r, nu - NU_H, False)) / (2.0 * NU_H)
            cols.append(s2 * nu * (dM @ a))
        cols.append(s2 * tau * a)
        cols.append(D[idx])
        W = torch.linalg.solve_triangular(L, torch.cat(cols, 2), upper=False)
        W, z = W[:, :, :P], W[:, :, P:]
        logl.append(torch.log(L[:, -1, -1]))
        zk.append(z[:, -1])
        wk.append(W[:, -1])
        wz.append(W.transpose(1, 2) @ z)
        aD.append((a * D[idx]).sum(1))
        F += torch.einsum("bip,biq->pq", W, W) - 0.5 * W[:, -1].T @ W[:, -1]
    logl, zk, wk, wz, aD = (torch.cat(v) for v in (logl, zk, wk, wz, aD))
    ay, aZ = aD[:, 0], aD[:, 1:]
    v = torch.ones(1 + q, dtype=torch.float64, device="cuda")
    if q:
        beta = torch.linalg.solve(aZ.T @ aZ + 1e-12 * torch.eye(q, dtype=torch.float64, device="cuda"),
                                  aZ.T @ ay)
        v[1:] = -beta
    zK = zk @ v
    ll = -0.5 * (math.log(2.0 * math.pi) + 2.0 * logl + zK * zK).sum()
    grad = -0.5 * (wk * (1.0 + zK * zK)[:, None] - 2.0 * zK[:, None] * (wz @ v)).sum(0)
    return float(ll), grad.cpu().numpy(), F.cpu().numpy(), (-v[1:]).cpu().numpy()


def _blocks(U, idx, theta, nu, mask):
    """Sigma of blocks of rows idx, the nugget on the rows that mask marks."""
    u = U[idx]
    S = math.exp(theta[0]) * _matern((u[:, :, None, :] - u[:, None, :, :]).square().sum(3).sqrt(), nu)[0]
    S.diagonal(dim1=1, dim2=2).add_(math.exp(theta[0] + theta[-1]) * mask)
    return S


def _nearest(U, Q, k, before=None):
    out = []
    for a in range(0, Q.shape[0], 256):
        s = torch.zeros(Q[a:a + 256].shape[0], U.shape[0], dtype=torch.float64, device="cuda")
        for l in range(U.shape[1]):
            s += (Q[a:a + 256, l, None] - U[None, :, l]).square()
        if before is not None:
            rows = before + a + torch.arange(s.shape[0], device="cuda")
            s.masked_fill_(torch.arange(U.shape[0], device="cuda")[None, :] >= rows[:, None], math.inf)
        out.append(s.topk(k, largest=False).indices)
    return torch.cat(out)


def _exact_predict(case, p):
    lam = np.exp(p["theta"][1:1 + case["d"]])
    U, Q = torch.from_numpy(p["X"] / lam).cuda(), torch.from_numpy(p["Xn"] / lam).cuda()
    res = torch.from_numpy(p["y"] - p["beta"][0]).cuda()
    n, ns, m = case["n"], case["ns"], min(case["m"], case["n"])
    nb = _nearest(U, Q, m)
    A = torch.cat([U, Q])
    mask = torch.ones(m + 1, dtype=torch.float64, device="cuda")
    mask[-1] = 0.0
    mean, var = [], []
    for a in range(0, ns, 512):
        idx = torch.cat([nb[a:a + 512], n + torch.arange(a, min(a + 512, ns), device="cuda")[:, None]], 1)
        L = torch.linalg.cholesky(_blocks(A, idx, p["theta"], 2.5, mask))
        w = torch.linalg.solve_triangular(L[:, :-1, :-1], res[idx[:, :-1]][..., None], upper=False)
        mean.append((L[:, -1, :-1] * w[..., 0]).sum(1))
        var.append(L[:, -1, -1] ** 2)
    mean, var = torch.cat(mean), torch.cat(var)
    return (0.3 + 1.7 * (mean + p["beta"][0])).cpu().numpy(), (1.7 * (1.1 * var).sqrt()).cpu().numpy()


def _farthest(X):
    """The exact maximin order, one row at a time."""
    cols = [np.ascontiguousarray(c) for c in X.T]
    n = X.shape[0]
    i = int(np.argmin(((X - X.mean(0)) ** 2).sum(1)))
    dist, order = np.full(n, np.inf), np.empty(n, dtype=np.int64)
    for t in range(n):
        order[t] = i
        s = (cols[0] - cols[0][i]) ** 2
        for c in cols[1:]:
            s += (c - c[i]) ** 2
        np.minimum(dist, np.sqrt(s), out=dist)
        dist[i] = -1.0
        i = int(np.argmax(dist))
    return order


def _exact_joint(case, p):
    n, ns, sims = case["n"], case["ns"], case["sims"]
    lam = np.exp(p["theta"][1:1 + case["d"]])
    Xs, Qs = p["X"] / lam, p["Xn"] / lam
    oo, op = _farthest(Xs), _farthest(Qs)
    A = torch.from_numpy(np.vstack([Xs[oo], Qs[op]])).cuda()
    res = torch.from_numpy((p["y"] - p["beta"][0])[oo]).cuda()
    k = min(case["m"], n)
    nb = _nearest(A, A[n:], k, before=n)
    dep, coef, rhs = [], [], []
    for a in range(0, ns, 512):
        idx = torch.cat([nb[a:a + 512], n + torch.arange(a, min(a + 512, ns), device="cuda")[:, None]], 1)
        obs = idx < n
        L = torch.linalg.cholesky(_blocks(A, idx, p["theta"], 2.5, obs.double()))
        e = torch.zeros(idx.shape[0], k + 1, 1, dtype=torch.float64, device="cuda")
        e[:, -1] = 1.0
        col = torch.linalg.solve_triangular(L.transpose(1, 2), e, upper=True)[..., 0]
        rhs.append(-(col * obs * res[idx.clamp(max=n - 1)]).sum(1))
        coef.append(torch.where(obs, torch.zeros_like(col), col))
        dep.append((idx - n).clamp(min=0))
    dep, coef, rhs = (torch.cat(v).cpu().numpy() for v in (dep, coef, rhs))
    R = np.hstack([rhs[:, None], np.random.default_rng(0).standard_normal((ns, sims))])
    S = np.empty_like(R)
    for i in range(ns):
        S[i] = (R[i] - coef[i, :-1] @ np.where(coef[i, :-1, None] != 0, S[dep[i, :-1]], 0.0)) / coef[i, -1]
    inv = np.empty(ns, dtype=np.int64)
    inv[op] = np.arange(ns)
    S = S[inv]
    return 0.3 + 1.7 * (S[:, :1] + p["beta"][0] + math.sqrt(1.1) * S[:, 1:]).T


def exact(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "loglik":
        p = _problem(rng, case["n"], case["d"], case["m"], case["nu"], case["est"], case["trend"], 50.0)
        return _exact_loglik(p, case["nu"], case["est"])
    if kind == "batched":
        res = [_exact_loglik(p, 2.5, False) for p in _batch(case, rng)]
        return dict(ll=np.array([r[0] for r in res]), grad=np.concatenate([r[1] for r in res]),
                    fisher=np.concatenate([r[2].ravel() for r in res]),
                    beta=np.concatenate([r[3] for r in res]))
    if kind == "predict":
        return _exact_predict(case, _model_parts(case, rng))
    if kind == "joint":
        return _exact_joint(case, _model_parts(case, rng))
    return None  # orders and neighbour sets are whole numbers; a fit's path is not one computation
