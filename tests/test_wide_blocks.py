"""Blocks that reach many ranges from their own point, with clusters and
replicates inside, in the fixed-point kernels (csrc/sv_fix.cuh,
sv_loglik_fix.cu, sv_predict_fix.cu).

On the CPU, the distance and Matern arithmetic against long double: a squared
distance is truncated once, at 2^-62 of itself (long double's own rounding
allows 2^-60), equal rows are at distance 0 and correlate by exactly 1, M and
the scaled derivative factor keep the 4 units of 2^-58 of the other arithmetic
tests.  On the GPU, results against long double evaluations of the same blocks.
Their tolerance is what errors of 2^-55 of the variance in the covariances and
in their derivatives do to the result, the largest of four random draws, eight
times: the kernels' entries are within a few 2^-58, and the factorisation's
backward error is 2^-57 of the diagonal."""
import math
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "pyscaledvecchia_gb300", "csrc")
L = np.longdouble

DRIVER = r"""
#include "sv_fix.cuh"
#include <cstdio>
#include <cmath>
using namespace sv;
typedef long double LD;
static uint64_t st = 88172645463325252ULL;
static uint64_t rnd() { st ^= st << 13; st ^= st >> 7; st ^= st << 17; return st; }
static int64_t coord() { return (int64_t)(rnd() >> 4) - (1ll << 59); }  // below 2^59
int main() {
  double es2 = 0, em = 0, eg = 0;
  long bad = 0;
  for (int it = 0; it < 200000; ++it) {
    const int d = 1 + (int)(rnd() % 12), code = 1 + (it & 1), es = (int)(rnd() % 35) - 27;
    const int near = (int)(rnd() % 62);  // how many bits closer than the extent
    FxSq q = {0, 0, 0};
    LD r2 = 0;
    for (int l = 0; l < d; ++l) {
      const int64_t x = it % 7 == 0 ? (l & 1 ? 1 : -1) * ((1ll << 59) - 1) : coord();
      int64_t y = it % 7 == 0 ? -x : near == 61 ? x : x + (coord() >> near);
      if (y >= 1ll << 59 || y <= -(1ll << 59)) y = -x;
      if (l == 8) fx_sqcarry(q);
      fx_sqdiff(q, fx_split(x), fx_split(y));
      const LD df = (LD)(x - y);
      r2 += df * df;
    }
    int E;
    const uint64_t s = fx_sqnorm(q, es, E);
    r2 = std::ldexp(r2, 2 * es - 122);
    bad += s < (1ull << 62);
    uint64_t M, g;
    if (code == 1) fx_matern_norm<1, true>(s, E, kFxExp2, M, g); else fx_matern_norm<2, true>(s, E, kFxExp2, M, g);
    if (r2 == 0) {
      bad += E != es - 92 || (M + 4) >> 3 != 1ull << 58;
      continue;
    }
    es2 = std::fmax(es2, (double)(std::fabs(std::ldexp((LD)s, 2 * E - 64) / r2 - 1) * std::ldexp((LD)1, 60)));
    const LD c = std::sqrt(r2 * (code == 1 ? 3 : 5)), e = std::exp(-c);
    const LD Mr = code == 1 ? (1 + c) * e : (1 + c + c * c / 3) * e;
    const LD gr = std::ldexp(code == 1 ? e : (1 + c) * e, 2 * E);
    em = std::fmax(em, (double)(std::fabs(std::ldexp((LD)M, -61) - Mr) * std::ldexp((LD)1, 58)));
    eg = std::fmax(eg, (double)(std::fabs(std::ldexp((LD)g, -61) - gr) * std::ldexp((LD)1, 58)));
    bad += gr > 1.5;
  }
  std::printf("%.4f %.4f %.4f %ld\n", es2, em, eg, bad);
}
"""


def test_distances(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(DRIVER)
    subprocess.run([gxx, "-O2", "-std=gnu++17", "-I" + CSRC, str(src), "-o", str(exe)], check=True)
    es2, em, eg, bad = (float(v) for v in
                        subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split())
    assert es2 <= 1 and em <= 4 and eg <= 4 and bad == 0, (es2, em, eg, bad)


# ------------------------------------------------------------------ long double

def _matern(r, nu):
    c = np.sqrt(L(2 * nu)) * r
    e = np.exp(-c)
    if nu == 2.5:
        return (1 + c + c * c / 3) * e, -(L(5) / 3) * (1 + c) * e
    return (1 + c) * e, -3 * e


def _chol(S):
    C = np.zeros_like(S)
    for j in range(S.shape[1]):
        v = S[:, j:, j] - (C[:, j:, :j] * C[:, j, None, :j]).sum(2)
        C[:, j, j] = np.sqrt(v[:, 0])
        C[:, j + 1:, j] = v[:, 1:] / C[:, j, j][:, None]
    return C


def _solve(C, V):
    W = np.zeros_like(V)
    for j in range(C.shape[1]):
        W[:, j] = (V[:, j] - (C[:, j, :j, None] * W[:, :j]).sum(1)) / C[:, j, j][:, None]
    return W


def _noise(rng, shape, eta):
    if eta == 0:
        return 0
    u = rng.uniform(-1.0, 1.0, shape)
    return (eta * (np.tril(u) + np.swapaxes(np.tril(u, -1), -1, -2))).astype(L)


def _loglik(X, y, nn, m, s2, tau, nu, rng=None, eta=0):
    """(ll, score, Fisher) without a trend, unit ranges."""
    n, d = X.shape
    U, y, s2, tau = X.astype(L), y.astype(L), L(s2), L(tau)
    P, ll, grad, F = d + 2, L(0), np.zeros(d + 2, L), np.zeros((d + 2, d + 2), L)
    for k in range(m + 1):
        rows = np.arange(n) if k == m else np.array([k])
        rows = rows[rows >= m] if k == m else rows
        idx = np.concatenate([nn[rows, 1:k + 1], rows[:, None]], 1)
        B, K = idx.shape
        sq = (U[idx][:, :, None] - U[idx][:, None]) ** 2
        M, g = _matern(np.sqrt(sq.sum(3)), nu)
        S = s2 * (M + _noise(rng, M.shape, eta))
        S[:, range(K), range(K)] += s2 * tau
        C = _chol(S)
        a = np.zeros((B, K), dtype=L)
        a[:, -1] = 1 / C[:, -1, -1]
        for j in range(K - 2, -1, -1):
            a[:, j] = -(C[:, j + 1:, j] * a[:, j + 1:]).sum(1) / C[:, j, j]
        cols = [(S * a[:, None]).sum(2)]
        for l in range(d):
            cols.append((s2 * (_noise(rng, M.shape, eta) - g * sq[..., l]) * a[:, None]).sum(2))
        W = _solve(C, np.stack(cols + [s2 * tau * a, y[idx]], 2))
        z, W = W[..., P], W[..., :P]
        zK, wK = z[:, -1], W[:, -1]
        ll -= (L(0.5) * np.log(2 * np.arctan2(L(0), L(-1))) + np.log(C[:, -1, -1]) + zK * zK / 2).sum()
        grad -= L(0.5) * (wK * (1 + zK * zK)[:, None] - 2 * zK[:, None] * (W * z[..., None]).sum(1)).sum(0)
        F += (W[..., :, None] * W[..., None, :]).sum((0, 1)) - L(0.5) * (wK[:, :, None] * wK[:, None]).sum(0)
    return ll, grad, F


def _predict(X, y, Xn, m, s2, tau, nu, rng=None, eta=0):
    X, Xn, y, s2, tau = X.astype(L), Xn.astype(L), y.astype(L), L(s2), L(tau)
    nb = np.argsort(((X[None] - Xn[:, None]) ** 2).sum(2), 1, kind="stable")[:, :m]
    U = np.concatenate([X[nb], Xn[:, None]], 1)
    M, _ = _matern(np.sqrt(((U[:, :, None] - U[:, None]) ** 2).sum(3)), nu)
    S = s2 * (M + _noise(rng, M.shape, eta))
    S[:, range(m), range(m)] += s2 * tau
    C = _chol(S)
    w = _solve(C[:, :-1, :-1], y[nb][..., None])[..., 0]
    return (C[:, -1, :-1] * w).sum(1), C[:, -1, -1] ** 2


def _check(got, f):
    ref = f()
    tol = [0.0] * len(ref)
    for seed in range(4):
        for i, v in enumerate(f(rng=np.random.default_rng(seed), eta=2.0 ** -55)):
            tol[i] = max(tol[i], float(np.abs(v - ref[i]).max()))
    for g, r, t in zip(got, ref, tol):
        # (and the result's own float64 rounding, over the sums)
        assert float(np.abs(np.asarray(g, dtype=L) - r).max()) <= 8 * t + 1e-15 * float(np.abs(r).max())


def _design(kind, d, reach, n, rng):
    """n rows whose 20 nearest earlier ones reach about `reach` ranges."""
    side = reach / (20.0 / n) ** (1.0 / d)
    if kind == "clusters":  # of six, 0.02 ranges across
        X = np.repeat(rng.random((n // 6, d)) * side, 6, 0) + 0.02 * rng.standard_normal((n, d))
    else:                   # three times each row
        X = np.repeat(rng.random((n // 3, d)) * side, 3, 0)
    return X[rng.permutation(n)]


CASES = [("clusters", 2, 8.0, 2.5), ("clusters", 3, 16.0, 1.5), ("clusters", 9, 28.0, 2.5),
         ("replicates", 2, 2.0, 1.5), ("replicates", 3, 8.0, 2.5), ("replicates", 10, 16.0, 1.5),
         ("replicates", 2, 28.0, 2.5)]


def _data(kind, d, reach):
    rng = np.random.default_rng(int(100 * d + reach))
    n, tau = 72, 1e-8
    X = _design(kind, d, reach, n, rng)
    y = np.sin(X @ (0.7 * rng.standard_normal((d, 6)))).sum(1) + math.sqrt(tau) * rng.standard_normal(n)
    return X, y, tau, rng


@pytest.mark.gpu
@pytest.mark.parametrize("kind,d,reach,nu", CASES)
def test_likelihood(kind, d, reach, nu):
    if np.finfo(L).eps > 1e-18:
        pytest.skip("no long double beyond float64")
    import pyscaledvecchia_gb300 as sv
    from pyscaledvecchia_gb300.likelihood import DeviceProblem
    from pyscaledvecchia_gb300.ordering import _nn_groups
    X, y, tau, _ = _data(kind, d, reach)
    nn = sv.find_ordered_nn(X, 20)
    theta = np.concatenate([[0.0], np.zeros(d), [math.log(tau)]])
    got = DeviceProblem(X, y, None, _nn_groups(nn, 20)).evaluate(theta, nu)
    # (the parameters as the device has them: exp of theta in float64)
    _check(got[:3], lambda **kw: _loglik(X, y, nn, 20, 1.0, np.exp(L(theta[-1])), nu, **kw))


@pytest.mark.gpu
@pytest.mark.parametrize("kind,d,reach,nu", CASES)
def test_prediction(kind, d, reach, nu):
    if np.finfo(L).eps > 1e-18:
        pytest.skip("no long double beyond float64")
    import pyscaledvecchia_gb300 as sv
    X, y, tau, rng = _data(kind, d, reach)
    Xn = X[:20] + 0.1 * rng.standard_normal((20, d))
    gp = sv.ScaledVecchiaGP(m_pred=40, nu=nu, trend="zero")
    gp.X_, gp.y_, gp.beta_, gp.b_, gp.d_ = X, y, np.zeros(0), 1.0, d
    gp.theta_ = np.concatenate([[0.0], np.zeros(d), [math.log(tau)]])
    gp._nu_fit, gp._lo, gp._span, gp._ymu, gp._ysd = nu, np.zeros(d), np.ones(d), 0.0, 1.0
    got = gp.predict(Xn, return_var=True)
    _check(got, lambda **kw: _predict(X, y, Xn, 40, 1.0, np.exp(L(gp.theta_[-1])), nu, **kw))
