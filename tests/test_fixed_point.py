"""The fixed-point block kernel (csrc/sv_fix.cuh, sv_loglik_fix.cu).

On the CPU, the arithmetic compiled as host C++ against long double: limbs
rejoin exactly, a product is within 2 units of 2^-58, a pivot's reciprocal
root within 4 relative units and the Matern terms within 4 units (their chain
of a dozen truncated 64-bit products, each below 2^-60, and the table's and
polynomial's 2^-62).  On the GPU, the kernel at the edges of its block sizes,
dimensions and ranges against the oracle; what it hands to the float64 kernels
must come out the same way."""
import math
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "pyscaledvecchia_gb300", "csrc")

DRIVER = r"""
#include "sv_fix.cuh"
#include <cstdio>
#include <cmath>
using namespace sv;
typedef long double LD;
static uint64_t st = 88172645463325252ULL;
static uint64_t rnd() { st ^= st << 13; st ^= st >> 7; st ^= st << 17; return st; }
static double uni() { return (double)(rnd() >> 11) / 9007199254740992.0; }
int main() {
  double em = 0, eg = 0, ep = 0, ex = 0;
  long bad = 0;
  for (int it = 0; it < 300000; ++it) {
    const int code = 1 + (it & 1), es = (int)(rnd() % 10) - 4;
    const double lg = (it % 3 == 0) ? -8 + 9 * uni() : -60 + 61 * uni();
    const uint64_t s = (uint64_t)std::ldexp(1.0 + uni(), 62 + (int)std::floor(lg)) ^ (rnd() & 1);
    uint64_t M, g;
    if (code == 1) fx_matern<1>(s, es, kFxExp2, M, g); else fx_matern<2>(s, es, kFxExp2, M, g);
    const LD c = std::sqrt((LD)s * (code == 1 ? 3 : 5)) * std::ldexp((LD)1, es - 31), e = std::exp(-c);
    const LD Mr = code == 1 ? (1 + c) * e : (1 + c + c * c / 3) * e, gr = code == 1 ? e : (1 + c) * e;
    em = std::fmax(em, (double)(std::fabs(std::ldexp((LD)M, -61) - Mr) * std::ldexp((LD)1, 58)));
    eg = std::fmax(eg, (double)(std::fabs(std::ldexp((LD)g, -61) - gr) * std::ldexp((LD)1, 58)));
    int64_t d = (int64_t)(rnd() >> 6) >> (rnd() % 41);
    if (d < 65536) d = 65536;
    int ee;
    const int64_t Y = fx_rsqrt_pivot(d, ee);
    bad += Y > (1ll << 58) || Y <= (1ll << 57) - 16 || ee < 0;
    const LD yr = std::ldexp((LD)Y, ee - 58) * std::sqrt(std::ldexp((LD)d, -58));
    ep = std::fmax(ep, (double)(std::fabs(yr - 1) * std::ldexp((LD)1, 58)));
    const int64_t x = ((int64_t)(rnd() >> 5) - (1ll << 58)), y = ((int64_t)(rnd() >> 5) - (1ll << 58));
    bad += fx_join(fx_split(x)) != x;
    bad += fx_split(x).l > (1 << 29) || fx_split(x).l < -(1 << 29);
    const __int128 pr = (__int128)x * y;
    const __int128 df = ((__int128)fx_mul(fx_split(x), fx_split(y)) << 58) - pr;
    ex = std::fmax(ex, std::fabs((double)df) * std::ldexp(1.0, -58));
  }
  std::printf("%.4f %.4f %.4f %.4f %ld\n", em, eg, ep, ex, bad);
}
"""


def test_arithmetic(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(DRIVER)
    subprocess.run([gxx, "-O2", "-std=gnu++17", "-I" + CSRC, str(src), "-o", str(exe)], check=True)
    em, eg, ep, ex, bad = (float(v) for v in
                           subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split())
    assert em <= 4 and eg <= 4 and ep <= 4 and ex <= 2 and bad == 0, (em, eg, ep, ex, bad)


CASES = [  # n, d, m, nu, trend columns, range lo, scale of y
    (40, 1, 5, 1.5, 0, 0.2, 1.0),
    (150, 12, 15, 2.5, 1, 0.5, 1.0),      # blocks of 16: two to a warp
    (150, 12, 16, 2.5, 1, 0.5, 1e30),     # blocks of 17
    (150, 4, 31, 1.5, 5, 0.2, 1e-30),     # blocks of 32, a linear trend
    (150, 2, 30, 2.5, 16, 0.2, 1.0),      # the most trend columns
    (150, 13, 20, 2.5, 1, 0.5, 1.0),      # d = 13: the float64 kernels
    (150, 3, 20, 2.5, 1, 0.005, 1.0),     # neighbours 32 ranges away and more
]


@pytest.mark.gpu
@pytest.mark.parametrize("n,d,m,nu,q,lo,ys", CASES)
def test_against_oracle(oracle, n, d, m, nu, q, lo, ys):
    import pyscaledvecchia_gb300 as sv
    from pyscaledvecchia_gb300.batched import BatchedLikelihood, BatchProblem
    from pyscaledvecchia_gb300.likelihood import DeviceProblem
    from pyscaledvecchia_gb300.ordering import _nn_groups
    rng = np.random.default_rng(100 * d + m)
    X = rng.random((n, d))
    y = ys * rng.standard_normal(n)
    Z = np.hstack([np.ones((n, 1)), rng.random((n, q - 1))]) if q else None
    lam = np.exp(rng.uniform(math.log(lo), math.log(20 * lo), d))
    theta = np.concatenate([[math.log(1.7)], np.log(lam), [math.log(2e-3)]])
    groups = _nn_groups(sv.find_ordered_nn(X / lam, m), m)
    ref = oracle.vecchia_loglik(theta, X, y, Z, groups, nu)
    prob = DeviceProblem(X, y, Z, groups)
    got = prob.evaluate(theta, nu)
    # conditioning up to 31 / tau ~ 2e4 times 31 float64 roundings, as the
    # float64 form's own oracle tests allow
    assert abs(got[0] - ref[0]) <= 1e-10 * abs(ref[0])
    for a, b in zip(got[1:], ref[1:]):
        np.testing.assert_allclose(a, b, rtol=1e-8, atol=1e-8 * (np.abs(b).max() if np.size(b) else 0.0))
    ll = prob.evaluate(theta, nu, need_grad=False)
    assert abs(ll[0] - got[0]) <= 1e-12 * abs(got[0])
    # the same bits in a batch that also holds a problem of another kind
    other = (X[:40, :1], y[:40], None, _nn_groups(sv.find_ordered_nn(X[:40, :1], 35), 35))
    BL = BatchedLikelihood([BatchProblem(X, y, Z, groups, nu=nu), BatchProblem(*other, nu=0.5)])
    r = BL.evaluate([theta, np.array([0.1, math.log(0.3), math.log(0.1)])])[0]
    assert r[0] == 0 and r[1] == got[0]
    for a, b in zip(r[2:], got[1:]):
        np.testing.assert_array_equal(a, b)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["float64", "split"])
@pytest.mark.parametrize("m,d,nu,lo", [(32, 1, 1.5, 0.3), (39, 5, 2.5, 0.3), (40, 12, 2.5, 0.5),
                                       (144, 3, 1.5, 0.3), (207, 4, 2.5, 0.3), (60, 13, 2.5, 0.5),
                                       (60, 2, 2.5, 0.004)])
def test_prediction_against_dense(m, d, nu, lo, precision):
    """Prediction blocks at the edges of the panels and of the kernel's range
    (d = 13 and ranges far below the neighbours' distances go elsewhere)
    against dense solves of the same blocks.  tau = 1e-2: conditioning below
    m / tau = 2e4, so float64 solves agree to 1e-10; the split form's float32
    entries to 1e-7 times that."""
    import pyscaledvecchia_gb300 as sv
    rng = np.random.default_rng(m + d)
    n, ns = 400, 9
    X, Xn = rng.random((n, d)), rng.random((ns, d))
    y = np.sin(4.0 * X.sum(1)) + 0.1 * rng.standard_normal(n)
    lam = np.exp(rng.uniform(math.log(lo), math.log(10 * lo), d))
    gp = sv.ScaledVecchiaGP(m_pred=m, nu=nu, trend="zero", precision=precision)
    gp.X_, gp.y_, gp.beta_, gp.b_, gp.d_ = X, y, np.zeros(0), 1.0, d
    gp.theta_ = np.concatenate([[math.log(1.3)], np.log(lam), [math.log(1e-2)]])
    gp._nu_fit, gp._lo, gp._span, gp._ymu, gp._ysd = nu, np.zeros(d), np.ones(d), 0.0, 1.0
    mu, var = gp.predict(Xn, return_var=True)

    def corr(r):
        c = math.sqrt(2.0 * nu) * r
        return (1.0 + c + (c * c / 3.0 if nu == 2.5 else 0.0)) * np.exp(-c)

    tol = 1e-10 if precision == "float64" else 2e-3
    for i in range(ns):
        nb = np.argsort((((X - Xn[i]) / lam) ** 2).sum(1), kind="stable")[:m]
        U, u = X[nb] / lam, Xn[i] / lam
        S = 1.3 * (corr(np.sqrt(((U[:, None] - U[None]) ** 2).sum(2))) + 1e-2 * np.eye(m))
        k = 1.3 * corr(np.sqrt(((U - u) ** 2).sum(1)))
        w = np.linalg.solve(S, k)
        assert abs(var[i] - (1.3 - w @ k)) <= tol * 1.3
        assert abs(mu[i] - w @ y[nb]) <= tol * max(1.0, np.abs(y).max())


@pytest.mark.gpu
@pytest.mark.parametrize("nu", [0.05, 1.0, 5.0, 9.99])
@pytest.mark.parametrize("lam", [1e-3, 1.0, 1e6])
def test_tables_against_bessel(nu, lam):
    """The general smoothness' tables in fixed point against the Bessel routine
    in every entry, from the smallest tabulated distances (ranges of 1e6) to
    those beyond the table (ranges of 1e-3).  Both forms' entries are within
    6e-15 of the variance; a block of 13 points and a nugget of 0.05 multiply
    that by 13 / 0.05 = 260 at most."""
    import pyscaledvecchia_gb300 as sv
    from pyscaledvecchia_gb300.batched import BatchedLikelihood, BatchProblem
    from pyscaledvecchia_gb300.likelihood import DeviceProblem
    from pyscaledvecchia_gb300.ordering import _nn_groups
    rng = np.random.default_rng(17)
    X = rng.random((300, 2))
    X[:40] = X[40:80] + 1e-6 * rng.standard_normal((40, 2))
    y = rng.standard_normal(300)
    theta = np.concatenate([[0.2], np.log([lam, 3 * lam]), [math.log(0.05)]])
    groups = _nn_groups(sv.find_ordered_nn(X / lam, 12), 12)
    BL = BatchedLikelihood([BatchProblem(X, y, None, groups, nu=nu)], matern_tables=False)
    st, *ref = BL.evaluate([theta])[0]
    if st:  # a rough field and distances on both sides of the floor: no covariance at all
        with pytest.raises(np.linalg.LinAlgError):
            DeviceProblem(X, y, None, groups).evaluate(theta, nu)
        return
    got = DeviceProblem(X, y, None, groups).evaluate(theta, nu)
    assert abs(got[0] - ref[0]) <= 260 * 6e-15 * 300
    for a, b in zip(got[1:3], ref[1:3]):
        np.testing.assert_allclose(a, b, rtol=0, atol=2 * 260 * 6e-15 * max(300.0, np.abs(b).max()))


@pytest.mark.gpu
def test_sums_do_not_depend_on_the_launch():
    """Six problems of up to 5,000 blocks together (reductions of one warp per
    CTA) and one by one (a warp per block of a lane): the same bits."""
    import pyscaledvecchia_gb300 as sv
    from pyscaledvecchia_gb300.batched import BatchedLikelihood, BatchProblem
    from pyscaledvecchia_gb300.likelihood import DeviceProblem
    from pyscaledvecchia_gb300.ordering import _nn_groups
    rng = np.random.default_rng(3)
    probs, thetas = [], []
    for n, d, m in ((5000, 3, 10), (4097, 9, 5), (700, 2, 20), (3000, 12, 18), (2500, 1, 4), (4999, 6, 8)):
        X, y, lam = rng.random((n, d)), rng.standard_normal(n), np.exp(rng.uniform(-1.0, 1.0, d))
        probs.append((X, y, np.ones((n, 1)), _nn_groups(sv.find_ordered_nn(X / lam, m), m)))
        thetas.append(np.concatenate([[0.1], np.log(lam), [math.log(1e-2)]]))
    together = BatchedLikelihood([BatchProblem(*p, nu=2.5) for p in probs]).evaluate(thetas)
    for p, th, r in zip(probs, thetas, together):
        one = DeviceProblem(*p).evaluate(th, 2.5)
        assert r[0] == 0 and r[1] == one[0]
        for a, b in zip(r[2:], one[1:]):
            np.testing.assert_array_equal(a, b)
