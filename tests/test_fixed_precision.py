"""The fixed-point kernels' results on evenly spread rows and nuggets of 0.01 to
1, where blocks are well conditioned and a limb's product left out anywhere
would show: against long double, with the tolerance of test_wide_blocks.py (what
errors of 2^-55 of the variance in the covariances and their derivatives do, eight
times, and 1e-15 for the results' own rounding)."""
import math

import numpy as np
import pytest
from test_wide_blocks import L, _check, _loglik, _predict

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(np.finfo(L).eps > 1e-18, reason="no long double beyond float64")]

CASES = [(1, 0.5, 1.0, 2.5), (2, 3.0, 0.1, 1.5), (4, 0.3, 0.01, 2.5), (8, 1.0, 0.1, 2.5), (12, 2.0, 1.0, 1.5)]


def _data(d, side, tau):
    rng = np.random.default_rng(int(100 * d + 10 * side))
    X = rng.random((72, d)) * side
    y = np.sin(X @ (0.7 * rng.standard_normal((d, 6)))).sum(1) + math.sqrt(tau) * rng.standard_normal(72)
    return X, y, rng


@pytest.mark.parametrize("m", [15, 31])
@pytest.mark.parametrize("d,side,tau,nu", CASES)
def test_likelihood(d, side, tau, nu, m):
    import pyscaledvecchia_gb300 as sv
    from pyscaledvecchia_gb300.likelihood import DeviceProblem
    from pyscaledvecchia_gb300.ordering import _nn_groups
    X, y, _ = _data(d, side, tau)
    nn = sv.find_ordered_nn(X, m)
    theta = np.concatenate([[0.0], np.zeros(d), [math.log(tau)]])
    got = DeviceProblem(X, y, None, _nn_groups(nn, m)).evaluate(theta, nu)
    _check(got[:3], lambda **kw: _loglik(X, y, nn, m, 1.0, np.exp(L(theta[-1])), nu, **kw))


@pytest.mark.parametrize("d,side,tau,nu", CASES)
def test_prediction(d, side, tau, nu):
    import pyscaledvecchia_gb300 as sv
    X, y, rng = _data(d, side, tau)
    Xn = rng.random((20, d)) * side
    gp = sv.ScaledVecchiaGP(m_pred=50, nu=nu, trend="zero")
    gp.X_, gp.y_, gp.beta_, gp.b_, gp.d_ = X, y, np.zeros(0), 1.0, d
    gp.theta_ = np.concatenate([[0.0], np.zeros(d), [math.log(tau)]])
    gp._nu_fit, gp._lo, gp._span, gp._ymu, gp._ysd = nu, np.zeros(d), np.ones(d), 0.0, 1.0
    got = gp.predict(Xn, return_var=True)
    _check(got, lambda **kw: _predict(X, y, Xn, 50, 1.0, np.exp(L(gp.theta_[-1])), nu, **kw))
