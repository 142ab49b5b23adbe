"""The fixed-point prediction kernel's back substitution (csrc/sv_predict_fix.cu):
a column's unit follows its largest weight, and the sums that the panels'
inverse blocks magnify keep what one rounding to 2^-58 loses."""
import math

import numpy as np
import pytest
from test_wide_blocks import L, _predict

pytestmark = pytest.mark.gpu


def test_unit_of_the_column():
    """Extrapolation from 36 points on a line, largest weight 15: every entry of
    the column is a whole multiple of the column's unit, which may not be
    coarser than float64's last place of the largest."""
    import torch
    from pyscaledvecchia_gb300 import _lib
    lib = _lib.load_library()
    k = 36
    X = np.concatenate([np.arange(k) / (k - 1.0), [1.2]])[:, None]
    D = _lib.PredDesc()
    D.nblk, D.nobs, D.d, D.k, D.ldnbr, D.nu = 1, k, 1, k, k, 2.5
    dev = lambda a, t: _lib.to_dev(torch, np.asarray(a), t)
    # s2 = 1/2, tau = 1e-6: the covariance's scale is 1, so the column is units times 2^n
    th, Xd = dev([math.log(0.5), 0.0, math.log(1e-6)], np.float64), dev(X, np.float64)
    tgt, nbr = dev([k], np.int32), dev(np.arange(k)[None], np.int32)
    acol, rhs = torch.empty((1, k + 1), dtype=torch.float64, device="cuda"), torch.empty(1, dtype=torch.float64,
                                                                                         device="cuda")
    resid = torch.zeros(k, dtype=torch.float64, device="cuda")
    info = _lib.new_info(torch)
    rc = lib.sv_predict_blocks(D, _lib.ptr(th), _lib.ptr(Xd), _lib.ptr(tgt), _lib.ptr(nbr), _lib.ptr(resid),
                               None, None, _lib.ptr(acol), _lib.ptr(rhs), _lib.ptr(info), _lib.stream_handle(torch))
    _lib.check(lib, rc, "sv_predict_blocks")
    a = acol.cpu().numpy()[0]
    assert 8.0 < np.abs(a[:k]).max() / a[k] < 16.0
    mant, ex = np.frexp(a)
    low = [int(e) - 53 + (int(abs(m) * 2 ** 53) & -int(abs(m) * 2 ** 53)).bit_length() - 1
           for m, e in zip(mant, ex) if m != 0]
    assert min(low) <= int(ex[np.abs(a).argmax()]) - 53


@pytest.mark.parametrize("d,reach,tau,nu", [(8, 1.5, 1e-4, 1.5), (8, 3.0, 1e-4, 2.5), (8, 0.5, 1e-4, 2.5),
                                            (6, 1.5, 1e-3, 2.5)])
def test_mean_of_clusters(d, reach, tau, nu):
    """Means over clusters 0.02 ranges across against long double: no further
    off than float64's rounding of the covariances makes them (the largest of
    four draws of errors of 2^-53 of the variance)."""
    if np.finfo(L).eps > 1e-18:
        pytest.skip("no long double beyond float64")
    import pyscaledvecchia_gb300 as sv
    rng = np.random.default_rng(int(10 * d + 100 * reach))
    n, m = 240, 60
    X = np.repeat(rng.random((n // 6, d)) * reach / 0.29, 6, 0) + 0.02 * rng.standard_normal((n, d))
    X = X[rng.permutation(n)]
    y = np.sin(X @ (0.7 * rng.standard_normal((d, 8)))).sum(1) / 2 + math.sqrt(tau) * rng.standard_normal(n)
    Xn = X[:30] + 0.1 * rng.standard_normal((30, d))
    Xn[15:] = X[:15] + 0.3 * rng.standard_normal((15, d))
    gp = sv.ScaledVecchiaGP(m_pred=m, nu=nu, trend="zero")
    gp.X_, gp.y_, gp.beta_, gp.b_, gp.d_ = X, y, np.zeros(0), 1.0, d
    gp.theta_ = np.concatenate([[0.0], np.zeros(d), [math.log(tau)]])
    gp._nu_fit, gp._lo, gp._span, gp._ymu, gp._ysd = nu, np.zeros(d), np.ones(d), 0.0, 1.0
    got = gp.predict(Xn)
    f = lambda **kw: _predict(X, y, Xn, m, 1.0, np.exp(L(gp.theta_[-1])), nu, **kw)[0]
    ref = f()
    tol = max(float(np.abs(f(rng=np.random.default_rng(s), eta=2.0 ** -53) - ref).max()) for s in range(4))
    assert float(np.abs(got - ref).max()) <= tol
