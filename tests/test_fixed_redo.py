"""Blocks that the fixed-point likelihood kernel hands to the float64 kernels
(csrc/sv_loglik_fix.cu) beside blocks that it keeps, in the two halves of one
warp (m = 7, 15), in whole warps and in a batch: rows in a dense cluster, whose
blocks are narrow, and rows 50 ranges and more apart, in random order."""
import math

import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("m", [7, 15, 24])
def test_kept_and_left_blocks_together(oracle, m):
    import pyscaledvecchia_gb300 as sv
    from pyscaledvecchia_gb300.batched import BatchedLikelihood, BatchProblem
    from pyscaledvecchia_gb300.likelihood import DeviceProblem
    from pyscaledvecchia_gb300.ordering import _nn_groups
    rng = np.random.default_rng(m)
    n, d = 203, 3
    X = rng.random((n, d))
    X[rng.permutation(n)[:n // 2]] *= 400.0
    y = rng.standard_normal(n)
    theta = np.concatenate([[0.2], np.zeros(d), [math.log(1e-2)]])
    groups = _nn_groups(sv.find_ordered_nn(X, m), m)
    ref = oracle.vecchia_loglik(theta, X, y, None, groups, 2.5)
    got = DeviceProblem(X, y, None, groups).evaluate(theta, 2.5)
    # pivots above 1e-2 of the variance: a few hundred float64 roundings each
    assert abs(got[0] - ref[0]) <= 1e-12 * abs(ref[0])
    for a, b in zip(got[1:3], ref[1:3]):
        np.testing.assert_allclose(a, b, rtol=0, atol=1e-11 * np.abs(b).max())
    r = BatchedLikelihood([BatchProblem(X, y, None, groups, nu=2.5)] * 3).evaluate([theta] * 3)
    for one in r:
        assert one[0] == 0 and one[1] == got[0]
        np.testing.assert_array_equal(one[2], got[1])
        np.testing.assert_array_equal(one[3], got[2])
