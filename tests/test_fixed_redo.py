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


@pytest.mark.gpu
@pytest.mark.parametrize("nus,d,launched", [((0.5, 0.5), 3, False), ((0.8, None), 3, False), ((2.5, 1.5), 13, False),
                                            ((0.5, 2.5), 3, True), ((1.5, 0.8), 12, True)])
def test_batch_knows_whether_it_has_work_for_the_kernel(nus, d, launched):
    """A batch without a problem for the fixed-point kernel does not launch it;
    the results are those of the problems alone either way."""
    import pyscaledvecchia_gb300 as sv
    from pyscaledvecchia_gb300.batched import BatchedLikelihood, BatchProblem
    from pyscaledvecchia_gb300.likelihood import DeviceProblem
    from pyscaledvecchia_gb300.ordering import _nn_groups
    rng = np.random.default_rng(d)
    probs, thetas = [], []
    for nu in nus:
        X, y = rng.random((120, d)), rng.standard_normal(120)
        groups = _nn_groups(sv.find_ordered_nn(X, 18), 18)
        probs.append(BatchProblem(X, y, None, groups, nu=nu, estimate_nu=nu is None))
        thetas.append(np.concatenate([[0.1], np.zeros(d), [math.log(1.2)] if nu is None else [], [-4.0]]))
    BL = BatchedLikelihood(probs)
    assert all((m["bdesc"].general_nu & 2 == 0) == launched for m in BL._modes.values())
    for pr, nu, th, r in zip(probs, nus, thetas, BL.evaluate(thetas)):
        one = DeviceProblem(pr.Xo, pr.yo, None, pr.groups).evaluate(th, nu, estimate_nu=nu is None)
        assert r[0] == 0 and r[1] == one[0]
        np.testing.assert_array_equal(r[2], one[1])
        np.testing.assert_array_equal(r[3], one[2])
