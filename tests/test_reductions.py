"""The evaluation's sums (csrc/sv_loglik.cu) have the same bits in every form of
the launch: clusters or one CTA per partition, sums in registers for 8, 16 or
of them at a time, one warp per run or several."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _problems(sizes):
    import pyscaledvecchia_gb300 as sv
    from pyscaledvecchia_gb300.ordering import _nn_groups
    rng = np.random.default_rng(len(sizes))
    probs, thetas = [], []
    for n, d, m in sizes:
        X, y, lam = rng.random((n, d)), rng.standard_normal(n), np.exp(rng.uniform(-1.0, 1.0, d))
        probs.append((X, y, np.ones((n, 1)), _nn_groups(sv.find_ordered_nn(X / lam, m), m)))
        thetas.append(np.concatenate([[0.1], np.log(lam), [math.log(1e-2)]]))
    return probs, thetas


@pytest.mark.parametrize("sizes,alone", [
    # a problem of 17 parameters: two rounds of 16, 3 warps a run
    (((5000, 3, 10), (4097, 9, 5), (700, 2, 20), (3000, 15, 6), (4999, 6, 8)), range(5)),
    # the same with 20,000 blocks (4 warps a run) and 66 parameters
    (((20000, 2, 4), (300, 64, 5), (1025, 14, 5)), range(3)),
    # partitions enough for a CTA each, of 3 to 128 blocks a run
    ([(130 + 17 * i, 1 + i % 13, 4) for i in range(48)] + [(3000, 5, 6)], (0, 12, 29, 47, 48)),
    ([(2990 + 5 * i, 1 + i % 3, 3) for i in range(46)] + [(8192, 2, 3), (9000, 4, 3)], (0, 21, 46, 47))])
def test_sums_are_those_of_the_problem_alone(sizes, alone):
    from pyscaledvecchia_gb300.batched import BatchedLikelihood, BatchProblem
    from pyscaledvecchia_gb300.likelihood import DeviceProblem
    probs, thetas = _problems(sizes)
    for nu in (2.5, 0.5):
        together = BatchedLikelihood([BatchProblem(*p, nu=nu) for p in probs]).evaluate(thetas)
        for i in alone:
            one = DeviceProblem(*probs[i]).evaluate(thetas[i], nu)
            r = together[i]
            assert r[0] == 0 and r[1] == one[0]
            for a, b in zip(r[2:], one[1:]):
                np.testing.assert_array_equal(a, b)
