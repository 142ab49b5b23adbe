"""DeviceProblem.launch on a caller's stream: the results and the status words
belong to that stream alone, whatever torch's current stream has left to do, and
the buffers handed out before the first launch are the ones it writes."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("est", [False, True])
def test_results_of_a_stream_ahead_of_the_current_one(est):
    import ctypes

    import torch
    import pyscaledvecchia_gb300 as sv
    from pyscaledvecchia_gb300 import _lib
    from pyscaledvecchia_gb300.likelihood import DeviceProblem
    from pyscaledvecchia_gb300.ordering import _nn_groups
    rng = np.random.default_rng(4)
    n, d, m = 400, 3, 10
    X, y = rng.random((n, d)), rng.standard_normal(n)
    groups = _nn_groups(sv.find_ordered_nn(X, m), m)
    theta = np.concatenate([[0.1], np.log([0.3, 0.5, 0.8]), [math.log(1.3)] if est else [], [math.log(1e-2)]])
    P = len(theta)
    prob, other = DeviceProblem(X, y, None, groups), DeviceProblem(X, y, None, groups)
    ref = other.evaluate(theta, None if est else 2.5, estimate_nu=est)
    th = _lib.to_dev(torch, theta, np.float64)
    prob.chunk_tensor(P)
    info = prob.info
    assert prob.out is None
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    torch.cuda._sleep(100_000_000)  # tens of milliseconds ahead of anything enqueued by launch()
    prob.launch(th, P, None if est else 2.5, est, True, 0.0, 0.0,
                stream=ctypes.c_void_p(side.cuda_stream))
    side.synchronize()
    torch.cuda.synchronize()
    out = prob.out.cpu().numpy()
    assert prob.info.data_ptr() == info.data_ptr() and int(info[0]) == 0
    assert out[0] == ref[0]
    np.testing.assert_array_equal(out[1:1 + P], ref[1])
    np.testing.assert_array_equal(out[1 + P:1 + P + P * P].reshape(P, P), ref[2])


def test_results_with_and_without_an_estimated_nu():
    """One handle evaluated both ways in turn: the two results lie side by side."""
    import pyscaledvecchia_gb300 as sv
    from pyscaledvecchia_gb300.likelihood import DeviceProblem
    from pyscaledvecchia_gb300.ordering import _nn_groups
    rng = np.random.default_rng(5)
    X, y = rng.random((300, 2)), rng.standard_normal(300)
    Z = np.hstack([np.ones((300, 1)), X])
    groups = _nn_groups(sv.find_ordered_nn(X, 8), 8)
    fixed, est = np.array([0.1, -1.0, -0.5, -4.0]), np.array([0.1, -1.0, -0.5, 0.3, -4.0])
    prob = DeviceProblem(X, y, Z, groups)
    for _ in range(2):
        for th, nu, e in ((fixed, 2.5, False), (est, None, True)):
            got = prob.evaluate(th, nu, estimate_nu=e)
            ref = DeviceProblem(X, y, Z, groups).evaluate(th, nu, estimate_nu=e)
            assert got[0] == ref[0]
            for a, b in zip(got[1:], ref[1:]):
                np.testing.assert_array_equal(a, b)
            held = prob.out
    first = prob.out.cpu().numpy()
    prob.evaluate(fixed, 2.5)
    np.testing.assert_array_equal(held.cpu().numpy(), first)
