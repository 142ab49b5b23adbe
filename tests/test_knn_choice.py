"""Ordered neighbour searches whose choice between box tree and screens is made
on the device (csrc/sv_knn.cu: 32,768 rows and more in more than 8 or 9
dimensions), on either side of it, against the oracle: arrays equal."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ranges", ["one", "spread"])  # the screens, the tree
@pytest.mark.parametrize("n,d,m,start", [(32768, 10, 5, 0), (33001, 16, 20, 0), (33000, 12, 50, 0), (32769, 9, 16, 0),
                                         (66000, 11, 30, 60000), (33000, 13, 15, 32990),
                                         (66000, 16, 20, 65900)])
def test_ordered(oracle, ranges, n, d, m, start):
    from pyscaledvecchia_gb300 import find_ordered_nn
    rng = np.random.default_rng(n + d)
    X = rng.random((n, d))
    if ranges == "spread":
        X *= np.exp(rng.uniform(math.log(0.02), math.log(20.0), d))
    nn = find_ordered_nn(X, m, start=start)
    ref = oracle.ordered_nn(X, m, start=start)
    np.testing.assert_array_equal(nn[start:], ref[start:])
    np.testing.assert_array_equal(nn[:start, 0], np.arange(start))
    assert (nn[:start, 1:] == -1).all()
