"""The box-tree neighbour searches (csrc/sv_knn.cu: sets of at least 16,384
rows) against the oracle: arrays equal, so the same sets in the same (distance,
index) order, on random rows, lattices full of ties and duplicates, rows far
from the origin, and at the edges of the tree's sizes and of the dimensions."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rows(kind, n, d, rng):
    if kind == "lattice":
        return np.round(rng.random((n, d)) * 6.0)
    X = rng.random((n, d)) * np.exp(rng.uniform(-2.0, 3.0, d))
    return X + 1e4 if kind == "far" else X


@pytest.mark.parametrize("kind,n,d,m,start", [
    ("random", 16384, 1, 7, 0), ("random", 16385, 12, 30, 0), ("random", 19999, 16, 31, 0),
    ("random", 20000, 4, 1, 0), ("lattice", 17001, 3, 25, 0), ("far", 17000, 5, 20, 0),
    ("random", 70000, 3, 20, 12345), ("random", 20000, 5, 12, 19999)])
def test_ordered(oracle, kind, n, d, m, start):
    from pyscaledvecchia_gb300 import find_ordered_nn
    X = _rows(kind, n, d, np.random.default_rng(n + d))
    nn = find_ordered_nn(X, m, start=start)
    ref = oracle.ordered_nn(X, m, start=start)
    np.testing.assert_array_equal(nn[start:], ref[start:])
    np.testing.assert_array_equal(nn[:start, 0], np.arange(start))
    assert (nn[:start, 1:] == -1).all()


@pytest.mark.parametrize("kind,n,nq,d,k", [("random", 16384, 2500, 6, 140), ("lattice", 16500, 2500, 3, 60),
                                           ("far", 66000, 40, 2, 20), ("random", 66000, 1, 16, 1),
                                           ("random", 20000, 2500, 9, 300)])
def test_query(oracle, kind, n, nq, d, k):
    import torch
    from pyscaledvecchia_gb300.ordering import knn_query_device
    rng = np.random.default_rng(n + k)
    X, Q = _rows(kind, n, d, rng), _rows(kind, nq, d, rng)
    nb, info = knn_query_device(torch, torch.from_numpy(X).cuda(), torch.from_numpy(Q).cuda(), k)
    assert int(info[0]) == 0
    np.testing.assert_array_equal(nb.cpu().numpy(), oracle.knn_query(X, Q, k))
