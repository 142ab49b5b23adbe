"""The pass maximin (csrc/sv_reorder.cu) where its tensor-core screen and its
lists can go wrong: rows at the edges of the 32-point tiles, coordinates at the
edges of the 16-wide steps, float32 and bf16 extremes of scale, images that
round to one value, duplicates.  The oracle's order, index by index."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rows(kind, n, d):
    rng = np.random.default_rng(1000 * n + d)
    X = rng.standard_normal((n, d))
    if kind == "tiny":        # squares below float32's range
        return X * 1e-27
    if kind == "huge":        # squares above it: refused
        return X * 1e25
    if kind == "far":         # images of one bf16 value, 1e-3 apart
        return X * 1e-3 + np.where(np.arange(n) % 2, 300.0, -300.0)[:, None]
    if kind == "scales":      # a cluster, and a few rows far away
        X *= 1e-4
        X[::97] *= 1e6
        return X
    if kind == "lattice":
        return np.round(X * 2.0)
    if kind == "line":        # evenly spaced: near ties everywhere
        return np.repeat(np.arange(n, dtype=np.float64)[:, None], d, 1) * 0.1
    return X


@pytest.mark.parametrize("flags", [0, 4])
@pytest.mark.parametrize("kind,n,d", [
    ("normal", 2, 1), ("normal", 31, 3), ("normal", 33, 15), ("normal", 700, 16), ("normal", 701, 17),
    ("normal", 1025, 32), ("normal", 900, 33), ("normal", 640, 64), ("normal", 6007, 2), ("tiny", 1500, 5),
    ("huge", 1500, 5), ("far", 3001, 4), ("scales", 4000, 6), ("lattice", 3000, 3), ("line", 2500, 2)])
def test_order(oracle, kind, n, d, flags):
    import torch
    from pyscaledvecchia_gb300.ordering import maximin_order_device
    X = _rows(kind, n, d)
    order, info = maximin_order_device(torch, torch.from_numpy(X).cuda(), n // 3, flags)
    if kind == "huge":
        assert int(info[0]) == 1  # SV_EINVAL: no finite float32 distance
        return
    assert int(info[0]) == 0
    np.testing.assert_array_equal(order.cpu().numpy(), oracle.maximin_order(X, first=n // 3))


def test_cluster_sizes_of_a_batch():
    """A problem takes more CTAs when the whole batch has room on the SMs: the
    same orders from a batch that has none (90 problems) and one by one."""
    import math
    from pyscaledvecchia_gb300.batched import BatchedLikelihood, BatchProblem, ordered_groups
    rng = np.random.default_rng(8)
    n, d, m, nprob = 600, 3, 5, 90
    raw = [(rng.random((n, d)), rng.standard_normal(n)) for _ in range(nprob)]
    thetas = [np.concatenate([[0.1], rng.uniform(-2.0, 2.0, d), [math.log(1e-3)]]) for _ in range(nprob)]
    BL = BatchedLikelihood([BatchProblem(X, y, None, ordered_groups(n, m)) for X, y in raw])
    BL.set_sources([r[0] for r in raw], [r[1] for r in raw], [None] * nprob, [m] * nprob)
    together = BL.reorder(list(range(nprob)), thetas, return_orders=True)
    for i in range(0, nprob, 30):
        np.testing.assert_array_equal(BL.reorder([i], [thetas[i]], return_orders=True)[0], together[i])
