"""The scratch that the neighbour searches ask for: a box tree is built over the
reference rows alone, so queries add only their images and bounds."""
import pytest


@pytest.mark.parametrize("d,DP", [(1, 4), (6, 8), (16, 16), (20, 24)])
def test_queries_add_images_and_bounds(d, DP):
    from pyscaledvecchia_gb300 import _lib
    lib = _lib.load_library()
    for nref in (0, 100, 16384, 70000):
        ref = lib.sv_ordered_knn_workspace_bytes(nref, d)
        for nq in (1, 5000, 20000, 100000):
            assert lib.sv_knn_query_workspace_bytes(nref, nq, d) - ref <= 512 + 4 * nq * (DP + 1) + 2 * 256
    # and the tree's part is there, from the size on at which it may be built
    if d <= 16:
        grown = lib.sv_ordered_knn_workspace_bytes(16384, d) - lib.sv_ordered_knn_workspace_bytes(16383, d)
        assert grown > 16384 * (2 * 8 + 2 * 4)
