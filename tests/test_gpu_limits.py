"""Counts where the counters' width and the padding of partly filled runs would
show (exact: integers, no tolerance)."""
import numpy as np
import pytest

from corruscant_b200 import _native as N
from oracle import oracle as O

pytestmark = pytest.mark.gpu

MODES = (N.KD_MODE_MIXED, N.KD_MODE_FP64)


def test_more_pairs_of_a_warp_than_32_bits():
    """More than 2^27 tree points below one edge, for 32 queries of one field
    in a block that holds two: their sum passes 2^32 (at 2^27 points it would
    wrap to zero).  Each tree place is taken 225 times, so that the tree itself
    stays small."""
    places, copies = 600_000, 225
    n = places * copies
    assert n > 2 ** 27
    rs = np.random.RandomState(1)
    t = N.build_tree(np.repeat(rs.rand(places, 3), copies, axis=0), None, 2)
    try:
        q = 0.5 + 0.01 * rs.rand(128, 3)
        f = np.zeros(128, np.int32)
        f[100] = 1
        for mode in MODES:
            got = N.count_points(t, q, f, 2, [10.0], mode=mode)
            assert np.array_equal(got, [[127 * n, 0, n, 0]]), mode  # query field by tree field
    finally:
        N.destroy(t)


@pytest.mark.parametrize("nt", [1, 2, 3, 4, 61, 62, 63, 64, 65, 1000])
def test_query_at_the_largest_coordinates(nt):
    """Queries in the corners of the coordinate range, where a run is not a
    multiple of the points that are staged together: no place is taken by
    anything but a point."""
    rs = np.random.RandomState(nt)
    tp = rs.rand(nt, 3)
    far = np.array([1e300, 1e290, 1.7e308, 1e200])
    q = np.concatenate([s * far[:, None] * np.ones(3) for s in (1.0, -1.0)] + [rs.rand(9, 3)])
    radii = np.array([0.3, 2.0, 1e150, 1e154, np.inf])
    want = O.OracleTree(tp).brute_counts(q, None, 1, radii, nthreads=4)
    t, tq = N.build_tree(tp, None, 1), N.build_tree(q, None, 1)
    try:
        for mode in MODES:
            assert np.array_equal(N.count_points(t, q, None, 1, radii, mode=mode), want), mode
            assert np.array_equal(N.count_radii(t, tq, radii, mode=mode), want), mode
            auto = N.count_radii(tq, tq, radii, mode=mode)
            assert np.array_equal(auto, O.OracleTree(q).brute_counts(q, None, 1, radii, nthreads=4)), mode
    finally:
        N.destroy(t)
        N.destroy(tq)
