"""Counts where the counters' width would show (exact: integers, no
tolerance)."""
import numpy as np
import pytest

from corruscant_b200 import _native as N

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
