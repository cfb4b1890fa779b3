"""Counts where the counters' width, the padding of partly filled runs, the
exponent range of the FP32 bounds, leaves of very different sizes and often
repeated points would show (exact: integers, no tolerance)."""
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


@pytest.mark.parametrize("seed", [0, 1, 2, 3])
@pytest.mark.parametrize("extent", [1e-15, 1e-18, 1e-19, 1e-20, 1e-21, 3e-22, 1e-22, 5e-23, 3e-23,
                                    1e-23, 1e-38, 1e-45, 1e-150])
def test_squares_below_the_normal_range(extent, seed):
    """Points so close that FP32 squares of their distances are subnormal or
    zero, alone and beside points far away."""
    rs = np.random.RandomState(seed)
    tp, q = extent * rs.rand(256, 3), extent * rs.rand(256, 3)
    radii = np.linspace(0.05, 1.7, 12) * extent
    for far in (0, 40):
        a = np.concatenate([tp, rs.rand(far, 3)])
        b = np.concatenate([q, rs.rand(far, 3)])
        r = np.concatenate([radii, [0.2, 0.6]]) if far else radii
        want = O.OracleTree(a).brute_counts(b, None, 1, r, nthreads=4)
        t = N.build_tree(a, None, 1)
        try:
            for mode in MODES:
                assert np.array_equal(N.count_points(t, b, None, 1, r, mode=mode), want), (far, mode)
        finally:
            N.destroy(t)


@pytest.mark.parametrize("gap,radius", [(2.8e-23, 3e-23), (2.6e-23, 2.7e-23), (3.7e-23, 3.8e-23),
                                        (4.5e-23, 4.4e-23), (1e-22, 0.999e-22)])
def test_gaps_of_a_few_subnormal_steps(gap, radius):
    """Two tight groups whose distance's square is a few steps of 2^-149."""
    rs = np.random.RandomState(3)
    a, b = 1e-27 * rs.rand(64, 3), 1e-27 * rs.rand(64, 3)
    b[:, 0] += gap
    want = O.OracleTree(a).brute_counts(b, None, 1, [radius], nthreads=4)
    assert want[0, 0] == (4096 if radius > gap else 0)
    t = N.build_tree(a, None, 1)
    try:
        for mode in MODES:
            assert np.array_equal(N.count_points(t, b, None, 1, [radius], mode=mode), want), mode
    finally:
        N.destroy(t)


@pytest.mark.parametrize("kind", ["groups", "groups and outlier", "decades", "infinite"])
@pytest.mark.parametrize("seed", [0, 1])
def test_leaves_of_very_different_sizes(kind, seed):
    """Tight groups beside leaves that span the catalog, with edges at the exact
    distances of pairs (those on an edge are not below it)."""
    rs = np.random.RandomState(seed)
    n = 5000
    if kind == "decades":
        p = 10.0 ** (-12 * rs.rand(n, 3)) * np.where(rs.rand(n, 3) < 0.5, -1, 1)
    else:
        p = rs.rand(12, 3)[rs.randint(0, 12, n)] + 1e-6 * rs.normal(size=(n, 3))
        p[::50] = rs.rand(len(p[::50]), 3)
        if kind == "groups and outlier":
            p[n // 3] = [1e12, -1e12, 1e12]
        elif kind == "infinite":
            p[n // 3, 0], p[n // 2, 2] = np.inf, -np.inf
    a, b = p[rs.randint(0, n, 4000)], p[rs.randint(0, n, 4000)]
    with np.errstate(invalid="ignore"):
        d = np.sqrt(((a - b) ** 2).sum(1))
    d = np.unique(d[np.isfinite(d) & (d > 0)])
    radii = np.concatenate([d[np.linspace(0, len(d) - 1, 25).astype(int)], [1e-8, 1e-7, 1e-6]])
    f = rs.randint(0, 2, n).astype(np.int32)
    want = O.OracleTree(p, f, 2).brute_counts(p, f, 2, radii, nthreads=4)
    t = N.build_tree(p, f, 2)
    try:
        for mode in MODES:
            assert np.array_equal(N.count_radii(t, t, radii, mode=mode), want), mode
            assert np.array_equal(N.count_points(t, p, f, 2, radii, mode=mode), want), mode
    finally:
        N.destroy(t)


@pytest.mark.parametrize("spread", [1.0, 1e-3, 1e-6])
def test_sparse_trees_and_dense_queries(spread):
    """A tree whose every leaf is far larger than the query blocks."""
    rs = np.random.RandomState(9)
    for nt in (3, 50, 200):
        tp = rs.rand(nt, 3)
        q = 0.5 + spread * (rs.rand(3000, 3) - 0.5)
        radii = np.logspace(-3, 0, 21)
        want = O.OracleTree(tp).brute_counts(q, None, 1, radii, nthreads=4)
        t = N.build_tree(tp, None, 1)
        try:
            got, st = N.count_points(t, q, None, 1, radii, with_stats=True)
            assert np.array_equal(got, want)
            # few of them need the exact path
            assert st["pairs_rechecked"] <= st["pairs_tested"] / 2
            assert np.array_equal(N.count_points(t, q, None, 1, radii, mode=N.KD_MODE_FP64), want)
        finally:
            N.destroy(t)


@pytest.mark.parametrize("kind", ["copies", "zeros", "one place"])
@pytest.mark.parametrize("n", [4097, 20001])
def test_repeated_query_points_over_several_chunks(n, kind):
    """Raw query points repeated more often than a tree accepts, at sizes of
    several chunks of the counting order."""
    rs = np.random.RandomState(n)
    if kind == "copies":
        q = rs.rand(1 + n // 300, 3)[rs.randint(0, 1 + n // 300, n)]
    elif kind == "zeros":
        q = rs.rand(n, 3)
        q[rs.rand(n) < 0.3] = 0.0
        q[rs.rand(n, 3) < 0.05] = -0.0
    else:
        q = np.tile(rs.rand(1, 3), (n, 1))
    f = rs.randint(0, 3, n).astype(np.int32)
    tp = np.unique(np.concatenate([q[:500], rs.rand(3000, 3)]), axis=0)
    tf = rs.randint(0, 3, len(tp)).astype(np.int32)
    radii = np.array([0.03, 0.1, 0.4, 1.2])
    want = O.OracleTree(tp, tf, 3).brute_counts(q, f, 3, radii, nthreads=8)
    t = N.build_tree(tp, tf, 3)
    try:
        for mode in MODES:
            assert np.array_equal(N.count_points(t, q, f, 3, radii, mode=mode), want), mode
    finally:
        N.destroy(t)
