"""Counts of catalogs whose field labels interleave in space, so that leaves
break into runs of one or two points and query blocks hold many fields, against
the oracle's exhaustive counts (exact: integers, no tolerance)."""
import numpy as np
import pytest

from corruscant_b200 import _native as N
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nf", [1, 2, 3, 4, 5, 6, 15, 16, 17, 33, 120, 255])
@pytest.mark.parametrize("n", [40, 128, 700, 2500])
def test_random_labels(n, nf):
    """Numbers of fields at and next to those where the kernel changes its way:
    symmetric, against queries that interleave as well, and against queries of
    one field."""
    rs = np.random.RandomState(1000 * n + nf)
    p, q = rs.rand(n, 3), rs.rand(n // 2 + 1, 3)
    f, g = (rs.randint(0, nf, len(x)).astype(np.int32) for x in (p, q))
    f[0] = g[0] = nf - 1
    one = np.full(len(q), nf // 2, np.int32)
    ot = O.OracleTree(p, f, nf)
    t, tq, t1 = N.build_tree(p, f, nf), N.build_tree(q, g, nf), N.build_tree(q, one, nf)
    try:
        for radii in (np.linspace(0.02, 1.2, 9), np.linspace(0.01, 1.8, 64), [2.0]):
            auto = ot.brute_counts(p, f, nf, radii, nthreads=4)
            cross = ot.brute_counts(q, g, nf, radii, nthreads=4)
            single = ot.brute_counts(q, one, nf, radii, nthreads=4)
            for mode in (N.KD_MODE_MIXED, N.KD_MODE_FP64):
                assert np.array_equal(N.count_radii(t, t, radii, mode=mode), auto), mode
                assert np.array_equal(N.count_radii(t, tq, radii, mode=mode), cross), mode
                assert np.array_equal(N.count_points(t, q, g, nf, radii, mode=mode), cross), mode
                assert np.array_equal(N.count_radii(t, t1, radii, mode=mode), single), mode
                assert np.array_equal(N.count_points(t, q, one, nf, radii, mode=mode), single), mode
            if nf < 20:
                assert np.array_equal(N.count_radii_static(t, tq, radii), cross)
                assert np.array_equal(N.count_radii_static(t, t1, radii), single)
    finally:
        for x in (t, tq, t1):
            N.destroy(x)


@pytest.mark.parametrize("nf", [40, 250])
def test_random_labels_at_any_coordinates(nf):
    """The same where distances overflow or are no numbers."""
    rs = np.random.RandomState(nf)
    p = rs.rand(900, 3)
    p[::7] *= 1e300
    p[3::50, 0], p[5::60, 1] = np.inf, -np.inf
    q = np.concatenate([p[::3], rs.rand(70, 3) * 1e-9])
    f, g = (rs.randint(0, nf, len(x)).astype(np.int32) for x in (p, q))
    radii = np.array([0.0, 1e-9, 0.1, 0.5, 1e150, 1e154, np.inf])
    t = N.build_tree(p, f, nf)
    try:
        for fq in (g, np.zeros(len(q), np.int32)):
            want = O.OracleTree(p, f, nf).brute_counts(q, fq, nf, radii, nthreads=4)
            for mode in (N.KD_MODE_MIXED, N.KD_MODE_FP64):
                assert np.array_equal(N.count_points(t, q, fq, nf, radii, mode=mode), want), mode
    finally:
        N.destroy(t)
